"""The bit-parallel band kernels at the sizes where they can go wrong: columns
around whole blocks of 32, texts either side of what tier 0 keeps in shared
memory, distances and length differences either side of the band's limit,
every byte alignment, pairs next to each other and apart; against the oracle."""
import numpy as np
import pytest

import wfe
from test_gpu_parity import _pinned, assert_same_cigars, compare_with_oracle, torch_cuda

pytestmark = pytest.mark.gpu


def bases(rng, n):
    return np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)].tobytes()


def edited(rng, text, edits):
    """`text` after `edits` random edits, a run of insertions or deletions among them now and then."""
    s = list(text)
    while edits > 0:
        k = int(rng.integers(1, 1 + min(edits, 6))) if rng.random() < 0.2 else 1
        at = int(rng.integers(0, len(s) + 1))
        kind = rng.integers(0, 3)
        if kind == 0:
            s[at:at] = bases(rng, k)
        elif kind == 1:
            del s[at:at + k]
        elif at < len(s):
            s[at] = b"ACGT"[(b"ACGT".index(s[at]) + 1) % 4]
        edits -= k
    return bytes(s)


def band_pairs(lengths, edits, seed):
    rng = np.random.default_rng(seed)
    seqs = []
    for n in lengths:
        unit = bases(rng, max(1, n if rng.random() < 0.7 else 1 + n // 9))
        text = (unit * (n // len(unit) + 1))[:n]  # repeats have many optimal paths: the tie order decides
        for e in edits:
            p = edited(rng, text, e)
            seqs.append((p, text) if rng.random() < 0.5 else (text, p))
    return seqs


@pytest.mark.parametrize("cap,stride,spread", [(0, 900, 0), (31, 900, 0), (32, 901, 0), (0, 16, 5000)])
def test_tier_0_band(cap, stride, spread):
    torch_cuda()
    lengths = [0, 1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 150, 159, 160, 161, 191, 192, 193, 320, 600]
    seqs = band_pairs(lengths, [0, 1, 3, 9, 25, 30, 31, 32, 33, 40], 11)
    for d in range(26, 36):  # the ends' diagonals at the edge of the band
        t = bases(np.random.default_rng(d), 150)
        seqs += [(t[d:], t), (t, t[:-d]), (t[:70] + t[70 + d:], t), (b"", t[:d]), (t[:d], b"")]
    ascii, pairs = wfe.pairs_from_list(seqs)
    if spread:  # apart, at every alignment: no warp's pairs lie in one span
        buf, q = np.zeros(spread * 2 * len(pairs), np.uint8), pairs.copy()
        for i, (p, t) in enumerate(seqs):
            for off, s, key in ((2 * i * spread + i % 16, p, "p_off"), ((2 * i + 1) * spread + i // 16 % 16, t, "t_off")):
                buf[off:off + len(s)] = np.frombuffer(s, np.uint8)
                q[key][i] = off
        ascii, pairs = buf, q
    with wfe.Context(max_seq_len=1000, cigar_stride=stride, max_distance=cap) as ctx:
        ctx.set_policy([1000], [0])
        dist, cg, st = ctx.align(_pinned(ascii), _pinned(pairs))  # read where they lie
        assert ctx.stats()["tier_entered"][0] >= len(pairs)
    assert (dist == 31).any() and (dist == 32).any()
    compare_with_oracle(ascii, pairs, stride, dist, cg, st, max_distance=cap)


def far_pairs(rng, n, length, edits):
    """n pairs of up to `length` bases, `edits` edits apart, long indels and repeats among them."""
    seqs = band_pairs([int(x) for x in rng.integers(max(1, length // 3), length + 1, n)], [edits], int(rng.integers(1 << 30)))
    out = []
    for p, t in seqs:
        if len(t) > 200 and rng.random() < 0.3:
            at, k = int(rng.integers(0, len(t) - 100)), int(rng.integers(20, 100))
            t = t[:at] + (bases(rng, k) + t[at:] if rng.random() < 0.5 else t[at + k:])
        out.append((p, t))
    return out


@pytest.mark.parametrize("cap", [0, 300])
@pytest.mark.parametrize("n", [600, 20000])  # the classes by several lanes per pair, and by one thread
@pytest.mark.parametrize("length,edits", [(90, 4), (700, 50), (1100, 110), (1300, 220), (1500, 450), (2200, 900)])
def test_wide_bands(length, edits, n, cap):
    torch_cuda()
    rng = np.random.default_rng(length)
    seqs = far_pairs(rng, 90, length, edits)
    t = bases(rng, length)
    seqs += [(t, t), (b"", t[:60]), (t[:60], b""), (b"", b""), (t[:33], t), (t, t[length // 2:]), (t[:1], t[:1]),
             (b"", t), (t, b""), (bases(rng, length // 2), bases(rng, length // 2))]
    ascii, pairs = wfe.pairs_from_list(seqs)
    pick = rng.permutation(np.arange(n) % len(pairs))
    with wfe.Context(max_seq_len=2500, cigar_stride=5000, max_distance=cap) as ctx:
        ctx.set_policy([2500], [5])
        dist, cg, st = ctx.align(ascii, pairs[pick])
    for i in range(len(pairs)):  # equal pairs have equal results, whatever their warp
        same = np.flatnonzero(pick == i)
        first = same[0]
        assert (dist[same] == dist[first]).all() and (st[same] == st[first]).all(), i
        assert_same_cigars(cg[same], np.repeat(cg[first:first + 1], len(same), 0))
    first = np.array([np.flatnonzero(pick == i)[0] for i in range(len(pairs))])
    compare_with_oracle(ascii, pairs, 5000, dist[first], cg[first], st[first], max_distance=cap)


def replayed(p, t, record, d, slot):
    """The slot and status of a backtrace record, replayed base by base into `slot`."""
    out, v, h, ok = [], 0, 0, True
    for k in range(d + 1):
        run = 0
        while v < len(p) and h < len(t) and p[v] == t[h]:
            v, h, run = v + 1, h + 1, run + 1
        out += [256 - 127] * (run // 127) + ([256 - run % 127] if run % 127 else [])
        op = int(record[k // 32]) >> 2 * (k % 32) & 3 if k < d else 0
        if k < d and op == 0:
            ok = False
            break
        if op:
            out.append(b"?IXD"[op])
            v, h = v + (op != 1), h + (op != 3)
    body = np.array(out + [0] * (-len(out) % 4 or 4 if len(slot) % 4 == 0 else 1), np.uint8)[:len(slot)]
    slot[:len(body)] = body.view(np.int8)
    return wfe.PAIR_BAD_HISTORY if not ok else wfe.PAIR_CIGAR_TRUNCATED if len(out) > len(slot) else wfe.PAIR_OK


@pytest.mark.parametrize("stride,copies", [(800, 1), (801, 1), (16, 1), (0, 1), (800, 90)])
def test_histories(stride, copies):
    """Backtrace records to CIGARs, with the narrow and the wide spans: the
    aligner's own CIGARs from their operations, and the bytes and statuses of
    records that no alignment leaves."""
    torch = torch_cuda()
    rng = np.random.default_rng(5)
    seqs = band_pairs([0, 1, 15, 31, 32, 33, 64, 65, 127, 128, 129, 150, 254, 255, 300, 480, 512], [0, 1, 2, 9, 30, 60], 17)
    seqs = [(p, t) for p, t in seqs if max(len(p), len(t)) <= 512]
    ascii, pairs = wfe.pairs_from_list(seqs)
    n = len(pairs)
    with wfe.Context(max_seq_len=512, cigar_stride=800, max_distance=63) as ctx:
        dist, cg, _ = ctx.align(ascii, pairs)
    hist = np.zeros((n, 2), np.uint64)
    for i in np.flatnonzero(dist < 64):
        ops = [b"?IXD".index(c) for c in cg[i].tobytes()[:cg[i].tobytes().find(0)] if c < 128]
        assert len(ops) == dist[i]
        for d, op in enumerate(ops):
            hist[i, d // 32] |= np.uint64(op << 2 * (d % 32))
    ok = dist < 64
    lone = np.arange(n) % 5 == 4  # codes of any kind, distances of any size
    given, records = dist.copy(), hist.copy()
    given[lone] = rng.integers(-1, 66, lone.sum())
    records[lone] = rng.integers(0, 1 << 63, (lone.sum(), 2), dtype=np.uint64) | np.uint64(0x5555555555555555)
    records[lone & (np.arange(n) % 10 == 9), 0] &= np.uint64(0xfffffffffff0ffff)
    d_a, d_p = torch.from_numpy(ascii).cuda(), torch.from_numpy(pairs.view(np.uint8)).cuda()
    d_d, d_h = torch.from_numpy(given).cuda(), torch.from_numpy(records.view(np.int64)).cuda()
    want, want_st = np.full((n, stride), 7, np.int8), np.zeros(n, np.uint8)
    for i, (p, t) in enumerate(seqs):
        if 0 <= given[i] < 64:
            want_st[i] = replayed(p, t, records[i], given[i], want[i])
        else:
            want[i, :1], want_st[i] = 0, wfe.PAIR_OVER_MAX_DISTANCE
    assert (want_st[lone] == wfe.PAIR_BAD_HISTORY).any()
    d_p, d_d, d_h, n = d_p.repeat(copies), d_d.repeat(copies), d_h.repeat(copies, 1), n * copies
    for max_len in (512, 200):
        out, st = torch.full((n, max(stride, 1)), 7, dtype=torch.int8, device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda")
        wfe.cigar_from_history_device(d_a, d_p, n, max_len, d_d, d_h, out, stride, st, torch.cuda.current_stream())
        torch.cuda.synchronize()
        got, got_st = out.cpu().numpy()[:, :stride], st.cpu().numpy()
        for c in range(1, copies):
            np.testing.assert_array_equal(got[:len(seqs)], got[c * len(seqs):(c + 1) * len(seqs)])
            np.testing.assert_array_equal(got_st[:len(seqs)], got_st[c * len(seqs):(c + 1) * len(seqs)])
        got, got_st = got[:len(seqs)], got_st[:len(seqs)]
        fits = np.maximum(pairs["p_len"], pairs["t_len"]) <= max_len
        np.testing.assert_array_equal(got_st, np.where(fits, want_st, wfe.PAIR_TOO_LONG))
        np.testing.assert_array_equal(got[fits], want[fits])
        if stride == 800:
            assert_same_cigars(got, cg, np.flatnonzero(ok & ~lone & fits))


def test_counters_between_batches():
    """Batches of every kind on one context, a captured one replayed between
    them: each finds the counters of its chain zero."""
    torch = torch_cuda()
    sets = []
    for n, lo, hi, p in [(64, 90, 150, .05), (5000, 300, 400, .3), (3000, 700, 900, .2), (20000, 500, 900, .1), (40, 800, 900, .3)]:
        ascii, pairs = wfe.generate(n, lo, hi, p_min=.01, p_max=p, seed=n)
        out = tuple(torch.zeros(s, dtype=t, device="cuda") for s, t in
                    ((n, torch.int32), ((n, 1200), torch.int8), (n, torch.uint8)))
        sets.append((n, ascii, pairs, torch.from_numpy(ascii).cuda(), torch.from_numpy(pairs.view(np.uint8)).cuda(), out))
    with wfe.Context(max_seq_len=1200, cigar_stride=1200, batch_size=20000, flags=wfe.FLAG_DEVICE_ONLY) as ctx:
        stream = torch.cuda.Stream()

        def run(k):
            n, _, _, a, p, out = sets[k]
            ctx.align_device(a, p, n, 1200, *out, stream)

        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            run(0)
            stream.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                run(0)
        for policy in (None, ([400, 1200], [0, 5]), ([1200], [5]), ([1200], [0])):
            if policy:
                ctx.set_policy(*policy)
            for k in (4, 0, 3, 2, 1, 2, 3, 4, 0):
                for d in sets[k][5] + sets[0][5]:
                    d.zero_()
                torch.cuda.synchronize()
                run(k)
                with torch.cuda.stream(stream):
                    graph.replay()
                stream.synchronize()
                for j in (k, 0):
                    dist, cg, st = (x.cpu().numpy() for x in sets[j][5])
                    some = slice(None, None, 1 + sets[j][0] // 300)
                    compare_with_oracle(sets[j][1], sets[j][2][some], 1200, dist[some], cg[some], st[some])
                    assert (st == wfe.PAIR_OK).all()


@pytest.mark.parametrize("buckets,n,lo,hi,p", [([200], 8192, 40, 180, .2), ([200], 8191, 40, 180, .2), ([256, 500], 40000, 60, 450, .15),
                                               ([64, 128, 512], 700, 10, 460, .15),
                                               ([512], 16384, 200, 460, .12), ([512], 16384, 200, 460, .005)])
def test_large_lists_from_tier_1(buckets, n, lo, hi, p):
    """A first tier of 1: by the band of tier 0, as planned, or by tier 1
    itself, the pairs count as tier 1's and come out the same."""
    torch = torch_cuda()
    ascii, pairs = wfe.generate(n, lo, hi, p_min=.001, p_max=p, seed=n)
    d_a, d_p = torch.from_numpy(ascii).cuda(), torch.from_numpy(pairs.view(np.uint8)).cuda()
    out = tuple(torch.zeros(s, dtype=t, device="cuda") for s, t in
                ((n, torch.int32), ((n, 600), torch.int8), (n, torch.uint8)))
    with wfe.Context(max_seq_len=buckets[-1], cigar_stride=600, flags=wfe.FLAG_DEVICE_ONLY) as ctx:
        ctx.set_policy(buckets, [1] * len(buckets))
        for _ in range(2):
            ctx.align_device(d_a, d_p, n, buckets[-1], *out, torch.cuda.current_stream())
        torch.cuda.synchronize()
        entered = ctx.stats()["tier_entered"]
    assert entered[0] == 0 and entered[1] == 2 * n
    compare_with_oracle(ascii, pairs, 600, *(x.cpu().numpy() for x in out))
