"""Distance classes of tier 5 that hold enough pairs for one thread each
(wide_kernel), and the same pairs in lists that several lanes take
(tile_kernel): every class's pairs walked back, against the oracle."""
import numpy as np
import pytest

import wfe
from test_gpu_band import band_pairs, bases, far_pairs
from test_gpu_parity import assert_same_cigars, compare_with_oracle, oracle_run, torch_cuda

pytestmark = pytest.mark.gpu

STRIDE = 4200


def class_pairs(low, limit, length, edits):
    """Pairs of distances in (low, limit], as sequences: scattered edits, long
    indels, repeats, and one operation throughout."""
    rng = np.random.default_rng(limit)
    lengths = [int(x) for x in rng.integers(2 * length // 3, length + 1, 40)]
    seqs = band_pairs(lengths, edits, limit) + far_pairs(rng, 60, length, edits[-1])
    t = bases(rng, length)
    k = (low + limit) // 2
    seqs += [(b"", t[:k]), (t[:k], b""), (t[:k + 40], t[:40]), (t[:33], t[:33 + k]), (t[k:], t), (t, t[:-k]),
             (t[:length // 2] + t[length // 2 + low + 1:], t), (t, t[:9] + t[9 + limit:])]
    ascii, pairs = wfe.pairs_from_list(seqs)
    dist = oracle_run(ascii, pairs, STRIDE)[0]
    return [s for s, d in zip(seqs, dist) if low < d <= limit]


@pytest.mark.parametrize("n", [1500, 28_000])
@pytest.mark.parametrize("low,limit,length,edits", [
    (64, 127, 900, [75, 95, 110]), (127, 193, 1200, [140, 160, 180]), (193, 257, 1300, [205, 230, 250]),
    (257, 321, 1500, [290, 320, 350, 380]), (321, 449, 1700, [370, 420, 470, 540]), (449, 577, 1900, [540, 620, 700, 780]),
    (577, 961, 2000, [760, 900, 1100, 1400])])
def test_pairs_of_one_class(low, limit, length, edits, n):
    torch_cuda()
    seqs = class_pairs(low, limit, length, edits)
    assert len(seqs) >= 40
    others = band_pairs([5, 64, 333, length], [0, 3, 40], 3) + [(b"", b""), (bases(np.random.default_rng(2), length), b"ACGT")]
    ascii, pairs = wfe.pairs_from_list(seqs + others)
    rng = np.random.default_rng(n)
    # every pair at least once, and the class has as many as one thread per pair wants: the scan's bounds put some a class up
    pick = np.concatenate([np.arange(len(pairs)), rng.integers(0, len(seqs), n - len(pairs))])
    pick = pick[rng.permutation(n)]
    assert n < 16384 or (pick < len(seqs)).sum() >= 16384
    with wfe.Context(max_seq_len=2100, cigar_stride=STRIDE) as ctx:
        ctx.set_policy([2100], [5])
        dist, cg, st = ctx.align(ascii, pairs[pick])
    first = np.array([np.flatnonzero(pick == i)[0] for i in range(len(pairs))])
    compare_with_oracle(ascii, pairs, STRIDE, dist[first], cg[first], st[first])
    for i in range(len(pairs)):  # equal pairs have equal results, whatever their warp
        same = np.flatnonzero(pick == i)
        assert (dist[same] == dist[first[i]]).all() and (st[same] == st[first[i]]).all(), i
        assert_same_cigars(cg[same], np.repeat(cg[first[i]:first[i] + 1], len(same), 0))


@pytest.mark.parametrize("n", [153, 384, 385, 1023])
def test_lists_by_cta(n):
    """Lists too short for the bulk kernels: one class, or two, with pairs on
    either side of the limit between them."""
    torch_cuda()
    seqs = [s for low, limit, length, edits in ((0, 127, 900, [30, 75, 110]), (193, 257, 1300, [205, 230, 250]),
                                               (449, 577, 1900, [540, 620, 700]), (577, 961, 2000, [900, 1100, 1400]))
            for s in class_pairs(low, limit, length, edits)[::4]]
    rng = np.random.default_rng(9)
    t = bases(rng, 2000)
    seqs += [(t, t[:1040]), (t, t[:1039]), (t, t[:1038]), (t[:900], t), (bases(rng, 1990), bases(rng, 60)), (b"", b"")]
    ascii, pairs = wfe.pairs_from_list(seqs)
    assert len(pairs) <= 153
    pick = rng.permutation(np.arange(n) % len(pairs))
    with wfe.Context(max_seq_len=2100, cigar_stride=STRIDE) as ctx:
        ctx.set_policy([2100], [5])
        dist, cg, st = ctx.align(ascii, pairs[pick])
    assert (dist > 961).any() and (dist == 961).any() and ((dist > 577) & (dist <= 961)).any()
    compare_with_oracle(ascii, pairs[pick], STRIDE, dist, cg, st)
