"""Calls whose pairs are routed to several lists of a chain: every pair is
aligned, whichever kernel the chain starts with.  Outputs hold other values
before each call, so that a pair that no kernel takes is seen."""
import ctypes

import numpy as np
import pytest

import wfe
from test_gpu_parity import compare_with_oracle, torch_cuda

pytestmark = pytest.mark.gpu


def joined(*sets):
    """The pairs of several generated sets as one, dealt in turn."""
    ascii = np.concatenate([a for a, _ in sets])
    shifted, at = [], 0
    for a, p in sets:
        q = p.copy()
        q["p_off"] += at
        q["t_off"] += at
        shifted.append(q)
        at += len(a)
    pairs = np.concatenate(shifted)
    return ascii, pairs[np.random.default_rng(1).permutation(len(pairs))]


def align_device(ctx, ascii, pairs, max_len, stride):
    torch = torch_cuda()
    n = len(pairs)
    d_a, d_p = torch.from_numpy(ascii).cuda(), torch.from_numpy(pairs.view(np.uint8)).cuda()
    out = (torch.full((n,), -7, dtype=torch.int32, device="cuda"), torch.full((n, stride), 55, dtype=torch.int8, device="cuda"),
           torch.full((n,), 99, dtype=torch.uint8, device="cuda"))
    ctx.align_device(d_a, d_p, n, max_len, *out, torch.cuda.current_stream())
    torch.cuda.synchronize()
    return tuple(x.cpu().numpy() for x in out)


def check(ascii, pairs, stride, got, some):
    dist, cg, st = got
    assert (st == wfe.PAIR_OK).all(), f"{(st != wfe.PAIR_OK).sum()} of {len(pairs)} pairs, statuses {np.unique(st)}"
    step = slice(None, None, max(1, len(pairs) // some))
    compare_with_oracle(ascii, pairs[step], stride, dist[step], cg[step], st[step])


@pytest.mark.parametrize("p", [.04, .12, .3])  # list 1 full and lists past it; most pairs past it; list 1 empty
def test_prediction_from_tier_1(p):
    """Routing by predicted distance puts pairs in the lists past the first
    tier's, which a plan from tier 1 does not look at."""
    torch_cuda()
    ascii, pairs = wfe.generate(50_000, 1000, p_min=p, p_max=p, seed=3)
    with wfe.Context(max_seq_len=1200, cigar_stride=1400, flags=wfe.FLAG_DEVICE_ONLY) as ctx:
        ctx.set_policy([1200], [1], predict=True)
        check(ascii, pairs, 1400, align_device(ctx, ascii, pairs, 1200, 1400), 400)


@pytest.mark.parametrize("n_long", [0, 20_000])  # an empty last bucket; one whose pairs the plan gives to tier 5
def test_tier_5_bucket_below_a_planned_one(n_long):
    """The last bucket's chain, planned from tier 1, beside a bucket that starts at tier 5."""
    torch_cuda()
    sets = [wfe.generate(40_000 - n_long, 100, 440, p_min=.01, p_max=.15, seed=4)]
    if n_long:
        sets.append(wfe.generate(n_long, 700, 1000, p_min=.1, p_max=.15, seed=5))
    ascii, pairs = joined(*sets)
    with wfe.Context(max_seq_len=1200, cigar_stride=1400, flags=wfe.FLAG_DEVICE_ONLY) as ctx:
        ctx.set_policy([512, 1200], [5, 1])
        check(ascii, pairs, 1400, align_device(ctx, ascii, pairs, 1200, 1400), 400)


@pytest.mark.parametrize("n", [64, 900])  # one batch; three, on two streams
def test_captured_call_clears_its_counters(n):
    """A captured call begins by clearing the counters of its batches, so that
    a replay does not depend on how the batch before it ended."""
    torch = torch_cuda()
    cuda = ctypes.CDLL("libcuda.so.1")
    ascii, pairs = wfe.generate(n, 150, p_min=.05, p_max=.05, seed=6)
    d_a, d_p = torch.from_numpy(ascii).cuda(), torch.from_numpy(pairs.view(np.uint8)).cuda()
    out = (torch.full((n,), -7, dtype=torch.int32, device="cuda"), torch.zeros((n, 152), dtype=torch.int8, device="cuda"),
           torch.full((n,), 99, dtype=torch.uint8, device="cuda"))
    with wfe.Context(max_seq_len=200, cigar_stride=152, batch_size=300, flags=wfe.FLAG_DEVICE_ONLY) as ctx:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.stream(stream):
            ctx.align_device(d_a, d_p, n, 200, *out, stream)
            stream.synchronize()
            for x in out:
                x.fill_(99)
            with torch.cuda.graph(graph, stream=stream):
                ctx.align_device(d_a, d_p, n, 200, *out, stream)
            roots, count = (ctypes.c_void_p * 8)(), ctypes.c_size_t(8)
            assert cuda.cuGraphGetRootNodes(ctypes.c_void_p(graph.raw_cuda_graph()), roots, ctypes.byref(count)) == 0
            kinds = [ctypes.c_int(-1) for _ in range(count.value)]
            assert all(cuda.cuGraphNodeGetType(ctypes.c_void_p(r), ctypes.byref(k)) == 0 for r, k in zip(roots, kinds))
            assert kinds and all(k.value == 2 for k in kinds)  # CU_GRAPH_NODE_TYPE_MEMSET
            graph.instantiate()
            for _ in range(2):
                graph.replay()
        stream.synchronize()
    check(ascii, pairs, 152, tuple(x.cpu().numpy() for x in out), n)


def test_prediction_of_edits_in_the_first_bases():
    """A few pairs have twice the edits in their first bases: they start no tier of their own."""
    ascii, pairs = wfe.generate(1000, 935, p_min=.12, p_max=.12, seed=5)
    with wfe.Context(max_seq_len=1100, cigar_stride=1100, flags=wfe.FLAG_DEVICE_ONLY) as ctx:
        ctx.set_policy([1100], [1], predict=True)
        got = align_device(ctx, ascii, pairs, 1100, 1100)
        assert list(ctx.stats()["tier_launches"][3:7]) == [1, 0, 0, 0]
    check(ascii, pairs, 1100, got, 1000)


@pytest.mark.parametrize("buckets,lo,hi,predict", [([512, 1200], 600, 1000, False), ([512, 1200], 300, 450, False),
                                                   ([150, 300], 70, 120, False), ([512, 1200], 600, 1000, True)])
def test_small_batches_of_buckets_left_to_their_lengths(buckets, lo, hi, predict):
    """Batches of few pairs start at tier 1, with several buckets as with one."""
    ascii, pairs = wfe.generate(64, lo, hi, p_min=.005, p_max=.005, seed=7)
    with wfe.Context(max_seq_len=buckets[-1], cigar_stride=1200, flags=wfe.FLAG_DEVICE_ONLY) as ctx:
        ctx.set_policy(buckets, predict=predict)
        got = align_device(ctx, ascii, pairs, buckets[-1], 1200)
        assert list(ctx.stats()["tier_entered"][:2]) == [0, 64]
    check(ascii, pairs, 1200, got, 64)
