"""The work that users of the aligner have it do, through its public entry
points, as cases that can be timed and compared.

A case names an entry point ("kind"), the pairs it gets (how many, their text
lengths, log-uniform in [len_min, len_max], and their edit probabilities,
uniform in [p_min, p_max]) and the context's options.  The pairs come from the
package's seeded generator, the one that the tests and the benchmark use.

Kinds:
  device    wfe_align_device: everything in GPU memory, asynchronous
  noalloc   wfe_align_device_noalloc: the same without a context
  pinned    wfe_align on page-locked host buffers, used in place
  pageable  wfe_align on ordinary numpy arrays (FLAG_PAGEABLE_IN_PLACE)
  history   wfe_cigar_from_history_device: the reference's 128-bit backtrace
            records to CIGARs
  serve     wfe_submit / wfe_poll: a burst of requests to the request server

Results are distances, CIGAR slots and statuses: whole numbers and bytes.  The
slots are zero before the first pass, so that the bytes behind a terminator,
which no entry point specifies, are the same for every correct version.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ewfa-gpu_gb300"))

import wfe  # noqa: E402

# length buckets of the mixed-length callers, and the first tier that the
# benchmark's tuning run picks for each (and for the bucket above them)
BUCKETS = [256, 512, 1024, 2048, 4096]
FIRST_TIERS = [1, 1, 5, 5, 5, 5]
# widest CIGAR slot that a caller lays out (the benchmark's mixed workload)
WIDEST_SLOT = 4096


def _case(name, kind, n, len_min, len_max, p_min, p_max, batch=100_000, max_distance=0, buckets=False, requests=0):
    c = {"kind": kind, "n": n, "len_min": len_min, "len_max": len_max, "p_min": p_min, "p_max": p_max,
         "batch": batch, "max_distance": max_distance, "buckets": buckets, "requests": requests}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one small request of a pipeline that aligns as its reads arrive: launch and latency
        _case("device_64_short", "device", 64, 150, 150, 0.05, 0.05),
        # the headline: a sequencer run's short reads, resident on the GPU
        _case("device_1m_short", "device", 1_000_000, 150, 150, 0.05, 0.05),
        # trimmed reads of unequal length and quality, with the reference's search limit
        _case("device_ragged_capped", "device", 200_003, 50, 300, 0.01, 0.12, max_distance=63),
        # a few long reads at a time (an interactive or polishing caller): latency of the long path
        _case("device_8_long", "device", 8, 4000, 6000, 0.04, 0.08),
        # the benchmark's long-read workload
        _case("device_200k_1kb", "device", 200_000, 1000, 1000, 0.10, 0.10, batch=20_000),
        # noisy long reads, the deep end of the distance range in bulk
        _case("device_8k_deep", "device", 8_000, 5000, 7000, 0.06, 0.10),
        # every length and error rate in one batch, in length buckets
        _case("device_mixed", "device", 50_000, 100, 10_000, 0.01, 0.15, buckets=True),
        # a caller whose memory another framework owns
        _case("noalloc_short", "noalloc", 300_000, 150, 150, 0.05, 0.05, max_distance=63),
        # short reads from page-locked host buffers and back: what the CLI does
        _case("pinned_short", "pinned", 500_000, 150, 150, 0.05, 0.05),
        # the same from ordinary numpy arrays, with a batch that does not divide the call
        _case("pageable_short", "pageable", 100_001, 100, 200, 0.02, 0.08, batch=30_000),
        # CIGARs from backtrace records that the reference's kernels left
        _case("history_short", "history", 200_000, 150, 150, 0.05, 0.05),
        # a burst of requests of unequal size to the server
        _case("serve_burst", "serve", 12_000, 100, 5000, 0.01, 0.10, buckets=True, requests=48),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mean_len(c):
    lo, hi = c["len_min"], c["len_max"]
    return (hi - lo) / math.log(hi / lo) if hi > lo else float(lo)


def _cost(c):
    """Wavefront cells and bases, roughly: what a drawn case is held to."""
    lo, hi = float(c["len_min"]), float(c["len_max"])
    p = 0.5 * (c["p_min"] + c["p_max"])
    sq = (hi * hi - lo * lo) / (2 * math.log(hi / lo)) if hi > lo else lo * lo  # mean squared length
    return c["n"] * (p * p * sq + 2.0 * _mean_len(c))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "device", "noalloc", "pinned", "pageable", "history", "serve"])
    most = {"device": 1_000_000, "noalloc": 300_000, "pinned": 500_000, "pageable": 150_000, "history": 200_000,
            "serve": 12_000}[kind]
    longest = {"device": 9000, "noalloc": 300, "pinned": 400, "pageable": 400, "history": 250, "serve": 4000}[kind]
    while True:
        len_min = _log_uniform(rng, 40, longest)
        len_max = len_min if rng.random() < 0.4 else min(longest, _log_uniform(rng, len_min, 8 * len_min) + 1)
        p_min = rng.uniform(0.005, 0.12)
        p_max = p_min if rng.random() < 0.4 else min(0.15, p_min * rng.uniform(1.0, 3.0))
        n = _log_uniform(rng, 16, most)
        batch = rng.choice([100_000, 20_000, 32_768])
        cap = 0
        if kind in ("noalloc", "history"):
            cap = 63
        elif kind == "device" and len_max <= 400 and rng.random() < 0.3:
            cap = 63
        requests = rng.randint(1, 40) if kind == "serve" else 0
        c = _case(None, kind, max(n, requests), len_min, len_max, round(p_min, 4), round(p_max, 4), batch=batch,
                  max_distance=cap, buckets=kind == "serve" or (kind == "device" and len_max >= 2 * len_min),
                  requests=requests)
        if _cost(c) <= 1.2e9:
            return c


def _longest(c):
    """The bound on a sequence's length that a caller states: insertions lengthen the patterns a little."""
    return int(c["len_max"] * 1.12) + 40


def _buckets(longest):
    bounds = [b for b in BUCKETS if b < longest] + [longest]
    return bounds, FIRST_TIERS[:len(bounds)]


def _histories(cg):
    """The 128-bit history of each pair (two words): the operation of score d
    (I = 1, X = 2, D = 3) in 2-bit field d - 1."""
    b = cg.view(np.uint8)
    words = np.zeros((len(cg), 2), np.uint64)
    count = np.zeros(len(cg), np.int64)
    live = np.ones(len(cg), bool)
    code = np.zeros(256, np.uint64)
    code[ord("I")], code[ord("X")], code[ord("D")] = 1, 2, 3
    for j in range(cg.shape[1]):
        live &= b[:, j] != 0
        if not live.any():
            break
        i = np.nonzero(live & (code[b[:, j]] > 0))[0]
        words[i, count[i] // 32] |= code[b[i, j]] << (2 * (count[i] % 32)).astype(np.uint64)
        count[i] += 1
    return words


def _device_outputs(n, stride):
    return (torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros((n, stride), dtype=torch.int8, device="cuda"),
            torch.zeros(n, dtype=torch.uint8, device="cuda"))


def _pinned(a):
    t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
    v = t.numpy().view(a.dtype).reshape(a.shape)
    v[...] = a
    return v


def prepare(case, seed):
    c, kind, n = case, case["kind"], case["n"]
    ascii, pairs = wfe.generate(n, c["len_min"], c["len_max"], p_min=c["p_min"], p_max=c["p_max"],
                                seed=1 + (int(seed) & 0x7FFFFFFF))
    longest = _longest(c)
    stride = min(WIDEST_SLOT, wfe.reference_cigar_stride(c["len_max"]))
    s = {"kind": kind, "n": n, "longest": longest, "stride": stride, "cap": c["max_distance"]}

    if kind in ("device", "noalloc", "history"):
        s["ascii"] = torch.from_numpy(ascii).cuda()
        s["pairs"] = torch.from_numpy(pairs.view(np.uint8)).cuda()
        s["out"] = _device_outputs(n, stride)
    if kind == "device":
        ctx = wfe.Context(max_seq_len=longest, batch_size=c["batch"], cigar_stride=stride,
                          max_distance=c["max_distance"], flags=wfe.FLAG_DEVICE_ONLY)
        if c["buckets"]:
            ctx.set_policy(*_buckets(longest))
        s["ctx"] = ctx
    elif kind == "history":
        # the records that an alignment with the reference's search limit leaves
        with wfe.Context(max_seq_len=longest, cigar_stride=stride, max_distance=63) as ctx:
            dist, cg, _ = ctx.align(_pinned(ascii), _pinned(pairs), out=(_pinned(np.zeros(n, np.int32)),
                                    _pinned(np.zeros((n, stride), np.int8)), _pinned(np.zeros(n, np.uint8))))
            s["dist"] = torch.from_numpy(dist.copy()).cuda()
            s["history"] = torch.from_numpy(_histories(cg).view(np.int64)).cuda()
    elif kind in ("pinned", "pageable"):
        arrays = [ascii, pairs, np.zeros(n, np.int32), np.zeros((n, stride), np.int8), np.zeros(n, np.uint8)]
        if kind == "pinned":
            arrays = [_pinned(a) for a in arrays]
        s["ascii"], s["pairs"] = arrays[:2]
        s["out"] = tuple(arrays[2:])
        s["ctx"] = wfe.Context(max_seq_len=longest, batch_size=c["batch"], cigar_stride=stride,
                               max_distance=c["max_distance"],
                               flags=wfe.FLAG_PAGEABLE_IN_PLACE if kind == "pageable" else 0)
    elif kind == "serve":
        s["ascii"] = _pinned(ascii)
        s["out"] = (np.zeros(n, np.int32), np.zeros((n, stride), np.int8), np.zeros(n, np.uint8))
        bounds, tiers = _buckets(longest)
        s["server"] = wfe.Server(max_seq_len=longest, cigar_stride=stride, memory_bytes=256 << 20,
                                 bucket_max_len=bounds, first_tier=tiers)
        rng = random.Random(seed)
        cuts = [0] + sorted(rng.sample(range(1, n), c["requests"] - 1)) + [n]
        s["requests"] = [(pairs[a:b].copy(), a, b) for a, b in zip(cuts, cuts[1:])]
    return s


def run(state):
    s, kind = state, state["kind"]
    dist, cigar, status = s["out"]
    if kind == "device":
        s["ctx"].align_device(s["ascii"], s["pairs"], s["n"], s["longest"], dist, cigar, status,
                              torch.cuda.current_stream())
    elif kind == "noalloc":
        wfe.align_device_noalloc(s["ascii"], s["pairs"], s["n"], s["longest"], s["cap"], dist, cigar, s["stride"],
                                 status, torch.cuda.current_stream())
    elif kind == "history":
        wfe.cigar_from_history_device(s["ascii"], s["pairs"], s["n"], s["longest"], s["dist"], s["history"], cigar,
                                      s["stride"], status, torch.cuda.current_stream())
        return {"cigar": cigar, "status": status}
    elif kind in ("pinned", "pageable"):
        s["ctx"].align(s["ascii"], s["pairs"], out=s["out"])
    else:
        srv = s["server"]
        sent = [srv.submit(s["ascii"], pairs, out=(dist[a:b], cigar[a:b], status[a:b]))
                for pairs, a, b in s["requests"]]
        for r in sent:
            srv.poll(r)
    return {"dist": dist, "cigar": cigar, "status": status}


def work(case):
    """Each base and descriptor read once, each distance, status and CIGAR
    byte written once (a CIGAR holds about two bytes per edit and one per 127
    matches); histories are read where they are the input.  No floating-point
    operations: the path is integer comparisons."""
    n, length = case["n"], _mean_len(case)
    edits = 0.97 * 0.5 * (case["p_min"] + case["p_max"]) * length
    cigar = 2.0 * edits + length / 127.0 + 2.0
    per = 2.0 * length + 24.0 + cigar + 5.0 + (16.0 if case["kind"] == "history" else 0.0)
    return {"bytes": float(n) * per, "flops": 0.0}


def _edit_distances(ascii, pairs, dev):
    """Edit distances by the textbook recurrence, a row for all pairs at a
    time, in 64-bit integers; bases compared by their 2-bit code."""
    code = torch.from_numpy((ascii.astype(np.int64) & 6) >> 1).to(dev)
    out = torch.zeros(len(pairs), dtype=torch.int64, device=dev)
    order = np.argsort(np.maximum(pairs["p_len"], pairs["t_len"]), kind="stable")
    step = max(1, 40_000_000 // (int(pairs["t_len"].max()) + 1))  # pairs whose rows are held at once
    for i in range(0, len(order), step):
        pick = order[i:i + step]
        p_len = torch.from_numpy(pairs["p_len"][pick].astype(np.int64)).to(dev)
        t_len = torch.from_numpy(pairs["t_len"][pick].astype(np.int64)).to(dev)
        p_off = torch.from_numpy(pairs["p_off"][pick].astype(np.int64)).to(dev)
        t_off = torch.from_numpy(pairs["t_off"][pick].astype(np.int64)).to(dev)
        rows, cols = int(p_len.max()), int(t_len.max())
        h = torch.arange(cols + 1, device=dev)
        text = code[(t_off[:, None] + h[None, :cols]).clamp_(max=len(code) - 1)]
        row = h.expand(len(pick), -1).clone()
        done = torch.where(p_len == 0, t_len, torch.zeros_like(t_len))
        for v in range(1, rows + 1):
            base = code[(p_off + (v - 1)).clamp_(max=len(code) - 1)]
            best = torch.minimum(row[:, 1:] + 1, row[:, :-1] + (text != base[:, None]))
            row = torch.cat([torch.full_like(row[:, :1], v), best], 1) - h
            row = torch.cummin(row, 1).values + h
            done = torch.where(p_len == v, row.gather(1, t_len[:, None])[:, 0], done)
        out[torch.from_numpy(pick).to(dev)] = done
    return out


def exact(case, seed):
    """The distances of small cases by dynamic programming; a CIGAR and a
    status are bytes that have no value to be near to."""
    if case["kind"] == "history" or case["n"] * _mean_len(case) ** 2 > 3e9 or case["len_max"] > 1500:
        return None
    ascii, pairs = wfe.generate(case["n"], case["len_min"], case["len_max"], p_min=case["p_min"], p_max=case["p_max"],
                                seed=1 + (int(seed) & 0x7FFFFFFF))
    dist = _edit_distances(ascii, pairs, "cuda" if torch.cuda.is_available() else "cpu")
    cap = case["max_distance"]
    if cap:
        dist = dist.clamp(max=cap + 1)
    return {"dist": dist, "cigar": None, "status": None}
