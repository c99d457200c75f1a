/*
 * wfe_kernels.cu -- the alignment path on sm_103a.
 *
 *   pack_kernel          ASCII -> 2-bit words (src/kernels.cu:313-394)
 *   band_kernel          one pair per thread in a bit-parallel band of 32
 *                        diagonals: tier 0, and predicted prefix distances
 *   tier_kernel<Tier>    tiers 1-4: fused load+pack, wavefront compute+extend, bit-packed
 *                        backtrace store, backtrace and CIGAR replay for one
 *                        pair per warp (src/kernels.cu:27-310 and 397-625 in
 *                        one kernel)
 *   long_kernel<GWF, NT> the same for one pair per CTA of NT threads
 *                        (tiers 5-6), over the target's cone when the pair
 *                        has a distance bound
 *   bound_kernel         distance bounds from a 32-diagonal band, one warp
 *                        per pair; routes tier 5's pairs to distance classes
 *   wide_kernel<NW, .>   tier 5 in bulk, one pair per thread, bands of 32 NW
 *                        diagonals: the scan that bounds distances, and the
 *                        classes with the most pairs
 *   tile_kernel          tier 5 in bulk, several lanes per pair
 *   plan_kernel          the first kernel of a large list, from a sample
 *   order_*_kernel       a list in order of length
 *   classify_kernel      length buckets and predicted tiers
 *   history_kernel       CIGARs from the reference's 128-bit histories
 *                        (src/kernels.cu:397-625)
 *
 * Wavefront layout of tier_kernel: lane l of a pair's warp holds, in register
 * chunk c (c = 0..2J), diagonal k = 32*(c-J) - 16 + l.  Neighbours k-1 and
 * k+1 come from one rotating shuffle each; the lanes at a chunk edge pick up
 * the neighbouring chunk's value.  A chunk is skipped (warp-uniformly) until
 * the wavefront [-d, d] reaches it; lanes outside [-d, d] hold -1, the
 * reference's sentinel (src/kernels.cu:205-219).
 *
 * Backtrace store: per score d and chunk, two ballots give the low and high
 * bits of the 2-bit operation of every diagonal of the chunk (2 bits per
 * cell).  The chain is then read back from (D, kt) to (0, 0); it equals the
 * reference's forward history, which copies the history of the source
 * diagonal k + op - 2 and adds op at field d-1 (src/kernels.cu:154-171).
 */
#include "wfe_kernels.cuh"
#include "wfe_band.cuh"

#include <algorithm>
#include <climits>
#include <map>
#include <mutex>
#include <tuple>

namespace wfe {

namespace {

/* Raise, never lower, a kernel's dynamic shared memory limit on the current
 * device.  The limit is a property of the kernel, and a tier launched on the
 * device by one bucket's chain relies on it still covering that bucket after
 * the host has launched the same tier for a smaller bucket. */
cudaError_t allow_smem(const void* fn, size_t bytes)
{
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, size_t> limit;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t& cur = limit[{fn, dev}];
    if (bytes <= cur) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;

enum : int { ST_IDLE = 0, ST_RUN, ST_DONE, ST_OVERFLOW, ST_OVERMAX, ST_TOOLONG, ST_BADWALK, ST_RANGE };

__host__ __device__ constexpr size_t round16(size_t x) { return (x + 15u) & ~size_t(15); }

/* Backtrace store entry of one chunk of one score step: the two ballots of
 * the warp -- the low and the high bits of the 2-bit operation of every lane's
 * diagonal -- written by lane 0.  The chunk's diagonal of lane l is bit l. */
__device__ __forceinline__ int op_of(uint2 e, int bit)
{
    return (int)(((e.x >> bit) & 1u) | (((e.y >> bit) & 1u) << 1));
}

/* One distance tier: a warp per pair, 2J+1 register chunks of 32 diagonals,
 * backtrace store in shared (SMEM_OPS) or global memory. */
template <int J_, bool SMEM_OPS_>
struct Tier {
    static constexpr int J = J_;
    static constexpr bool SMEM_OPS = SMEM_OPS_;
    static constexpr int NC = 2 * J + 1;
    static constexpr int DCAP = 32 * J + 15;
    /* Row d of the backtrace store: only the chunks that score step d touches
     * -- the contiguous range whose diagonals meet [-d, d] -- row after row (a
     * triangle, 55-68 % of DCAP x NC entries), which keeps tier 1's store in
     * shared memory small and tiers 2-4's global scratch mostly in L2. */
    static __host__ __device__ constexpr int chunk_lo(int d) { return J - (d + 15) / 32 < 0 ? 0 : J - (d + 15) / 32; }
    static __host__ __device__ constexpr int chunk_hi(int d)
    {
        return J + (d + 16) / 32 > 2 * J ? 2 * J : J + (d + 16) / 32;
    }
    static __host__ __device__ constexpr int row_entries(int d) { return chunk_hi(d) - chunk_lo(d) + 1; }
    /* entries of rows 1..rows */
    static constexpr int store_entries(int rows = DCAP)
    {
        int t = 0;
        for (int d = 1; d <= rows && d <= DCAP; ++d) t += row_entries(d);
        return t;
    }
    static constexpr size_t ops_bytes = round16(8u * (size_t)store_entries());
    /* one warp's store in global scratch for distances up to max_len */
    static size_t store_bytes(uint32_t max_len)
    {
        return round16(8u * (size_t)store_entries((int)std::min<uint32_t>(max_len, (uint32_t)DCAP)));
    }
    static int store_rows(uint32_t max_len) { return (int)std::min<uint32_t>(max_len, (uint32_t)DCAP); }
    static constexpr size_t chain_bytes = round16((size_t)DCAP + 1);
    static constexpr size_t runs_bytes = round16(sizeof(int) * ((size_t)DCAP + 1));
};

inline uint32_t seq_words_for(uint32_t max_len) { return std::max<uint32_t>(1u, (max_len + 15u) / 16u); }

/* Shared memory of one warp: both sequences, the operation chain, then one
 * region that first holds the backtrace store (when it lives in shared memory)
 * and, once the chain has been read from it, the CIGAR stage and the runs of
 * the replay. */
template <class T>
size_t union_bytes(uint32_t cigar_stride)
{
    const size_t replay = round16(cigar_stride) + T::runs_bytes;
    return T::SMEM_OPS ? std::max(T::ops_bytes, replay) : replay;
}

template <class T>
size_t warp_smem_bytes(uint32_t max_len, uint32_t cigar_stride)
{
    return 16u * (size_t)seq_words_for(max_len) + T::chain_bytes + union_bytes<T>(cigar_stride);
}

template <class T>
size_t cta_smem_bytes(uint32_t max_len, uint32_t cigar_stride)
{
    return warp_smem_bytes<T>(max_len, cigar_stride) * (size_t)kWarps;
}

/* The alignment kernel of tiers 1-4.  Chains launch it from the device, so it
 * declares no launch bounds: a grid launched from the device whose kernel
 * declares launch bounds and uses dynamic shared memory was measured to run
 * one CTA per SM at a time, whatever the bounds say. */
template <class T>
__global__ void tier_kernel(const __grid_constant__ AlignLaunch A, uint32_t seq_words, uint32_t gbytes);

/* launched from the device too: no launch bounds (see tier_kernel) */
template <bool GLOBAL_WF, int NT>
__global__ void long_kernel(const __grid_constant__ AlignLaunch A);
__global__ void bound_kernel(const __grid_constant__ AlignLaunch A, uint32_t seq_words, uint32_t unused);
template <int NW, bool SCAN>
__global__ void wide_kernel(const __grid_constant__ AlignLaunch A);
__global__ void tile_kernel(const __grid_constant__ AlignLaunch A);
template <bool PREDICT>
__global__ void band_kernel(const __grid_constant__ AlignLaunch A, uint32_t nw, uint32_t words);
__device__ uint32_t tile_chunks(const LongClasses& C);
/* The classes of a list of `count` pairs that the bound pass routes, aligned
 * by a CTA per pair.  With so few pairs that nearly every one has a CTA's slot
 * at once, one launch after another costs more than CTAs that fit the
 * distance give: the last class alone, or with the shortest (8 pairs of 4-6
 * kb 0.70 -> 0.36 ms, 256 of 5-7 kb 1.41 -> 0.76 ms; 600 of 2-8 kb at 3-12% 0.72
 * -> 0.55, of 1-9 kb 0.77 -> 0.56).  Pairs of one distance between the two
 * classes lose by it: 600 of 6 kb at 12% 0.61 -> 0.77 ms, 0.63 with the classes
 * between, which cost the lists above 0.76 and 1.04. */
constexpr uint32_t kFewPairs = 384, kSomePairs = 1024;
__device__ __forceinline__ bool class_by_cta(int dlim, uint32_t count)
{
    return count > kFewPairs &&
           (dlim == kCtaClassShort || (count > kSomePairs && (dlim == kCtaClassMiddle || dlim == kCtaClassUpper)));
}
__device__ __forceinline__ bool tile_takes(const LongClasses& C, int c, uint32_t count)
{
    return c + 1 < C.n && C.tile.grid > 0 && count > 0u && !(C.wide[c].grid > 0 && count >= kWidePairs);
}
using T1 = Tier<2, true>;   /* distance <= 79  */
using T2 = Tier<4, false>;  /* distance <= 143; backtrace store in global scratch: 8 CTAs per SM */
using T3 = Tier<8, false>;  /* distance <= 271 */
using T4 = Tier<16, false>; /* distance <= 527 */

/* Which first kernel a list of `count` pairs takes, from the sums over a
 * sample of it: pairs, bases (of the longer sequence), predicted distances D
 * and their squares, and the bulk kernels' work.  Microseconds: the
 * latency of one pair, or the time of all at the rate of a full GPU, measured
 * on lists of 8 to 65,536 pairs of 150 to 9,000 bases at 1-20% edits.
 *   one thread per pair in a 32-diagonal band (tier 0): columns
 *   32 lanes per pair (tier 1, distances to 79): scores
 *   a CTA per pair (bound pass and classes): scores, and cells of D^2
 *   scan and bulk classes: columns times the band's words
 * A list that the host knows to be short never gets here.  8.5 kb at 1.5%
 * edits, 2,048 pairs: a CTA per pair 454 us, in bulk 1,631; 5-7 kb at 6-10%:
 * 2,033 and 1,495; 600 bases at 6%, 4,096 pairs: tier 1 105, bulk 121, tier 0
 * (and what follows it) 195. */
__device__ __forceinline__ int plan_choice(const AlignLaunch& A, uint32_t count, const volatile float* sums)
{
    const float c = sums[0];
    if (c <= 0.f) return kPlanCta;
    const float n = (float)count * 1e-3f, len = sums[1] / c, d = sums[2] / c, dd = sums[3] / c, u = sums[4] / c;
    const float cta = 60.f + fmaxf(d + 0.0045f * d * d, n * (3.2f + 0.0043f * len + 0.2145f * d + 0.0021f * dd));
    const float bulk = 50.f + fmaxf(0.2f * len, n * u);
    int best = bulk < cta ? kPlanBulk : kPlanCta;
    if (A.plan_tiers) {
        float t = fminf(bulk, cta);
        const float reg = 30.f + fmaxf(0.5f * d, n * (0.3f + 0.0015f * len + 0.325f * d));
        const float spread = 2.f * sqrtf(fmaxf(dd - d * d, d));
        if (d + spread < 79.f && reg < t) {
            best = kPlanRegister;
            t = reg;
        }
        const float band = 28.f + fmaxf(0.1f * len, n * 0.0055f * len);
        if (A.plan_tiers == kPlanAll && d + spread < 31.f && band < t) best = kPlanBand;
    }
    return best;
}

/* Whether the plan, if there is one, chose the scan. */
__device__ __forceinline__ bool planned(const AlignLaunch& A) { return !A.plan || *A.plan == (uint32_t)kPlanBulk; }

/* The end of a chain: its counters are zero again for the stage's next batch
 * (Chain::clear).  By the last CTA of its last kernel: nothing reads them any
 * more. */
__device__ __forceinline__ void end_chain(const AlignLaunch& A)
{
    if (!A.chain.clear) return;
    for (int i = 0; i < kTierWords; ++i) A.chain.counts[i] = 0u;
    if (A.tier >= 5 && A.chain.cls.n > 0)
        for (int i = 0; i < kClassWords; ++i) A.chain.cls.counts[i] = 0u;
}

/* Record that the device-side launch of tier u failed: a plain store of one
 * byte (one per tier, so no two writers share a byte) into host memory that
 * the host reads once the chain has completed.  The chain ends here. */
__device__ __forceinline__ void note_launch_error(const AlignLaunch& A, int u)
{
    end_chain(A);
    if (A.chain.launch_error) {
        *reinterpret_cast<volatile uint8_t*>(A.chain.launch_error + u) = 1u;
        __threadfence_system();
    }
}

/* Pairs of a chain cut short were deferred: the host aligns them once the
 * deeper tiers' scratch exists.  (Host memory the device writes in place,
 * like the launch failures.) */
__device__ __forceinline__ void note_deferred(const AlignLaunch& A)
{
    if (A.chain.launch_error) {
        *reinterpret_cast<volatile uint8_t*>(A.chain.launch_error + kDeferByte) = 1u;
        __threadfence_system();
    }
}

/* Tail launch of tier u over its list of `count` pairs, built in the launch's
 * own parameter buffer: A (a __grid_constant__ kernel parameter, read in
 * place) is copied word by word and the per-tier fields are patched
 * (own_list: its work list stays A's; bounds: it has distance bounds, or
 * computes them).  No
 * copy of the launch record is made on the stack -- a kernel whose code
 * holds a large stack frame keeps only a few CTAs resident per SM, and that
 * limit is also what a grid launched from the device runs with. */
template <typename K>
__device__ __forceinline__ void tail_launch(K kernel, const AlignLaunch& A, int u, int grid, int threads,
                                            uint32_t smem, bool tier_args, uint32_t seq_words, uint32_t gbytes,
                                            int bulk = 0, bool own_list = false, bool bounds = true)
{
    void* buf = cudaGetParameterBufferV2((void*)kernel, dim3((unsigned)grid), dim3((unsigned)threads), smem);
    if (!buf) {
        note_launch_error(A, u);
        return;
    }
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&A);
    unsigned long long* dst = static_cast<unsigned long long*>(buf);
    static_assert(sizeof(AlignLaunch) % 8 == 0, "launch record is copied in 8-byte words");
#pragma unroll 4
    for (unsigned i = 0; i < sizeof(AlignLaunch) / 8; ++i) dst[i] = src[i];
    AlignLaunch* n = static_cast<AlignLaunch*>(buf);
    n->tier = u;
    n->cls = -1;
    n->plan = nullptr;
    n->bulk = bulk;
    if (!bounds) n->bound = nullptr;
    if (!own_list) {
        n->work = A.chain.list[u];
        n->work_count = A.chain.counts + u;
    }
    n->retry = u < A.chain.last_tier ? A.chain.list[u + 1] : A.chain.defer;
    n->retry_count = u < A.chain.last_tier ? A.chain.counts + u + 1 : A.chain.defer_count;
    n->passed_total = A.chain.passed ? A.chain.passed + u : nullptr;
    if (tier_args) {
        uint32_t* extra = reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(buf) + sizeof(AlignLaunch));
        extra[0] = seq_words;
        extra[1] = gbytes;
    }
    if (cudaLaunchDeviceV2(buf, cudaStreamTailLaunch) != cudaSuccess) {
        note_launch_error(A, u);
        return;
    }
    if (A.chain.launched) atomicAdd(A.chain.launched + u, 1ull);
}

template <class T>
__device__ __forceinline__ void launch_on_device(const AlignLaunch& A, int u, uint32_t count, bool own_list = false)
{
    const TierShape& sh = A.chain.shape[u];
    const uint32_t per_cta = (uint32_t)kWarps;
    const int grid = max(1, min(sh.grid, (int)((count + per_cta - 1u) / per_cta)));
    tail_launch(tier_kernel<T>, A, u, grid, kThreads, sh.smem, true, sh.seq_words, sh.gbytes, 0, own_list);
}

/* Tail launch of tier 5's start over `count` pairs: the bound pass, or the
 * tier itself for pairs that it takes without (alone_in_tier_5). */
__device__ __forceinline__ void launch_bound_on_device(const AlignLaunch& A, uint32_t count, bool own_list)
{
    if (alone_in_tier_5(count, A.max_len)) {
        const TierShape& sh = A.chain.shape[5];
        tail_launch(long_kernel<false, kLongThreads>, A, 5, max(1, min(sh.grid, (int)count)), kLongThreads, sh.smem,
                    false, 0u, 0u, 0, own_list, false);
        return;
    }
    const TierShape& b = A.chain.bound_shape;
    const uint32_t per_cta = (uint32_t)b.threads / 32u;
    const int grid = max(1, min(b.grid, (int)((count + per_cta - 1u) / per_cta)));
    tail_launch(bound_kernel, A, 5, grid, b.threads, b.smem, true, b.seq_words, 0u, 0, own_list);
}

/* Tail launch of distance class c of tier 5 over its list of `count`
 * pairs.  A pair that a class hands on (its bound was not one) goes to the
 * next class; the last class hands on to tier 6. */
__device__ void launch_class_on_device(const AlignLaunch& A, int c, uint32_t count)
{
    const LongClasses& C = A.chain.cls;
    const TierShape& sh = C.shape[c];
    /* one thread per pair or a CTA per pair, by the number of pairs */
    const bool wide = A.bulk && C.wide[c].grid > 0 && count >= kWidePairs;
    const TierShape& use = wide ? C.wide[c] : sh;
    const int grid = max(1, min(use.grid, wide ? ((int)count + 31) / 32 : (int)count));
    const void* kernel = wide ? (use.dlim == 127   ? (const void*)wide_kernel<4, false>
                                 : use.dlim == 255 ? (const void*)wide_kernel<8, false>
                                 : use.dlim == 511 ? (const void*)wide_kernel<16, false>
                                                   : (const void*)wide_kernel<32, false>)
                         : sh.threads == kLongTinyThreads    ? (const void*)long_kernel<false, kLongTinyThreads>
                         : sh.threads == kLongSmallThreads ? (const void*)long_kernel<false, kLongSmallThreads>
                                                           : (const void*)long_kernel<false, kLongThreads>;
    void* buf = cudaGetParameterBufferV2((void*)kernel, dim3((unsigned)grid), dim3((unsigned)use.threads),
                                         use.smem);
    if (!buf) {
        note_launch_error(A, 5);
        return;
    }
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&A);
    unsigned long long* dst = static_cast<unsigned long long*>(buf);
#pragma unroll 4
    for (unsigned i = 0; i < sizeof(AlignLaunch) / 8; ++i) dst[i] = src[i];
    AlignLaunch* n = static_cast<AlignLaunch*>(buf);
    const bool last = c + 1 >= C.n;
    n->tier = 5;
    n->cls = c;
    n->plan = nullptr;
    n->work = C.list[c];
    n->work_count = C.counts + c;
    /* a class of the bulk kernels hands on to the last, which has no such limits */
    const int up = A.bulk ? C.n - 1 : c + 1;
    n->retry = !last ? C.list[up] : (5 < A.chain.last_tier ? A.chain.list[6] : nullptr);
    n->retry_count = !last ? C.counts + up : A.chain.counts + 6;
    n->passed_total = last && A.chain.passed ? A.chain.passed + 5 : nullptr;
    if (cudaLaunchDeviceV2(buf, cudaStreamTailLaunch) != cudaSuccess) {
        note_launch_error(A, 5);
        return;
    }
    if (A.chain.launched) atomicAdd(A.chain.launched + 5, 1ull);
}

/* Called by the last CTA of tier A.tier: tier u (> A.tier) runs over its
 * list of `count` pairs once this grid has completed.  Tier 5 with
 * distance classes starts with the bound pass, which routes its list into
 * the classes. */
__device__ void launch_tier_on_device(const AlignLaunch& A, int u, uint32_t count)
{
    switch (u) {
    case 1: launch_on_device<T1>(A, u, count); break;
    case 2: launch_on_device<T2>(A, u, count); break;
    case 3: launch_on_device<T3>(A, u, count); break;
    case 4: launch_on_device<T4>(A, u, count); break;
    case 5:
        if (A.bound && A.chain.cls.n > 0 && A.chain.cls.scan.grid > 0 && count >= kScanMin) {
            tail_launch(wide_kernel<2, true>, A, u, max(1, min(A.chain.cls.scan.grid, (int)((count + 31u) / 32u))), 32,
                        0u, false, 0u, 0u, 1);
        } else if (A.bound && A.chain.cls.n > 0) {
            launch_bound_on_device(A, count, false);
        } else {
            const TierShape& sh = A.chain.shape[u];
            tail_launch(long_kernel<false, kLongThreads>, A, u, max(1, min(sh.grid, (int)count)), kLongThreads,
                        sh.smem, false, 0u, 0u);
        }
        break;
    case 6: {
        const TierShape& sh = A.chain.shape[u];
        tail_launch(long_kernel<true, kLongThreads>, A, u, max(1, min(sh.grid, (int)count)), kLongThreads, sh.smem,
                    false, 0u, 0u);
        break;
    }
    default: return;
    }
}

/* Tail launch of the tile kernel over the classes it takes. */
__device__ void launch_tile_on_device(const AlignLaunch& A, uint32_t chunks)
{
    const LongClasses& C = A.chain.cls;
    void* buf = cudaGetParameterBufferV2((void*)tile_kernel, dim3((unsigned)max(1, min(C.tile.grid, (int)chunks))),
                                         dim3((unsigned)C.tile.threads), 0u);
    if (!buf) {
        note_launch_error(A, 5);
        return;
    }
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&A);
    unsigned long long* dst = static_cast<unsigned long long*>(buf);
#pragma unroll 4
    for (unsigned i = 0; i < sizeof(AlignLaunch) / 8; ++i) dst[i] = src[i];
    AlignLaunch* n = static_cast<AlignLaunch*>(buf);
    n->tier = 5;
    n->cls = kTileClass;
    n->plan = nullptr;
    n->retry = C.list[C.n - 1];
    n->retry_count = C.counts + C.n - 1;
    n->passed_total = nullptr;
    if (cudaLaunchDeviceV2(buf, cudaStreamTailLaunch) != cudaSuccess) {
        note_launch_error(A, 5);
        return;
    }
    if (A.chain.launched) atomicAdd(A.chain.launched + 5, 1ull);
}

/* The launch that follows this one in the chain: within tier 5 with classes,
 * after the scan (A.bulk) the tile kernel if it takes any class, then the
 * classes that it does not take, in order; else the next tier that has work
 * (pairs handed on, or routed to it up front). */
__device__ void launch_next(const AlignLaunch& A)
{
    if (A.tier == 5 && A.chain.cls.n > 0) {
        const LongClasses& C = A.chain.cls;
        if (A.bulk && A.cls == -1) {
            const uint32_t chunks = tile_chunks(C);
            if (chunks > 0u) {
                launch_tile_on_device(A, chunks);
                return;
            }
        }
        for (int c = A.cls == kTileClass ? 0 : A.cls + 1; c < C.n; ++c) {
            const uint32_t front = *reinterpret_cast<volatile const uint32_t*>(C.counts + c);
            const uint32_t cnt = front + *reinterpret_cast<volatile const uint32_t*>(C.low_counts + c);
            if (cnt > 0u && !(A.bulk && tile_takes(C, c, front))) {
                launch_class_on_device(A, c, cnt);
                return;
            }
        }
    }
    for (int u = A.tier + 1; u <= A.chain.last_tier; ++u) {
        const uint32_t cnt = *reinterpret_cast<volatile const uint32_t*>(A.chain.counts + u);
        if (cnt > 0u) {
            launch_tier_on_device(A, u, cnt);
            return;
        }
    }
    end_chain(A);
}

/* End of a chained kernel: the last CTA to finish starts the next launch. */
__device__ __forceinline__ void chain_next(const AlignLaunch& A)
{
    if (!A.chain.cta_done) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        uint32_t* done = A.cls >= 0 ? A.chain.cls.cta_done + A.cls : A.chain.cta_done + A.tier;
        const unsigned t = atomicAdd(done, 1u);
        if (t == gridDim.x - 1u) {
            __threadfence();
            launch_next(A);
        }
    }
}

/* What becomes of a pair that a tier did not align, by one thread: a pair
 * past the tier's distance goes to the next tier's list (or is deferred, by a
 * chain cut short), the others get their status. */
__device__ __forceinline__ void finish_unaligned(const AlignLaunch& A, uint32_t pi, int state)
{
    if (state == ST_OVERFLOW && A.retry) {
        const uint32_t s = atomicAdd(A.retry_count, 1u);
        if (A.retry != A.chain.defer) {
            A.retry[s] = pi;
        } else {
            if (s < A.chain.defer_cap) A.retry[s] = A.chain.defer_base + pi;
            note_deferred(A);
        }
        if (A.passed_total) atomicAdd(A.passed_total, 1ull);
        return;
    }
    A.dist[pi] = state == ST_OVERMAX ? A.max_distance + 1 : -1;
    if (A.status)
        A.status[pi] = state == ST_OVERMAX  ? (uint8_t)WFE_PAIR_OVER_MAX_DISTANCE
                       : state == ST_BADWALK ? (uint8_t)WFE_PAIR_BAD_HISTORY
                       : state == ST_RANGE   ? (uint8_t)WFE_PAIR_OUT_OF_RANGE
                                             : (uint8_t)WFE_PAIR_TOO_LONG;
    if (A.cigar_stride) A.cigar[(size_t)pi * A.cigar_stride] = 0;
}

template <class T>
__device__ __forceinline__ void tier_body(const AlignLaunch& A, uint32_t seq_words, uint32_t gbytes)
{
    constexpr int J = T::J, NC = T::NC, DCAP = T::DCAP;
    extern __shared__ __align__(16) unsigned char smem[];

    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);

    /* the warp's sequences, chain and union region */
    unsigned char* ws = smem + (size_t)warp * gbytes;
    uint2* QP = reinterpret_cast<uint2*>(ws);
    uint2* QT = QP + seq_words;
    uint8_t* chain = ws + 16u * (size_t)seq_words;
    unsigned char* uni = chain + T::chain_bytes;
    uint2* ops;
    /* last score step the backtrace store holds: a pair that would go past
     * it (never expected: a distance is at most the longest sequence, and
     * the store holds that many rows) goes on to the next tier instead */
    int store_last = DCAP;
    if constexpr (T::SMEM_OPS) {
        ops = reinterpret_cast<uint2*>(uni);
    } else {
        const TierShape& tsh = A.chain.shape[A.tier];
        const size_t slot = (size_t)blockIdx.x * kWarps + (size_t)warp;
        ops = reinterpret_cast<uint2*>(A.ops_scratch + slot * tsh.ops_warp_bytes);
        store_last = min(DCAP, tsh.ops_rows);
    }
    int8_t* stage = reinterpret_cast<int8_t*>(uni);
    int* runs = reinterpret_cast<int*>(uni + round16(A.cigar_stride));

    const uint32_t count = A.work_count ? min(*A.work_count, A.n_work) : A.n_work;
    /* work stealing: each warp takes the next item from the launch's counter
     * (or, without one, every gridDim-th block of items) */
    uint32_t* const work_next = A.chain.work_next ? A.chain.work_next + A.tier : nullptr;
    const uint32_t step = gridDim.x * (uint32_t)kWarps;
    uint32_t item = blockIdx.x * kWarps + (uint32_t)warp;
    if (work_next) {
        uint32_t v = 0;
        if (lane == 0) v = atomicAdd(work_next, 1u);
        item = __shfl_sync(kFull, v, 0);
    }
    while (item < count) {
        const uint32_t pi = A.work ? A.work[item] : item;
        const PairRef pr = get_pair(A.L, pi);
        const uint32_t mx = max(pr.plen, pr.tlen);
        int state = !pr.in_range ? ST_RANGE : (mx > A.max_len || mx > 16u * seq_words) ? ST_TOOLONG : ST_RUN;
        const uint32_t lp = state == ST_RUN ? pr.plen : 0u, lt = state == ST_RUN ? pr.tlen : 0u;
        load_packed<1>(pr.p, lp, QP, lane);
        load_packed<1>(pr.t, lt, QT, lane);
        __syncwarp();

        const int plen = (int)lp, tlen = (int)lt, kt = tlen - plen;
        int O[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) O[c] = -1;
        int D = 0;
        /* score 0: the lane of diagonal 0 extends from the origin
         * (src/kernels.cu:249-258) */
        if (state == ST_RUN && lane == 16) O[J] = extend_lane(QP, QT, plen, tlen, 0, 0);
        {
            const bool hit = state == ST_RUN && lane == 16 && kt == 0 && O[J] == tlen;
            if (__any_sync(kFull, hit)) state = ST_DONE;
        }
        int rowbase = 0;  /* first store entry of step d's row */
        int rowD = 0;     /* ... of step D's row */
        for (int d = 1;; rowbase += T::row_entries(d), ++d) {
            if (!__any_sync(kFull, state == ST_RUN)) break; /* a vote: the branch is the warp's */
            if (d > store_last || (A.max_distance > 0 && d > A.max_distance)) {
                state = (A.max_distance > 0 && d > A.max_distance) ? ST_OVERMAX : ST_OVERFLOW;
                break;
            }
            const int clo = T::chunk_lo(d);
            int N[NC];
            /* compute (src/kernels.cu:129-152) */
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int lo_k = 32 * (c - J) - 16;
                N[c] = -1;
                if (lo_k <= d && lo_k + 31 >= -d) {
                    const int upsrc = (c + 1 < NC) ? O[(c + 1 < NC) ? c + 1 : 0] : -1;
                    const int dnsrc = (c > 0) ? O[(c > 0) ? c - 1 : 0] : -1;
                    const int up = __shfl_sync(kFull, lane == 0 ? upsrc : O[c], (lane + 1) & 31);
                    const int dn = __shfl_sync(kFull, lane == 31 ? dnsrc : O[c], (lane + 31) & 31);
                    const int m = piggyback_max(up, O[c], dn);
                    const unsigned blo = __ballot_sync(kFull, m & 1);
                    const unsigned bhi = __ballot_sync(kFull, m & 2);
                    if (lane == 0) ops[rowbase + c - clo] = make_uint2(blo, bhi);
                    const int k = lo_k + lane;
                    N[c] = (k >= -d && k <= d) ? (m >> 2) : -1;
                }
            }
            /* extend and test the target (src/kernels.cu:173-176, 268) */
            bool hit = false;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int lo_k = 32 * (c - J) - 16;
                if (lo_k <= d && lo_k + 31 >= -d) {
                    const int k = lo_k + lane;
                    if (N[c] >= 0) {
                        N[c] = extend_lane(QP, QT, plen, tlen, k, N[c]);
                        hit |= (k == kt) && (N[c] == tlen);
                    }
                    O[c] = N[c];
                }
            }
            if (__any_sync(kFull, hit)) {
                state = ST_DONE;
                D = d;
                rowD = rowbase;
            }
        }

        if (state == ST_DONE) {
            /* backtrace: from (D, kt) back to (0, 0); a walk that leaves the
             * wavefront (never expected) is reported, not followed */
            int walk_ok = 1;
            if (lane == 0) {
                int k = kt;
                int row = rowD;
                for (int s = D; s >= 1; --s) {
                    if (k < -s || k > s) { walk_ok = 0; break; }
                    const int idx = k + 16 + 32 * J;
                    const int op = op_of(ops[row + idx / 32 - T::chunk_lo(s)], idx & 31);
                    chain[s - 1] = (uint8_t)op;
                    k += op - 2;
                    if (s > 1) row -= T::row_entries(s - 1);
                }
                if (k != 0) walk_ok = 0;
            }
            walk_ok = __shfl_sync(kFull, walk_ok, 0);
            if (!walk_ok) state = ST_BADWALK;
        }
        if (state == ST_DONE) {
            __syncwarp();
            const int len = replay_chain(QP, QT, plen, tlen, chain, D, runs, stage, A.cigar_stride, lane);
            if (A.cigar_stride)
                store_cigar(stage, (uint32_t)len, A.cigar_stride, A.cigar + (size_t)pi * A.cigar_stride, lane);
            if (lane == 0) {
                A.dist[pi] = D;
                if (A.status)
                    A.status[pi] = (uint32_t)len > A.cigar_stride ? (uint8_t)WFE_PAIR_CIGAR_TRUNCATED
                                                                  : (uint8_t)WFE_PAIR_OK;
            }
        } else if (lane == 0) {
            finish_unaligned(A, pi, state);
        }
        __syncwarp();
        if (work_next) {
            uint32_t v = 0;
            if (lane == 0) v = atomicAdd(work_next, 1u);
            item = __shfl_sync(kFull, v, 0);
        } else {
            item += step;
        }
    }

    /* the last CTA to finish starts the next tier that has work */
    chain_next(A);
}

template <class T>
__global__ void tier_kernel(const __grid_constant__ AlignLaunch A, uint32_t seq_words, uint32_t gbytes)
{
    tier_body<T>(A, seq_words, gbytes);
}

/* ------------------------------------------------------------------------ */
/* Tier 0: one pair per thread, a 32-diagonal band (see wfe_band.cuh),
 * distances up to 31.  A warp takes 32 pairs.
 *
 * Bound by the integer pipe.  About 35 instructions a column -- 18 for the
 * column, 8 for the transposition, 1 store, the rest the walk back, which
 * takes one step per edit or block -- and none of it depends on the data but
 * the walk, so the 32 pairs of a warp stay in step.  The wavefront kernel
 * that this replaced (4 lanes per pair) spent 981 warp instructions on a
 * 150-base pair at 5% edits and stepped every pair of a warp to the largest
 * distance of the eight.  1M such pairs, device-resident: 1,032 us before,
 * 395 us now; 300k without a context 391 and 143 us; 500k from page-locked
 * host memory 940 and 900 us (the CPU-GPU link bounds it); 200k pairs of
 * 50-300 bases at 1-12% edits 470 and 186 us.  130 registers (144 allocated)
 * keep 12 warps on an SM: with 128, 120 or 112 and 13 warps, 1M pairs took
 * 398, 400 and 405 us.
 *
 * The warp's shared memory (words; a lane owns column `lane` of every row):
 *   blocks  D0 of 32 columns, transposed: row q holds band bit q's
 *   ckpt    VP and VN before every block of 32 columns
 *   planes  the two bit planes of pattern and text, rows of 33 words, so that
 *           a lane reading its own words and eight lanes writing one pair's
 *           consecutive words are both free of bank conflicts
 *   bytes   the CIGAR, written backwards
 * The warp keeps as many of the last blocks as fit, 16 rows of each around
 * the ends' diagonals.  The blocks before them, and all blocks for a walk that
 * leaves those rows, are computed again from their checkpoints, with the rows
 * around the walk, when it reaches them. */
constexpr int kSpanWords = 160; /* 16-byte blocks of a span: 8 pairs of 150 bases with their file's line marks */
constexpr int kPlaneRow = 33;
/* a span's words, and those read past its last block */
__host__ __device__ constexpr int span_row(int span) { return span + 4; }
static_assert(4 * span_row(kSpanWords) <= 1024, "the spans use the blocks' space");

__host__ __device__ constexpr uint32_t band_words(uint32_t max_len) { return (max_len + 31u) / 32u; }
/* words of a CIGAR of texts of n blocks: 31 operations, 32 runs, and a byte per 127 matches */
__host__ __device__ constexpr uint32_t band_byte_words(uint32_t n) { return (63u + 32u * n / 127u + 3u) / 4u; }
/* words of a warp for texts of n blocks without the blocks, and blocks that are always there */
__host__ __device__ constexpr uint32_t band_fixed_words(uint32_t n)
{
    return 64u * n + 2u * kPlaneRow * (2u * n + 1u) + 32u * band_byte_words(n);
}
constexpr uint32_t kBandBlockWords = 512;
/* Words given to a warp: all blocks of texts up to 160 bases (room for 13 warps
 * per SM, registers for 12; 150-base reads take 0.40 ns a pair; with room for
 * 224 bases, and 8 warps, an eighth more). */
__host__ __device__ constexpr uint32_t band_smem_words(uint32_t max_len)
{
    const uint32_t n = band_words(max_len) + (max_len == 0u), m = n < 5u ? n : 5u;
    const uint32_t all = band_fixed_words(m) + (m > 2u ? m : 2u) * kBandBlockWords;
    const uint32_t one = band_fixed_words(n) + 2u * kBandBlockWords;
    return all > one ? all : one;
}

/* Bit planes of the warp's 32 pairs.  Eight neighbouring pairs that lie in
 * one span of SPAN blocks are read by all lanes in consecutive 16-byte
 * blocks: whole 512-byte rows per instruction, which the CPU-GPU link serves
 * 20% faster than a short run per pair.  Blocks that fall in gaps between the
 * pairs are read too: a span is shorter than a 4 KiB page, so it lies within
 * the page of its first block and the page of its last, and both of those
 * hold a base, so both are mapped.  The sequences of the other pairs are read
 * by eight lanes each, 256 bases at a time, in blocks that hold a base.
 * Words past a sequence's end are not written: rows and columns past the
 * ends are never used.  A word w >= cap is dropped. */
template <int SPAN>
__device__ __forceinline__ void band_load(const char* p, uint32_t lp, const char* t, uint32_t lt, uint32_t* words,
                                          uint32_t* P0, int capP, uint32_t* T0, int capT, int lane)
{
    static_assert(SPAN * 16 <= 4096, "a span must fit in one 4 KiB page");
    constexpr int kRow = span_row(SPAN);
    unsigned long long lo = ~0ull, hi = 0ull;
    if (lp) {
        lo = (unsigned long long)(uintptr_t)p;
        hi = lo + lp;
    }
    if (lt) {
        lo = min(lo, (unsigned long long)(uintptr_t)t);
        hi = max(hi, (unsigned long long)(uintptr_t)t + lt);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(kFull, lo, o));
        hi = max(hi, __shfl_xor_sync(kFull, hi, o));
    }
    lo &= ~15ull;
    const unsigned long long blocks = hi > lo ? (hi - lo + 15ull) >> 4 : 0ull;
    const bool spans = blocks <= (unsigned long long)SPAN;
    const int nblk = spans ? (int)blocks : 0;
    constexpr int R = (SPAN + 31) / 32;
#pragma unroll
    for (int r = 0; r < 4; r += 2) {
        uint4 v[2][R];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4* base = reinterpret_cast<const uint4*>((uintptr_t)__shfl_sync(kFull, lo, 8 * (r + h)));
            const int nb = __shfl_sync(kFull, nblk, 8 * (r + h));
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int b = lane + 32 * i;
                v[h][i] = b < nb ? __ldg(base + b) : make_uint4(0u, 0u, 0u, 0u);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < R; ++i) words[(r + h) * kRow + lane + 32 * i] = planes16(v[h][i]);
    }
    __syncwarp();
    if (spans) {
        const uint32_t* mine = words + (lane >> 3) * kRow;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(which ? t : p);
            const uint32_t len = which ? lt : lp, sh = (uint32_t)(a & 15u);
            const int n = min((int)((len + 31u) >> 5), which ? capT : capP);
            const uint32_t* x = mine + (int)((a - sh - (uintptr_t)lo) >> 4);
            uint32_t* out = (which ? T0 : P0) + lane;
            const int plane = kPlaneRow * (which ? capT : capP);
            uint32_t x0 = n > 0 ? x[0] : 0u;
            for (int w = 0; w < n; ++w) {
                const uint32_t x1 = x[2 * w + 1], x2 = x[2 * w + 2];
                uint32_t b0, b1;
                planes32(x0, x1, x2, sh, b0, b1);
                out[w * kPlaneRow] = b0;
                out[w * kPlaneRow + plane] = b1;
                x0 = x2;
            }
        }
    }
    if (__any_sync(kFull, !spans)) {
        const int g = lane & 7;
#pragma unroll 1
        for (int it = 0; it < 16; ++it) {
            const int own = 2 * it + (lane >> 4), which = (lane >> 3) & 1;
            const char* sp = reinterpret_cast<const char*>(
                __shfl_sync(kFull, (unsigned long long)(uintptr_t)p, own));
            const char* st = reinterpret_cast<const char*>(
                __shfl_sync(kFull, (unsigned long long)(uintptr_t)t, own));
            const uint32_t np = __shfl_sync(kFull, lp, own), nt = __shfl_sync(kFull, lt, own);
            const bool skip = __shfl_sync(kFull, (int)spans, own) != 0;
            const uintptr_t a = reinterpret_cast<uintptr_t>(which ? st : sp);
            const uint32_t len = skip ? 0u : (which ? nt : np), sh = (uint32_t)(a & 15u);
            const uint4* base = reinterpret_cast<const uint4*>(a - sh);
            const int nb = len ? (int)((sh + len + 15u) >> 4) : 0;
            const int cap = which ? capT : capP;
            const int n = min((int)((len + 31u) >> 5), cap);
            const int most = __reduce_max_sync(kFull, n);
            uint32_t* out = (which ? T0 : P0) + own;
            for (int w0 = 0; w0 < most; w0 += 8) {
                const int w = w0 + g, b = 2 * w;
                const uint4 z = make_uint4(0u, 0u, 0u, 0u);
                const uint32_t x0 = planes16(b < nb ? __ldg(base + b) : z);
                const uint32_t x1 = planes16(b + 1 < nb ? __ldg(base + b + 1) : z);
                uint32_t x2 = __shfl_down_sync(kFull, x0, 1, 8);
                if (g == 7) x2 = planes16(b + 2 < nb ? __ldg(base + b + 2) : z);
                uint32_t b0, b1;
                planes32(x0, x1, x2, sh, b0, b1);
                if (w < n) {
                    out[w * kPlaneRow] = b0;
                    out[w * kPlaneRow + kPlaneRow * cap] = b1;
                }
            }
        }
    }
    __syncwarp();
}

extern __shared__ __align__(16) uint32_t band_smem[];

/* D0 of the 32 columns of block m, from VP/VN before it: its rows first ..
 * first + 15, transposed, to the lane's column at `out`; returns VP/VN after
 * it.  P and T: where the lane's columns of the planes begin in band_smem, as
 * out does (pointers would lose their address space); b: see wfe_band.cuh. */
__device__ __forceinline__ uint2 band_rows(int P, int planeP, int T, int planeT, int m, int b, uint32_t vp,
                                           uint32_t vn, int first, int out)
{
    const uint32_t* pw = band_smem + P + m * kPlaneRow;
    const uint32_t l0 = m > 0 ? pw[-kPlaneRow] : 0u, l1 = m > 0 ? pw[planeP - kPlaneRow] : 0u;
    const uint32_t c0 = pw[0], c1 = pw[planeP], n0 = pw[kPlaneRow], n1 = pw[planeP + kPlaneRow];
    const uint32_t a0 = __funnelshift_l(l0, c0, (uint32_t)b), e0 = __funnelshift_l(c0, n0, (uint32_t)b);
    const uint32_t a1 = __funnelshift_l(l1, c1, (uint32_t)b), e1 = __funnelshift_l(c1, n1, (uint32_t)b);
    const uint32_t t0 = band_smem[T + m * kPlaneRow], t1 = band_smem[T + m * kPlaneRow + planeT];
    uint32_t d0[32], rows[16];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const uint32_t x = __funnelshift_r(a0, e0, (uint32_t)j) ^ bit_mask(t0, j);
        const uint32_t eq = ~(x | (__funnelshift_r(a1, e1, (uint32_t)j) ^ bit_mask(t1, j)));
        d0[j] = band_column(eq, vp, vn);
    }
    transpose16(d0, first, rows);
#pragma unroll
    for (int r = 0; r < 16; ++r) band_smem[out + 32 * r] = rows[r];
    return make_uint2(vp, vn);
}

/* One copy of it, for blocks that are computed twice: with the forward pass
 * inlined, texts of 200-300 bases take 8-10% longer.  The forward pass of
 * texts that are stored whole is inlined: 5% less on 150 bases. */
__device__ __noinline__ uint2 band_rows_call(int P, int planeP, int T, int planeT, int m, int b, uint32_t vp,
                                             uint32_t vn, int first, int out)
{
    return band_rows(P, planeP, T, planeT, m, b, vp, vn, first, out);
}

/* A CIGAR of len bytes from the end of a column of backwards-written words
 * (`top` of them, `row` apart) to its slot, words g, g + G, ... by lane g of
 * G: up to the terminator (when it fits) and zeros to the end of its word,
 * or byte by byte where the slots are not word-aligned. */
__device__ __forceinline__ void store_back_bytes(const uint32_t* col, int row, int top, uint32_t len, uint32_t cap,
                                                 int8_t* dst, int g, int G, bool aligned)
{
    const uint32_t nbytes = len < cap ? len + 1u : cap;
    for (uint32_t i = (uint32_t)g; 4u * i < nbytes; i += (uint32_t)G) {
        const uint32_t off = 4u * (uint32_t)top - len + 4u * i; /* byte of the column */
        const int k = (int)(off >> 2);
        const uint32_t w0 = k < top ? col[row * k] : 0u, w1 = k + 1 < top ? col[row * (k + 1)] : 0u;
        const uint32_t w = __funnelshift_r(w0, w1, 8u * (off & 3u));
        if (aligned) {
            reinterpret_cast<uint32_t*>(dst)[i] = w;
        } else {
            for (uint32_t j = 0; j < 4u && 4u * i + j < nbytes; ++j) dst[4u * i + j] = (int8_t)(w >> (8u * j));
        }
    }
}

template <bool PREDICT>
__global__ void __maxnreg__(144) band_kernel(const __grid_constant__ AlignLaunch A, uint32_t nw, uint32_t words)
{
    const int lane = (int)(threadIdx.x & 31u);
    const uint32_t count = A.work_count ? min(*A.work_count, A.n_work) : A.n_work;
    uint32_t* const work_next = A.chain.work_next ? A.chain.work_next + A.tier : nullptr;
    uint32_t wb = blockIdx.x * 32u;
    if (work_next) {
        uint32_t v = 0;
        if (lane == 0) v = atomicAdd(work_next, 32u);
        wb = __shfl_sync(kFull, v, 0);
    }
    while (wb < count) {
        const uint32_t item = wb + (uint32_t)lane;
        int state = ST_IDLE;
        uint32_t pi = 0;
        PairRef pr;
        pr.p = nullptr; pr.t = nullptr; pr.plen = 0; pr.tlen = 0;
        if (item < count) {
            pi = A.work ? A.work[item] : item;
            pr = get_pair(A.L, pi);
            const uint32_t mx = max(pr.plen, pr.tlen);
            state = !pr.in_range ? ST_RANGE
                    : PREDICT ? ST_RUN
                    : (mx > A.max_len || mx > 32u * nw) ? ST_TOOLONG : ST_RUN;
            if constexpr (PREDICT) {
                pr.plen = min(pr.plen, (uint32_t)kPredictPrefix);
                pr.tlen = min(pr.tlen, (uint32_t)kPredictPrefix);
            }
        }
        /* a distance past the band: the next tier's, or past the caller's cap */
        const int past = A.max_distance > 0 && A.max_distance <= kBandDistance ? ST_OVERMAX : ST_OVERFLOW;
        if (state == ST_RUN && abs((int)pr.tlen - (int)pr.plen) > kBandDistance) state = past;
        const uint32_t lp = state == ST_RUN ? pr.plen : 0u, lt = state == ST_RUN ? pr.tlen : 0u;
        const int tlen = (int)lt, kt = tlen - (int)lp, wide = abs(kt);
        /* diagonals b-31..b hold 0 and kt, with as many on either side */
        const int b = kBandDistance + min(0, kt) - (kBandDistance - wide) / 2;
        const int it = b - kt; /* the target's band bit */
        const int nb = max(1, (__reduce_max_sync(kFull, tlen) + 31) >> 5);
        /* rows first .. first + 15 of the band, around both ends' diagonals, or
         * the target's where they lie too far apart */
        const bool apart = wide > 12;
        int first = min(max((apart ? it : (b + it) >> 1) - 8, 0), 16);
        /* blocks from `kept` on are stored */
        const int room = (int)(words - band_fixed_words((uint32_t)nb));
        const int kept = PREDICT ? nb : max(0, nb - room / (int)kBandBlockWords);
        uint32_t* const blocks = band_smem;
        uint32_t* const ckpt = band_smem + room + lane;
        uint32_t* const P0 = ckpt - lane + 64 * nb;
        uint32_t* const T0p = P0 + 2 * kPlaneRow * (nb + 1);
        uint32_t* const bytes = T0p + 2 * kPlaneRow * nb;
        const int top = (int)band_byte_words((uint32_t)nb);
        band_load<kSpanWords>(pr.p, lp, pr.t, lt, blocks, P0, nb + 1, T0p, nb, lane);
        const int P = room + 64 * nb + lane, T = P + 2 * kPlaneRow * (nb + 1);
        const int planeP = kPlaneRow * (nb + 1), planeT = kPlaneRow * nb;

        /* every column, and the distance: |kt| and the increments along the
         * target's diagonal */
        uint32_t vp = ~0u << b, vn = ~vp;
        int D = wide;
        const auto forward = [&](const auto& block) {
#pragma unroll 1
            for (int m = 0; m < nb; ++m) {
                ckpt[64 * m] = vp;
                ckpt[64 * m + 32] = vn;
                const int out = (int)kBandBlockWords * max(0, m - kept) + lane;
                const uint2 v = block(m, out);
                vp = v.x;
                vn = v.y;
                D += __popc(~blocks[out + 32 * (it - first)] & low_bits(min(32, max(0, tlen - 32 * m))));
            }
        };
        if (kept == 0)
            forward([&](int m, int out) { return band_rows(P, planeP, T, planeT, m, b, vp, vn, first, out); });
        else
            forward([&](int m, int out) { return band_rows_call(P, planeP, T, planeT, m, b, vp, vn, first, out); });
        if constexpr (PREDICT) {
            if (item < count)
                A.pred[pi] = (uint16_t)(state == ST_RUN ? min(D, kPredictMost) : state == past ? kPredictMost : 0xffff);
            wb += gridDim.x * 32u;
            __syncwarp();
            continue;
        }
        if (state == ST_RUN)
            state = D > kBandDistance ? past : (A.max_distance > 0 && D > A.max_distance) ? ST_OVERMAX : ST_DONE;

        /* the walk back from the target (see walk_step) */
        BackBytes cg{bytes + lane, 0u, 0, top};
        int m = 0, hb = 0, q = 0, s = 0, run = 0;
        bool walking = state == ST_DONE;
        const auto start = [&] {
            m = tlen > 0 ? (tlen - 1) >> 5 : 0;
            hb = tlen - 32 * m;
            q = it;
            s = D;
            run = 0;
            cg.acc = 0u;
            cg.n = 0;
        };
        /* one step on rows first .. first + 15; false once they do not hold
         * both neighbours (the band's own edges are not passed) */
        const auto step = [&](const uint32_t* rows) {
            const uint32_t* w = rows + 32 * (q - first);
            const int best = walk_step(~w[0], q > first ? ~w[-32] : 0u, q < first + 15 ? ~w[32] : 0u, ckpt[64 * m],
                                       ckpt[64 * m + 32], q, kBandDistance, hb);
            if (best >= 0) {
                const int op = best & 3, x = best >> 2;
                cg.push_run(run + hb - x, 32);
                cg.push((uint32_t)op_letter(op), 32);
                run = 0;
                hb = op == kOpDel ? x : x - 1;
                q += op == kOpDel ? -1 : (op == kOpIns ? 1 : 0);
                if (--s < 0) walking = false; /* never expected */
            } else {
                run += hb;
                hb = 0;
                if (m == 0) walking = false;
            }
            if (hb == 0 && m > 0) {
                --m;
                hb = 32;
            }
            return q >= (first > 0 ? first + 1 : 0) && q <= (first < 16 ? first + 14 : kBandDistance);
        };
        start();
        bool inside = !apart;
        while (walking && inside && m >= kept) inside = step(blocks + (int)kBandBlockWords * (m - kept) + lane);
        if (walking && m >= kept) start(); /* left the stored rows */
        if (__any_sync(kFull, walking)) {
            const int most = __reduce_max_sync(kFull, walking ? m : 0);
#pragma unroll 1
            for (int blk = most; blk >= 0; --blk) {
                while (walking && m == blk) {
                    first = min(max(q - 8, 0), 16);
                    band_rows_call(P, planeP, T, planeT, blk, b, ckpt[64 * blk], ckpt[64 * blk + 32], first, lane);
                    inside = true;
                    while (walking && inside && m == blk) inside = step(blocks + lane);
                }
            }
        }
        if (state == ST_DONE) {
            if (s != 0 || q != b) {
                state = ST_BADWALK;
            } else {
                cg.push_run(run, 32);
                cg.finish(32);
            }
        }
        __syncwarp();

        /* CIGARs: four lanes write a pair's words, eight pairs at a time */
        const uint32_t cap = A.cigar_stride;
        if (cap) {
            const bool aligned = (cap & 3u) == 0u && (reinterpret_cast<uintptr_t>(A.cigar) & 3u) == 0u;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int own = 8 * r + (lane >> 2), g = lane & 3;
                const bool done = __shfl_sync(kFull, state, own) == ST_DONE;
                const uint32_t len = (uint32_t)__shfl_sync(kFull, cg.n, own);
                int8_t* dst = A.cigar + (size_t)__shfl_sync(kFull, pi, own) * cap;
                if (done) store_back_bytes(bytes + own, 32, top, len, cap, dst, g, 4, aligned);
            }
        }
        if (state == ST_DONE) {
            A.dist[pi] = D;
            if (A.status)
                A.status[pi] = (uint32_t)cg.n > cap ? (uint8_t)WFE_PAIR_CIGAR_TRUNCATED : (uint8_t)WFE_PAIR_OK;
        } else if (state != ST_IDLE) {
            finish_unaligned(A, pi, state);
        }
        __syncwarp();
        if (work_next) {
            uint32_t v = 0;
            if (lane == 0) v = atomicAdd(work_next, 32u);
            wb = __shfl_sync(kFull, v, 0);
        } else {
            wb += gridDim.x * 32u;
        }
    }
    chain_next(A);
}

/* ------------------------------------------------------------------------ */
/* Tiers 5 and 6: one CTA of NT threads (128 or 256) per pair, for distances
 * beyond the register tiers.  Step d computes the 2d+1 cells of [-d, d] in
 * 32-cell chunks, one warp per chunk (src/kernels.cu:111-180 with every
 * thread of the CTA); a barrier separates the steps and every thread then
 * tests the target cell (src/kernels.cu:268).  The wavefront's two buffers
 * live in shared memory (tier 5, distances up to kLongSmemDistance, or up
 * to the limit of the launch's distance class) or in the CTA's global
 * scratch (tier 6).  Each step also writes -1 two cells beyond its
 * range, so the next step reads the reference's sentinel there.  The 2-bit
 * backtrace store is in global scratch, row d holding ceil((2d+1)/32) 64-bit
 * entries (low and high operation bits of 32 diagonals). */

/* first entry of row d (d >= 1) of the long-tier backtrace store:
 * sum over e in [1, d-1] of ceil((2e+1)/32) = floor(e/16) + 1 */
__host__ __device__ __forceinline__ uint64_t long_row(int d)
{
    const uint64_t n = (uint64_t)(d - 1);
    const uint64_t a = n >> 4, b = n & 15u;
    return n + 8u * a * (a >= 1 ? a - 1 : 0) + a * (b + 1);
}

template <bool GLOBAL_WF, int NT>
__global__ void long_kernel(const __grid_constant__ AlignLaunch A)
{
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int kW = NT / 32;
    static_assert(kW >= 1, "at least one warp");
    const bool in_class = A.cls >= 0;
    const TierShape& sh = in_class ? A.chain.cls.shape[A.cls] : A.chain.shape[A.tier];
    const int dlim = sh.dlim;
    const int W = 2 * dlim + 5; /* entries per wavefront buffer, centre dlim + 2 */
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
    const uint32_t seq_words = sh.seq_words;
    uint2* QP = reinterpret_cast<uint2*>(smem);
    uint2* QT = QP + seq_words;
    unsigned char* slab = sh.scratch + (size_t)blockIdx.x * sh.slab;
    uint2* ops = reinterpret_cast<uint2*>(slab);
    const uint64_t ops_entries = long_row(dlim + 1);
    uint8_t* chain = slab + ops_entries * 8u;
    int* runs = reinterpret_cast<int*>(chain + ((dlim + 16) & ~15));
    int* wf;
    if constexpr (GLOBAL_WF)
        wf = runs + ((dlim + 4) & ~3);
    else
        wf = reinterpret_cast<int*>(QT + seq_words);
    int* bufA = wf + dlim + 2;     /* centred */
    int* bufB = wf + W + dlim + 2;

    /* a class list: its front part, then its back part from the end */
    const uint32_t front = A.work_count ? *A.work_count : A.n_work;
    const uint32_t count = min(front + (in_class ? A.chain.cls.low_counts[A.cls] : 0u), A.n_work);
    __shared__ uint32_t s_item;
    uint32_t* const work_next = !A.chain.work_next ? nullptr
                                : in_class ? A.chain.cls.work_next + A.cls : A.chain.work_next + A.tier;
    uint32_t item = blockIdx.x;
    if (work_next) {
        if (threadIdx.x == 0) s_item = atomicAdd(work_next, 1u);
        __syncthreads();
        item = s_item;
    }
    while (item < count) {
        const uint32_t pi = !A.work ? item : item < front ? A.work[item] : A.work[A.chain.cls.cap - 1u - (item - front)];
        const PairRef pr = get_pair(A.L, pi);
        const uint32_t mx = max(pr.plen, pr.tlen);
        int state = !pr.in_range ? ST_RANGE : (mx > A.max_len || mx > 16u * seq_words) ? ST_TOOLONG : ST_RUN;
        const int plen = state == ST_RUN ? (int)pr.plen : 0, tlen = state == ST_RUN ? (int)pr.tlen : 0;
        const int kt = tlen - plen;
        /* warps 0 and 1 load the two sequences (warp 0 both, in a one-warp CTA) */
        if (warp == 0) load_packed<4>(pr.p, (uint32_t)plen, QP, lane);
        if (warp == (kW > 1 ? 1 : 0)) load_packed<4>(pr.t, (uint32_t)tlen, QT, lane);
        __syncthreads();
        int D = 0;
        /* last step: the tier's limit or the caller's cap */
        const int dstop = A.max_distance > 0 ? min(dlim, A.max_distance) : dlim;
        /* Cone of the target.  Cell (d, kt) depends only on the cells
         * (s, k) with |k - kt| <= d - s, so the cells that any step up to
         * dub depends on are those with |k - kt| <= dub - s: a step computes
         * [-d, d] cut to [kt - (dub - d), kt + (dub - d)], and every cell
         * it reads lies in the previous step's cut range or on the -1
         * sentinels just beyond [-(d-1), d-1].  Each cell computed holds the
         * full recurrence's value, so the first hit at a step <= dub, and
         * the walk back from it (which stays in the cone), are exactly the
         * full recurrence's.  dub is dstop, or the pair's bound when one was
         * computed below it; a pair with no hit by a bound below dstop (the
         * bound was not one) is aligned again with dub = dstop. */
        int dub = dstop;
        if (state == ST_RUN && A.bound) {
            const int bnd = A.bound[pi];
            if (bnd >= 0 && bnd < dstop)
                dub = max(bnd, abs(kt));
            else if (bnd > dstop && A.retry && (A.max_distance <= 0 || A.max_distance > dlim))
                state = ST_OVERFLOW; /* past this tier: straight to the next */
        }
        while (state == ST_RUN) {
            /* score 0 (src/kernels.cu:249-258) */
            if (threadIdx.x == 0) {
                bufA[0] = extend_lane(QP, QT, plen, tlen, 0, 0);
                bufA[1] = bufA[-1] = bufA[2] = bufA[-2] = -1;
            }
            __syncthreads();
            int* prev = bufA;
            int* next = bufB;
            bool again = false;
            if (!(kt == 0 && prev[0] == tlen)) {
                uint2* row = ops; /* row d of the backtrace store: long_row(d), kept running */
                for (int d = 1;; ++d) {
                    if (d > dub) {
                        if (dub < dstop)
                            again = true;
                        else
                            state = (A.max_distance > 0 && d > A.max_distance) ? ST_OVERMAX : ST_OVERFLOW;
                        break;
                    }
                    const int ncell = 2 * d + 1;
                    const int nchunk = (ncell + 31) >> 5;
                    /* cells i = k + d of [ilo, ihi] */
                    const int ilo = max(0, kt - dub + 2 * d), ihi = min(2 * d, kt + dub);
                    for (int q = (ilo >> 5) + warp; q <= (ihi >> 5); q += kW) {
                        const int i = 32 * q + lane;
                        const int k = i - d;
                        const bool valid = i >= ilo && i <= ihi;
                        int m = 0;
                        if (valid) {
                            m = piggyback_max(prev[k + 1], prev[k], prev[k - 1]);
                            next[k] = extend_lane(QP, QT, plen, tlen, k, m >> 2);
                        }
                        const unsigned lo = __ballot_sync(kFull, m & 1);
                        const unsigned hi = __ballot_sync(kFull, m & 2);
                        if (lane == 0) row[q] = make_uint2(lo, hi);
                    }
                    if (threadIdx.x == 0) next[d + 1] = next[-d - 1] = next[d + 2] = next[-d - 2] = -1;
                    __syncthreads();
                    if (kt >= -d && kt <= d && next[kt] == tlen) { D = d; break; }
                    int* t = prev; prev = next; next = t;
                    row += nchunk;
                }
            }
            if (!again) {
                if (state == ST_RUN) state = ST_DONE;
                break;
            }
            /* every thread has read the last step's target cell before
             * thread 0 rewrites the buffers */
            __syncthreads();
            dub = dstop;
        }
        if (state == ST_DONE && warp == 0) {
            /* backtrace, 32 rows per round: lane r fetches row s-r's entries
             * around the walk (it moves 0-2 positions down per row), then
             * all lanes walk them through shuffles */
            int p = kt + D;
            int s = D;
            bool ok = true;
            while (s >= 1 && ok) {
                const int ctop = p >> 5;
                const int sr = s - lane;
                uint2 e0 = make_uint2(0, 0), e1 = e0, e2 = e0;
                if (sr >= 1) {
                    const uint2* rw = ops + long_row(sr);
                    const int last = (2 * sr) >> 5;
                    if (ctop - 2 >= 0 && ctop - 2 <= last) e0 = rw[ctop - 2];
                    if (ctop - 1 >= 0 && ctop - 1 <= last) e1 = rw[ctop - 1];
                    if (ctop <= last) e2 = rw[ctop];
                }
                const int steps = min(32, s);
                for (int r = 0; r < steps; ++r) {
                    const int sel = (p >> 5) - (ctop - 2);
                    const uint2 mine = sel == 0 ? e0 : (sel == 1 ? e1 : e2);
                    const unsigned lo = __shfl_sync(kFull, mine.x, r);
                    const unsigned hi = __shfl_sync(kFull, mine.y, r);
                    const int bit = p & 31;
                    const int op = (int)(((lo >> bit) & 1u) | (((hi >> bit) & 1u) << 1));
                    const int row = s - r;
                    if (op == 0 || sel < 0 || sel > 2 || p < 0 || p > 2 * row) { ok = false; break; }
                    if (lane == 0) chain[row - 1] = (uint8_t)op;
                    p += op - 3;
                }
                s -= steps;
            }
            if (ok && p != 0) ok = false;
            if (!ok) state = ST_BADWALK;
            __syncwarp();
            if (state == ST_DONE) {
                int8_t* dst = A.cigar_stride ? A.cigar + (size_t)pi * A.cigar_stride : nullptr;
                const int len = replay_chain(QP, QT, plen, tlen, chain, D, runs, dst, dst ? A.cigar_stride : 0u, lane);
                if (lane == 0) {
                    if (dst && (uint32_t)len < A.cigar_stride) dst[len] = 0;
                    A.dist[pi] = D;
                    if (A.status)
                        A.status[pi] = (uint32_t)len > A.cigar_stride ? (uint8_t)WFE_PAIR_CIGAR_TRUNCATED
                                                                      : (uint8_t)WFE_PAIR_OK;
                }
            }
        }
        if (threadIdx.x == 0 && state != ST_DONE && state != ST_IDLE) {
            if (state == ST_OVERFLOW && A.retry) {
                const uint32_t s = atomicAdd(A.retry_count, 1u);
                A.retry[s] = pi;
                if (A.passed_total) atomicAdd(A.passed_total, 1ull);
            } else {
                A.dist[pi] = state == ST_OVERMAX ? A.max_distance + 1 : -1;
                if (A.status)
                    A.status[pi] = state == ST_OVERMAX  ? (uint8_t)WFE_PAIR_OVER_MAX_DISTANCE
                                   : state == ST_BADWALK ? (uint8_t)WFE_PAIR_BAD_HISTORY
                                   : state == ST_RANGE   ? (uint8_t)WFE_PAIR_OUT_OF_RANGE
                                                         : (uint8_t)WFE_PAIR_TOO_LONG;
                if (A.cigar_stride) A.cigar[(size_t)pi * A.cigar_stride] = 0;
            }
        }
        __syncthreads();
        if (work_next) {
            if (threadIdx.x == 0) s_item = atomicAdd(work_next, 1u);
            __syncthreads();
            item = s_item;
        } else {
            item += gridDim.x;
        }
    }

    chain_next(A);
}

/* ------------------------------------------------------------------------ */
/* Long pairs in bulk: one pair per thread, a band of 32 * NW diagonals.
 *
 * wide_kernel<2, true>, the scan, takes tier 5's list.  Its 64 diagonals
 * follow the path (they move by 16 when the column's smallest value nears an
 * edge), so its distance is an upper bound: it routes the pair to the class
 * whose limit covers it.  A pair at distance 63 or less whose band never had
 * to move is aligned on the spot, if half of its warp's pairs are.
 * wide_kernel<NW, false> aligns a class: the bound puts the distance below
 * 32 * NW, so a fixed band that holds both ends' diagonals is exact.
 *
 * Bound by the integer pipe: 13 instructions per word and column and 5 per
 * column, then one pass over 32 diagonals for the walk back.  The wavefront
 * kernels (bound_kernel, long_kernel) spend 72 warp instructions on 32 cells
 * of one pair and 56 more per warp and score, on D^2 / 2 cells; here it is
 * 32 * NW cells a base, for 32 pairs at once and without divergence, but a
 * launch lasts a sequence's length of dependent columns, however few its
 * pairs, and longer the wider its band: a class of fewer than kWidePairs
 * pairs goes to tile_kernel.  200k pairs of 1,000 bases at 10% edits, in
 * batches of 20,000: 15.3 ms from tier 0 up, 8.1 ms from the bound pass and
 * its classes, 1.92 ms so (2.10 with a walk over 64 diagonals).
 *
 * Scratch of a warp (slab; rows of 32 words, a lane's column each): the bit
 * planes of both sequences, VP/VN before every block of 32 columns, and the
 * CIGAR bytes (a lane's words together, written backwards).  The walk goes
 * back block by block: the block's columns are computed again from the
 * checkpoint, but only 32 diagonals around the path, transposed in shared
 * memory, and when the walk nears their edge the block is computed again
 * around where it is.  The 32 diagonals are enough when no optimal path to
 * the cell where the walk enters can leave them: a path that touches an edge
 * diagonal e costs at least V(c0, e) + |e - q|, with V the matrix at the
 * block's first column c0 and q the cell's diagonal (V changes by at most 1
 * per row, and a diagonal is left at a cost of 1), and the cell itself costs
 * at most V(c0, q) + its increments in the block.  Where that test fails (an
 * indel of a dozen bases inside a block), the pair goes to the wavefront
 * kernels. */
struct WideSlab {
    uint32_t p, t, ckpt, bytes; /* first words */
    uint32_t np, nt;            /* plane words per sequence */
    uint32_t bw;                /* words of a lane's CIGAR */
    uint32_t words;             /* of the whole slab */
};

template <int NW>
__host__ __device__ __forceinline__ WideSlab wide_slab(uint32_t max_len)
{
    WideSlab s{};
    s.np = s.nt = (max_len + 31u) / 32u;
    s.p = 0u;
    s.t = s.p + 64u * s.np;
    s.ckpt = s.t + 64u * s.nt;
    s.bytes = s.ckpt + 64u * (uint32_t)NW * s.nt;
    /* at most 32 * NW operations, a run before and after each, a byte per 127 matches */
    s.bw = (64u * (uint32_t)NW + 1u + max_len / 127u + 3u) / 4u;
    s.words = (s.bytes + 32u * s.bw + 63u) & ~63u;
    return s;
}

/* Words [w, end) of a sequence's bit planes, 32 bases each, into rows of the
 * slab (`row` words; the second plane's row after the first's); four words'
 * blocks are loaded at once. */
__device__ __forceinline__ void wide_pack(const char* seq, uint32_t len, uint32_t* out, int row, int w, int end)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(seq);
    const uint32_t sh = (uint32_t)(a & 15u);
    const uint4* base = reinterpret_cast<const uint4*>(a - sh);
    const int nblk = len ? (int)((sh + len + 15u) >> 4) : 0;
    uint32_t x0 = w < end ? planes16(__ldg(base + 2 * w)) : 0u;
    for (; w < end; w += 4) {
        uint4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = 2 * w + 1 + i < nblk ? __ldg(base + 2 * w + 1 + i) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (w + i >= end) break;
            const uint32_t x1 = planes16(v[2 * i]), x2 = planes16(v[2 * i + 1]);
            uint32_t lo, hi;
            planes32(x0, x1, x2, sh, lo, hi);
            out[(size_t)(2 * row) * (w + i)] = lo;
            out[(size_t)(2 * row) * (w + i) + row] = hi;
            x0 = x2;
        }
    }
}

/* sum of the vertical differences of bits [0, n) of NW words */
template <int NW>
__device__ __forceinline__ int column_sum(const uint32_t (&vp)[NW], const uint32_t (&vn)[NW], int n)
{
    int s = 0;
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        const uint32_t m = low_bits(min(32, max(0, n - 32 * i)));
        s += __popc(vp[i] & m) - __popc(vn[i] & m);
    }
    return s;
}

/* The walk back of a pair, by one thread. */
struct Walk {
    int m, hb; /* block of 32 columns, and columns into it */
    int q, b;  /* band bit, and the band's highest diagonal (bit 0) */
    int W;     /* bits of the band, at least 32 */
    int s;     /* score left */
    int run;
    BackBytes cg;
};

/* The window of a walk: the 32 diagonals from this band bit. */
__device__ __forceinline__ int walk_window(int q, int W) { return min(max(q - 16, 0), W - 32); }

/* Rows of a block in a thread's column of shared memory: D0 of the window's
 * 32 bits, transposed, and their vertical differences before the block. */
constexpr int kWalkRows = 34;

/* Fill the rows of block m.  P, T: the thread's columns of the bit planes
 * (rows of `row` words), np words of the pattern's; src(m, t, vp, vn) gives
 * the vertical differences before block m of the band's bits 32t .. 32t+31. */
template <class Src>
__device__ __forceinline__ void walk_fill(uint32_t* rows, int m, int b, int e, const uint32_t* P, const uint32_t* T,
                                          int row, int np, const Src& src)
{
    const uint32_t es = (uint32_t)(e & 31);
    uint32_t vp, vn, p1 = 0u, n1 = 0u;
    src(m, e >> 5, vp, vn);
    if (es) src(m, (e >> 5) + 1, p1, n1);
    vp = __funnelshift_r(vp, p1, es);
    vn = __funnelshift_r(vn, n1, es);
    rows[32 * 32] = vp;
    rows[32 * 33] = vn;
    uint32_t a0[2], a1[2];
    plane_window<2>(P, 2 * row, np, 32 * m - b + e, a0);
    plane_window<2>(P + row, 2 * row, np, 32 * m - b + e, a1);
    const uint32_t t0 = T[(size_t)(2 * row) * m], t1 = T[(size_t)(2 * row) * m + row];
    uint32_t d0[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const uint32_t x = __funnelshift_r(a0[0], a0[1], (uint32_t)j) ^ bit_mask(t0, j);
        d0[j] = band_column(~(x | (__funnelshift_r(a1[0], a1[1], (uint32_t)j) ^ bit_mask(t1, j))), vp, vn);
    }
    transpose32(d0);
#pragma unroll
    for (int r = 0; r < 32; ++r) rows[32 * r] = d0[r];
}

/* Walk through block k.m, whose rows are filled with window w, to the block
 * before it or to the window's edge.  Returns ST_RUN while there is more to
 * walk, ST_DONE at the origin, ST_OVERFLOW when the window's diagonals do not hold every optimal path. */
__device__ __forceinline__ int walk_block(Walk& k, const uint32_t* rows, int e)
{
    const uint32_t vp = rows[32 * 32], vn = rows[32 * 33];
    int c = k.q - e; /* the path's row */
    const int ex = __popc(~rows[32 * c] & low_bits(k.hb));
    {
        /* V(q) - V(first) and V(last) - V(q) at the block's first column */
        const uint32_t above = low_bits(c), below = ~above & 0x7fffffffu;
        const int su = __popc(vp & above) - __popc(vn & above), sd = __popc(vp & below) - __popc(vn & below);
        if ((e > 0 && c - su <= ex) || (e < k.W - 32 && 31 - c + sd <= ex)) return ST_OVERFLOW;
    }
    /* rows to walk on: the band's own edges may be reached, the others not left */
    const int lo = e > 0 ? 1 : 0, hi = e + 32 < k.W ? 30 : 31;
    int state = ST_RUN;
    bool here = true;
    do {
        const int best = walk_step(~rows[32 * c], ~rows[32 * max(c - 1, 0)], ~rows[32 * min(c + 1, 31)], vp, vn, c, 31,
                                   k.hb);
        if (best >= 0) {
            const int op = best & 3, x = best >> 2;
            k.cg.push_run(k.run + k.hb - x, 1);
            k.cg.push((uint32_t)op_letter(op), 1);
            k.run = 0;
            k.hb = op == kOpDel ? x : x - 1;
            c += op == kOpDel ? -1 : (op == kOpIns ? 1 : 0);
            if (--k.s < 0) state = ST_DONE; /* never expected */
        } else {
            k.run += k.hb;
            k.hb = 0;
            if (k.m == 0) state = ST_DONE;
        }
        if (k.hb == 0 && k.m > 0) {
            --k.m;
            k.hb = 32;
            here = false;
        }
    } while (state == ST_RUN && here && c >= lo && c <= hi);
    k.q = e + c;
    return state;
}

/* The end of a walk: at the origin with no score left, or not (never expected). */
__device__ __forceinline__ int walk_end(Walk& k)
{
    if (k.s != 0 || k.q != k.b) return ST_BADWALK;
    k.cg.push_run(k.run, 1);
    k.cg.finish(1);
    return ST_DONE;
}

/* CIGARs and results of up to 32 pairs that one warp walked, bytes at
 * `bytes`, bw words a pair: eight lanes write a pair's words, four pairs at a
 * time. */
__device__ __forceinline__ void store_walked(const AlignLaunch& A, const uint32_t* bytes, int bw, int state, uint32_t pi,
                                             int D, int n, int lane)
{
    const uint32_t cap = A.cigar_stride;
    if (cap) {
        const bool aligned = (cap & 3u) == 0u && (reinterpret_cast<uintptr_t>(A.cigar) & 3u) == 0u;
#pragma unroll 1
        for (int r = 0; r < 8; ++r) {
            const int own = 4 * r + (lane >> 3), g = lane & 7;
            const bool done = __shfl_sync(kFull, state, own) == ST_DONE;
            const uint32_t len = (uint32_t)__shfl_sync(kFull, n, own);
            int8_t* dst = A.cigar + (size_t)__shfl_sync(kFull, pi, own) * cap;
            if (done) store_back_bytes(bytes + (size_t)own * bw, 1, bw, len, cap, dst, g, 8, aligned);
        }
    }
    if (state == ST_DONE) {
        A.dist[pi] = D;
        if (A.status) A.status[pi] = (uint32_t)n > cap ? (uint8_t)WFE_PAIR_CIGAR_TRUNCATED : (uint8_t)WFE_PAIR_OK;
    } else if (state != ST_IDLE && state != ST_RUN) {
        finish_unaligned(A, pi, state);
    }
}

/* Routes a scanned pair by the bound on its distance, as the bound pass does. */
__device__ __forceinline__ void route_by_bound(const AlignLaunch& A, uint32_t pi, int bound, int need, uint32_t count);

template <int NW, bool SCAN>
__device__ __forceinline__ void wide_body(const AlignLaunch& A, uint32_t* blocks)
{
    static_assert(!SCAN || NW == 2, "the scan moves a band of two words");
    constexpr int W = 32 * NW;
    constexpr int kUnroll = NW <= 4 ? 4 : (NW <= 8 ? 2 : 1);
    const int lane = (int)(threadIdx.x & 31u);
    const TierShape& sh = SCAN ? A.chain.cls.scan : A.chain.cls.wide[A.cls];
    const WideSlab S = wide_slab<NW>(A.max_len);
    uint32_t* const slab = reinterpret_cast<uint32_t*>(sh.scratch + (size_t)blockIdx.x * sh.slab);
    uint32_t* const P = slab + S.p + lane;
    uint32_t* const T = slab + S.t + lane;
    uint32_t* const ckpt = slab + S.ckpt + lane;
    /* a class list: its front part, then its back part from the end */
    const uint32_t front = A.work_count ? min(*A.work_count, A.n_work) : A.n_work;
    const uint32_t count = SCAN ? front : min(front + A.chain.cls.low_counts[A.cls], A.n_work);
    uint32_t* const work_next = SCAN ? A.chain.work_next + A.tier : A.chain.cls.work_next + A.cls;
    for (;;) {
        uint32_t wb = 0;
        if (lane == 0) wb = atomicAdd(work_next, 32u);
        wb = __shfl_sync(kFull, wb, 0);
        if (wb >= count) break;
        const uint32_t item = wb + (uint32_t)lane;
        int state = ST_IDLE;
        uint32_t pi = 0;
        PairRef pr;
        pr.p = nullptr; pr.t = nullptr; pr.plen = 0; pr.tlen = 0;
        if (item < count) {
            pi = !A.work ? item : item < front ? A.work[item] : A.work[A.chain.cls.cap - 1u - (item - front)];
            pr = get_pair(A.L, pi);
            state = !pr.in_range ? ST_RANGE : max(pr.plen, pr.tlen) > A.max_len ? ST_TOOLONG : ST_RUN;
        }
        /* a class of the caller's cap may get pairs past its band */
        const int past = A.max_distance > 0 && A.max_distance <= W - 1 ? ST_OVERMAX : ST_OVERFLOW;
        if (!SCAN && state == ST_RUN && abs((int)pr.tlen - (int)pr.plen) > W - 1) state = past;
        const int plen = state == ST_RUN ? (int)pr.plen : 0, tlen = state == ST_RUN ? (int)pr.tlen : 0;
        const int np = (plen + 31) >> 5;
        const int kt = tlen - plen, wide = abs(kt);
        wide_pack(pr.p, (uint32_t)plen, P, 32, 0, np);
        wide_pack(pr.t, (uint32_t)tlen, T, 32, 0, (tlen + 31) >> 5);
        /* diagonals b-W+1..b: 0 and kt, with as many on either side; a scan
         * whose ends lie too far apart starts around 0 */
        bool fixed = !SCAN || wide < W;
        int b = fixed ? (W - 1) + min(0, kt) - (W - 1 - wide) / 2 : W / 2;
        int top = b; /* the value on bit 0 */
        uint32_t vp[NW], vn[NW];
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            vn[i] = low_bits(min(32, max(0, b - 32 * i)));
            vp[i] = ~vn[i];
        }
        for (int m = 0; 32 * m < tlen; ++m) {
            if constexpr (SCAN) {
                if (m > 0) {
                    const int up = __popc(vp[0]) - __popc(vn[0]), down = __popc(vp[1]) - __popc(vn[1]);
                    /* V(32) > V(0): the path runs above; V(64) < V(32): below */
                    if (up > 0 || down < 0) {
                        const int move = up > -down ? -16 : 16;
                        top += move_band(vp, vn, move);
                        b -= move;
                        fixed = false;
                    }
                }
            }
            uint32_t* ck = ckpt + (size_t)(64 * NW) * m;
#pragma unroll
            for (int i = 0; i < NW; ++i) {
                ck[64 * i] = vp[i];
                ck[64 * i + 32] = vn[i];
            }
            uint32_t a0[NW + 1], a1[NW + 1];
            plane_window<NW + 1>(P, 64, np, 32 * m - b, a0);
            plane_window<NW + 1>(P + 32, 64, np, 32 * m - b, a1);
            const uint32_t t0 = T[64 * m], t1 = T[64 * m + 32];
            const int n = min(32, tlen - 32 * m);
            uint32_t on = 0; /* bit 0 of D0, column after column */
#pragma unroll kUnroll
            for (int j = 0; j < n; ++j) {
                uint32_t d0[NW];
                wide_column<NW>(a0, a1, t0, t1, j, vp, vn, d0);
                on = __funnelshift_r(on, d0[0], 1u);
            }
            top += n - __popc(on);
        }
        const int it = b - kt; /* the target's band bit */
        int D = top + column_sum<NW>(vp, vn, min(max(it, 0), W - 1));
        if (SCAN) D += it < 0 ? -it : max(0, it - (W - 1)); /* a row away changes the value by at most 1 */

        if (state == ST_RUN) {
            if (D <= W - 1 && fixed)
                state = A.max_distance > 0 && D > A.max_distance ? ST_OVERMAX : ST_DONE;
            else if (!SCAN)
                state = past;
        }
        if constexpr (SCAN) {
            /* a walk costs the whole warp: with few pairs to align here, a class takes them */
            const unsigned done = __ballot_sync(kFull, state == ST_DONE), running = __ballot_sync(kFull, state == ST_RUN);
            if (state == ST_DONE && 2 * __popc(done) < __popc(done | running)) state = ST_RUN;
            if (state == ST_RUN) {
                A.bound[pi] = D;
                route_by_bound(A, pi, D, A.max_distance > 0 ? min(D, A.max_distance) : D, count);
            }
        }

        Walk k{};
        k.m = tlen > 0 ? (tlen - 1) >> 5 : 0;
        k.hb = tlen - 32 * k.m;
        k.q = it;
        k.b = b;
        k.W = W;
        k.s = D;
        k.cg = BackBytes{slab + S.bytes + (size_t)lane * S.bw, 0u, 0, (int)S.bw};
        bool walking = state == ST_DONE;
        if (walking && tlen == 0) { /* only deletions */
            for (; k.s > 0; --k.s) k.cg.push((uint32_t)'D', 1);
            k.q = b;
            walking = false;
        }
        const int most = __reduce_max_sync(kFull, walking ? k.m + 1 : 0);
        for (int blk = most - 1; blk >= 0; --blk) {
            while (walking && k.m == blk) {
                const int w = walk_window(k.q, W);
                walk_fill(blocks + lane, blk, b, w, P, T, 32, np, [&](int m, int t, uint32_t& p, uint32_t& v) {
                    const uint32_t* c = ckpt + (size_t)(64 * NW) * m + 64 * t;
                    p = c[0];
                    v = c[32];
                });
                const int st = walk_block(k, blocks + lane, w);
                walking = st == ST_RUN;
                if (!walking) state = st;
            }
        }
        if (state == ST_DONE) state = walk_end(k);
        if (SCAN && state == ST_OVERFLOW) {
            /* to the last class, as from the other classes */
            const LongClasses& C = A.chain.cls;
            A.bound[pi] = D;
            C.list[C.n - 1][atomicAdd(C.counts + C.n - 1, 1u)] = pi;
            state = ST_IDLE;
        }
        __syncwarp();
        store_walked(A, slab + S.bytes, (int)S.bw, state, pi, D, k.cg.n, lane);
        __syncwarp();
    }
    chain_next(A);
}

/* Launched from the device too, so a register limit and no launch bounds (see
 * tier_kernel). */
template <int NW, bool SCAN>
__global__ void __maxnreg__(NW <= 4 ? 96 : (NW <= 8 ? 128 : (NW <= 16 ? 168 : 255))) wide_kernel(const __grid_constant__ AlignLaunch A)
{
    __shared__ uint32_t blocks[32 * kWalkRows];
    if (SCAN && !planned(A)) return;
    wide_body<NW, SCAN>(A, blocks);
}

/* ------------------------------------------------------------------------ */
/* Long pairs by several lanes: G lanes per pair, tiles of 32 x 32 cells.
 *
 * Row block bi (32 pattern rows) crosses the column blocks bj = bi + delta of
 * the band, delta in [dlo, dhi], one per step: tile (bi, bj) is computed at
 * step bi + bj by lane bi mod G, from the vertical differences that the lane
 * kept from its previous tile and the horizontal differences that the lane
 * above handed down a step before, two shuffles for 32 columns of about 21
 * instructions.  A band of nd tile diagonals has at most (nd + 1) / 2 tiles
 * per step, so nd <= 2 G.  Differences that come from outside the band count
 * as +1, an upper bound.  The tile diagonals hold every diagonal of
 * [32 dlo, 32 dhi]; dlo and dhi are the least that certify the pair's bound.
 * The vertical differences into each tile are kept for the walk back, which a
 * warp does for all pairs of the CTA, one per thread: four blocks of 32
 * columns at a time, from the operation codes of 32 diagonals around the path,
 * transposed, so that a step is the last set bit of a row.  All warps compute
 * the codes and, at the end, write the CIGARs from the walk's events: the
 * walk is a serial chain beside other CTAs' busy warps, and everything that
 * could be taken out of it was (two fifths of a CTA's time before, one step
 * comparing three diagonals as walk_step does and writing the bytes).
 *
 * A CTA of eight warps takes chunks of up to 32 pairs of a class, the widest
 * class first and each class from the end of its list (the scan's longest
 * pairs come last), all classes in one launch: launched one after another,
 * each class left most of the GPU idle for the length of its longest pair.
 * A pair takes L / 16 steps whatever its band, so the kernel needs tens of
 * times fewer pairs than one thread per pair to fill the GPU, for 1.5 to 2
 * times its instructions.  80 registers keep three CTAs on an SM, so that
 * two compute while the third walks back (128 and two CTAs: 1.2 times the
 * time; 64, with which four fit: 1.04 times).  8,000 pairs of 5,000-7,000 bases
 * at 6-10% edits: 3.9 ms with a CTA per pair, 1.36 ms so, a call among others of
 * three contexts; 50,000 pairs of 100-10,000 bases at 1-15%: 9.3 and 3.55 ms. */
constexpr int kTileWarps = 8;
constexpr int kTileThreads = 32 * kTileWarps;
/* lanes per pair for distances up to dlim: nd <= 2 G for any ends */
__host__ __device__ constexpr int tile_lanes(int dlim) { return (dlim + 126) / 64 < 2 ? 2 : (dlim + 126) / 64; }
__host__ __device__ constexpr int tile_groups(int G) { return 32 / G; } /* pairs per warp */
/* pairs of a CTA: one warp walks them back */
__host__ __device__ constexpr int tile_pairs(int G)
{
    return tile_groups(G) * kTileWarps < 32 ? tile_groups(G) * kTileWarps : 32;
}

struct TileSlab {
    uint32_t t, chars, ckpt, events; /* first words (the pattern's planes at 0) */
    uint32_t nw, nd, ne;            /* words of a plane; tiles kept per column block; events of a pair */
    uint64_t words;
};

__host__ __device__ __forceinline__ TileSlab tile_slab(uint32_t max_len, int dlim)
{
    TileSlab s{};
    const uint32_t G = (uint32_t)tile_lanes(dlim), n = (uint32_t)tile_pairs((int)G), nw = (max_len + 31u) / 32u;
    s.nw = nw;
    s.nd = 2u * G;
    s.t = 2u * n * nw;
    s.chars = (2u * s.t + 3u) & ~3u;
    s.ckpt = s.chars + 8u * n * nw;
    s.events = s.ckpt + 2u * n * nw * s.nd;
    s.ne = (uint32_t)dlim;
    s.words = ((uint64_t)s.events + (uint64_t)n * s.ne + 63u) & ~uint64_t(63);
    return s;
}

/* CTA loads of the classes that the tile kernel takes */
__device__ uint32_t tile_chunks(const LongClasses& C)
{
    uint32_t n = 0;
    for (int c = 0; c + 1 < C.n; ++c) {
        const uint32_t count = *reinterpret_cast<volatile const uint32_t*>(C.counts + c);
        const uint32_t np = (uint32_t)tile_pairs(tile_lanes(C.shape[c].dlim));
        if (tile_takes(C, c, count)) n += (count + np - 1u) / np;
    }
    return n;
}

/* The text of a pair as one byte per base, its code times 64, by the eight
 * threads of a group (g): words of four, from the aligned words that hold a
 * base. */
__device__ __forceinline__ void tile_chars(const char* seq, uint32_t len, uint32_t* out, int g)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(seq);
    const uint32_t sh = (uint32_t)(a & 3u);
    const uint32_t* in = reinterpret_cast<const uint32_t*>(a - sh);
    const int n = (int)((len + 3u) >> 2), last = len ? (int)((sh + len - 1u) >> 2) : -1;
#pragma unroll 4
    for (int k = g; k < n; k += 8) {
        const uint32_t x = __ldg(in + k), y = k < last ? __ldg(in + k + 1) : 0u;
        out[k] = (__funnelshift_r(x, y, 8u * sh) & 0x06060606u) << 5;
    }
}

constexpr int kTileBlocks = kTileWarps / 2; /* blocks whose codes are computed at a time: two warps each */
constexpr int kTileRows = 66;              /* of a block: two planes of 32 rows, and the vertical differences */

/* A CIGAR from a walk's n events -- 4 * (matches after the operation) +
 * operation, last operation first -- and the `lead` matches before the first
 * operation, by a warp. */
__device__ __forceinline__ uint32_t store_events(const uint32_t* ev, int n, int lead, int8_t* dst, uint32_t cap,
                                                 int lane)
{
    uint32_t total = 0;
    for (int base = 0; base <= n; base += 32) {
        const int d = base + lane;
        int r = 0, letter = 0, nb = 0;
        if (d <= n) {
            r = d == 0 ? lead : (int)(ev[n - d] >> 2);
            letter = d < n ? (int)op_letter((int)(ev[n - 1 - d] & 3u)) : 0;
            nb = r / 127 + (r % 127 != 0) + (letter != 0);
        }
        int x = nb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += y;
        }
        uint32_t pos = total + (uint32_t)(x - nb);
        for (int j = r / 127; j > 0; --j, ++pos)
            if (pos < cap) dst[pos] = (int8_t)-127;
        if (r % 127) {
            if (pos < cap) dst[pos] = (int8_t)(-(r % 127));
            ++pos;
        }
        if (letter && pos < cap) dst[pos] = (int8_t)letter;
        total += (uint32_t)__shfl_sync(kFull, x, 31);
    }
    if (lane == 0 && total < cap) dst[total] = 0;
    return total;
}

__global__ void __maxnreg__(80) tile_kernel(const __grid_constant__ AlignLaunch A)
{
    __shared__ uint32_t blocks[kTileBlocks * 32 * kTileRows];
    /* matching rows of each base, per lane: a warp's 512 bytes hold 256 of
     * each half warp, base c of lane l at 64 c + 4 (l % 16), so that a
     * byte of the text, with 4 (l % 16) added, is the address's low byte */
    __shared__ __align__(256) unsigned char match[kTileWarps * 512];
    __shared__ uint32_t s_item;
    __shared__ uint32_t s_pi[32];
    __shared__ int s_plen[32], s_tlen[32], s_dlo[32], s_dhi[32], s_state[32], s_m[32], s_q[32], s_n[32], s_lead[32];
    __shared__ const char* s_seq[64];
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
    const LongClasses& C = A.chain.cls;
    uint32_t* const slab = reinterpret_cast<uint32_t*>(C.tile.scratch + (size_t)blockIdx.x * C.tile.slab);
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(C.work_next + kTileClass, 1u);
        __syncthreads();
        /* chunk s_item, counted from the widest class and from the end of its list */
        uint32_t chunk = s_item, count = 0;
        int cls = C.n - 2, npair = 1;
        for (; cls >= 0; --cls) {
            count = C.counts[cls];
            if (!tile_takes(C, cls, count)) continue;
            npair = tile_pairs(tile_lanes(C.shape[cls].dlim));
            const uint32_t chunks = (count + (uint32_t)npair - 1u) / (uint32_t)npair;
            if (chunk < chunks) break;
            chunk -= chunks;
        }
        if (cls < 0) break;
        const uint32_t first = chunk * (uint32_t)npair;
        const int limit = C.shape[cls].dlim, G = tile_lanes(limit);
        const TileSlab S = tile_slab(A.max_len, limit);
        uint2* const ckpt = reinterpret_cast<uint2*>(slab + S.ckpt);
        const int past = A.max_distance > 0 && A.max_distance <= limit ? ST_OVERMAX : ST_OVERFLOW;
        if (warp == 0) {
            int state = ST_IDLE, plen = 0, tlen = 0, dlo = 0, dhi = 0;
            const uint32_t item = first + (uint32_t)lane;
            if (lane < npair && item < count) {
                const uint32_t pi = C.list[cls][count - 1u - item];
                const PairRef pr = get_pair(A.L, pi);
                s_pi[lane] = pi;
                s_seq[2 * lane] = pr.p;
                s_seq[2 * lane + 1] = pr.t;
                state = !pr.in_range ? ST_RANGE : max(pr.plen, pr.tlen) > A.max_len ? ST_TOOLONG : ST_RUN;
                if (state == ST_RUN) {
                    const int kt = (int)pr.tlen - (int)pr.plen, wide = abs(kt), bound = A.bound[pi];
                    const int dub = bound >= 0 ? min(bound, limit) : limit;
                    if (wide > dub) {
                        state = past;
                    } else {
                        plen = (int)pr.plen;
                        tlen = (int)pr.tlen;
                        const int x = (dub - wide) >> 1;
                        dlo = (min(0, kt) - x) >> 5;
                        dhi = (max(0, kt) + x + 31) >> 5;
                        if (dhi == dlo) ++dhi; /* the walk wants 32 diagonals */
                    }
                }
            }
            s_state[lane] = state;
            s_plen[lane] = plen;
            s_tlen[lane] = tlen;
            s_dlo[lane] = dlo;
            s_dhi[lane] = dhi;
        }
        __syncthreads();
        /* bit planes: every thread a part of a sequence */
        {
            const int parts = kTileThreads / (2 * npair);
            const int seq = (int)threadIdx.x % (2 * npair), part = (int)threadIdx.x / (2 * npair);
            const int own = seq >> 1;
            if (part < parts) {
                const int len = (seq & 1) ? s_tlen[own] : s_plen[own];
                const int n = (len + 31) >> 5, each = (n + parts - 1) / parts, w0 = part * each;
                wide_pack(s_seq[seq], (uint32_t)len, slab + ((seq & 1) ? S.t : 0u) + own, npair, w0, min(n, w0 + each));
            }
            const int who = (int)threadIdx.x >> 3;
            if (who < npair)
                tile_chars(s_seq[2 * who + 1], (uint32_t)s_tlen[who], slab + S.chars + (size_t)(8u * S.nw) * who,
                           (int)threadIdx.x & 7);
        }
        __syncthreads();
        /* forward */
        {
            const int groups = tile_groups(G), grp = lane / G, l = lane - grp * G;
            const int own = warp * groups + grp;
            const bool in = grp < groups && own < npair && s_state[own & 31] == ST_RUN;
            const int plen = in ? s_plen[own] : 0, tlen = in ? s_tlen[own] : 0;
            const int dlo = in ? s_dlo[own] : 0, dhi = in ? s_dhi[own] : 0;
            const int Bp = (plen + 31) >> 5, Bt = (tlen + 31) >> 5;
            const int src = grp * G + (l == 0 ? G - 1 : l - 1);
            const uint32_t* const P = slab + own;
            const uint4* const T = reinterpret_cast<const uint4*>(slab + S.chars + (size_t)(8u * S.nw) * (in ? own : 0));
            unsigned char* const table = match + warp * 512 + (lane >> 4) * 256;
            const uint32_t page = (uint32_t)(warp * 512 + (lane >> 4) * 256), mine = 4u * (uint32_t)(lane & 15);
            const int steps = __reduce_max_sync(kFull, Bp > 0 && Bt > 0 ? Bp + Bt - 1 : 0);
            int bi = l;
            uint32_t vp = 0, vn = 0, hp = 0, hn = 0;
            for (int s = 0; s < steps; ++s) {
                const uint32_t up_p = __shfl_sync(kFull, hp, src), up_n = __shfl_sync(kFull, hn, src);
                while (bi < Bp && s - bi > bi + dhi) bi += G; /* the row block has left the band */
                const int bj = s - bi, lead = max(0, bi + dlo);
                if (bi >= Bp || bj < lead || bj >= Bt) continue;
                if (bj == lead) {
                    vp = ~0u;
                    vn = 0u;
                    const uint32_t p0 = P[(size_t)(2 * npair) * bi], p1 = P[(size_t)(2 * npair) * bi + npair];
                    uint32_t* const rows = reinterpret_cast<uint32_t*>(table + mine);
                    rows[0] = ~(p0 | p1);
                    rows[16] = p0 & ~p1;
                    rows[32] = ~p0 & p1;
                    rows[48] = p0 & p1;
                }
                const bool edge = bi == 0 || bj - bi == dhi;
                const uint32_t in_p = edge ? ~0u : up_p, in_n = edge ? 0u : up_n;
                ckpt[((size_t)bj * S.nd + (size_t)(bi - bj + dhi)) * npair + own] = make_uint2(vp, vn);
                const uint4 ca = T[2 * bj], cb = T[2 * bj + 1];
                const uint32_t chars[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
                /* the bytes past the text's end hold anything: masked, they are bases too */
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const uint32_t at =
                        __byte_perm((chars[j >> 2] & 0xc0c0c0c0u) | mine * 0x01010101u, page, 0x7650u + (j & 3));
                    tile_column(*reinterpret_cast<const uint32_t*>(match + at), in_p << j, in_n << j, vp, vn, hp, hn);
                }
            }
        }
        __syncthreads();
        /* The walk back, a pair per lane of the first warp, with one window of
         * 32 diagonals around where it is for the next four blocks: it seldom
         * moves by 15 diagonals in 128 columns.  When it does, or enters a
         * block too near the window's edge for the test (see wide_kernel), it
         * goes back to the block's entry and the codes are computed again
         * from there. */
        const int dhi = s_dhi[lane], nd = dhi - s_dlo[lane] + 1, W = 32 * (nd - 1) + 1, b = 32 * dhi;
        const int own = lane < npair ? lane : 0, Bp = (s_plen[lane] + 31) >> 5;
        uint32_t* const ev = slab + S.events + (size_t)own * S.ne;
        int state = ST_IDLE, m = 0, hb = 0, q = 0, run = 0, n = 0;
        bool walking = false;
        if (warp == 0) {
            state = s_state[lane];
            const int plen = s_plen[lane], tlen = s_tlen[lane];
            m = tlen > 0 ? (tlen - 1) >> 5 : 0;
            hb = tlen - 32 * m;
            q = b - (tlen - plen);
            walking = state == ST_RUN && plen > 0 && tlen > 0;
            if (state == ST_RUN && !walking) { /* one operation throughout */
                for (; n < plen + tlen; ++n) ev[n] = (uint32_t)(plen ? kOpDel : kOpIns);
                state = ST_DONE;
            }
        }
        for (;;) {
            if (warp == 0) {
                s_m[lane] = walking ? m : -1;
                s_q[lane] = q;
            }
            if (!__syncthreads_or(walking)) break;
            const int m0 = s_m[lane], e = walk_window(s_q[lane], W);
            {
                const int blk = m0 - (warp >> 1);
                uint32_t* const rows = blocks + (warp >> 1) * (32 * kTileRows) + lane;
                const bool high = (warp & 1) != 0;
                if (blk >= 0) {
                    /* tile t of the column block: rows above the matrix or below the pattern are virtual */
                    const auto edge = [&](int t) {
                        const int bi = t + blk - dhi;
                        return bi < 0 ? make_uint2(0u, ~0u)
                               : bi < Bp && t < nd ? ckpt[((size_t)blk * S.nd + (size_t)t) * npair + own]
                                                   : make_uint2(~0u, 0u);
                    };
                    const uint32_t es = (uint32_t)(e & 31);
                    const uint2 c0 = edge(e >> 5), c1 = es ? edge((e >> 5) + 1) : make_uint2(0u, 0u);
                    uint32_t vp = __funnelshift_r(c0.x, c1.x, es), vn = __funnelshift_r(c0.y, c1.y, es);
                    if (!high) {
                        rows[32 * 64] = vp;
                        rows[32 * 65] = vn;
                    }
                    const uint32_t* const P = slab + own;
                    const uint32_t* const T = slab + S.t + own + (size_t)(2 * npair) * blk;
                    uint32_t a0[2], a1[2], code[32];
                    plane_window<2>(P, 2 * npair, Bp, 32 * blk - b + e, a0);
                    plane_window<2>(P + npair, 2 * npair, Bp, 32 * blk - b + e, a1);
                    const uint32_t t0 = T[0], t1 = T[npair];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const uint32_t x = __funnelshift_r(a0[0], a0[1], (uint32_t)j) ^ bit_mask(t0, j);
                        const uint32_t eq = ~(x | (__funnelshift_r(a1[0], a1[1], (uint32_t)j) ^ bit_mask(t1, j)));
                        code[j] = band_column_ops(eq, vp, vn, high);
                    }
                    transpose32(code);
                    uint32_t* const out = rows + (high ? 32 * 32 : 0);
#pragma unroll
                    for (int r = 0; r < 32; ++r) out[32 * r] = code[r];
                }
            }
            __syncthreads();
            if (warp == 0) {
                /* rows to walk on: the band's own edges may be reached, the others not left */
                const int lo = e > 0 ? 1 : 0, hi = e + 32 < W ? 30 : 31;
                int c = q - e;
                /* the walk at the entry of its block */
                int c_in = c, hb_in = hb, run_in = run, n_in = n;
                bool here = walking;
                while (here) {
                    const uint32_t* const rows = blocks + (m0 - m) * (32 * kTileRows) + lane;
                    const uint32_t low = rows[32 * c], high = rows[32 * (32 + c)];
                    const int at = 31 - __clz((int)((low | high) & low_bits(hb)));
                    if (at >= 0) {
                        const int op = (int)((low >> at) & 1u) + 2 * (int)((high >> at) & 1u);
                        if (n < limit) ev[n] = 4u * (uint32_t)(run + hb - 1 - at) + (uint32_t)op;
                        ++n;
                        run = 0;
                        hb = at + (op == kOpDel ? 1 : 0);
                        c += op == kOpDel ? -1 : (op == kOpIns ? 1 : 0);
                    } else {
                        run += hb;
                        hb = 0;
                    }
                    bool again = c < lo || c > hi;
                    if (hb == 0) {
                        /* at the block's first column: could an optimal path leave the window? */
                        const uint32_t vp = rows[32 * 64], vn = rows[32 * 65];
                        const uint32_t above = low_bits(c), below = ~above & 0x7fffffffu;
                        const int su = __popc(vp & above) - __popc(vn & above);
                        const int sd = __popc(vp & below) - __popc(vn & below);
                        again = c < 0 || c > 31 || (e > 0 && c_in - su <= n - n_in) ||
                                (e + 32 < W && 31 - c_in + sd <= n - n_in);
                    }
                    if (again) {
                        here = false;
                        if (m == m0 && c_in == q - e) { /* nor from a window around the path */
                            walking = false;
                            state = ST_OVERFLOW;
                        }
                        c = c_in;
                        hb = hb_in;
                        run = run_in;
                        n = n_in;
                    } else if (n > limit) {
                        here = walking = false;
                        state = past;
                    } else if (hb == 0) {
                        if (m == 0) {
                            /* the rows left are deleted */
                            here = walking = false;
                            const int left = c + e - b;
                            state = left < 0 ? ST_BADWALK : n + left > limit ? past : ST_DONE;
                            for (int v = state == ST_DONE ? left : 0; v > 0; --v) {
                                ev[n++] = 4u * (uint32_t)run + (uint32_t)kOpDel;
                                run = 0;
                            }
                        } else {
                            --m;
                            hb = 32;
                            c_in = c;
                            hb_in = hb;
                            run_in = run;
                            n_in = n;
                            here = m0 - m < kTileBlocks && c >= lo && c <= hi;
                        }
                    }
                }
                q = c + e;
            }
        }
        if (warp == 0) {
            if (state == ST_DONE && A.max_distance > 0 && n > A.max_distance) state = ST_OVERMAX;
            s_state[lane] = state;
            s_n[lane] = n;
            s_lead[lane] = run;
        }
        __syncthreads();
        /* CIGARs and results, a pair per warp */
        for (int p = warp; p < npair; p += kTileWarps) {
            const int st = s_state[p], nev = s_n[p];
            if (st == ST_IDLE) continue;
            const uint32_t pi = s_pi[p], cap = A.cigar_stride;
            if (st == ST_DONE) {
                const uint32_t len = store_events(slab + S.events + (size_t)p * S.ne, nev, s_lead[p],
                                                  A.cigar + (size_t)pi * cap, cap, lane);
                if (lane == 0) {
                    A.dist[pi] = nev;
                    if (A.status) A.status[pi] = len > cap ? (uint8_t)WFE_PAIR_CIGAR_TRUNCATED : (uint8_t)WFE_PAIR_OK;
                }
            } else if (lane == 0) {
                finish_unaligned(A, pi, st);
            }
        }
        __syncthreads();
    }
    chain_next(A);
}

/* ------------------------------------------------------------------------ */
/* Distance bounds for the CTA-per-pair tiers, one warp per pair.  The warp
 * runs the recurrence of the tiers restricted to a band of 32 diagonals
 * (lane l: diagonal b + l) that follows the cell furthest along its
 * antidiagonal (largest min(h, t_len) + min(v, p_len): offsets the
 * recurrence carries past a sequence's end count that end, so that the band
 * turns towards the target diagonal once one sequence is consumed): one
 * score step after it is seen the band moves one
 * diagonal towards that cell when it lies outside lanes 15-16.  Cells
 * outside the band count as the -1 sentinel, and a cell whose offset would
 * put its pattern position below 0 is dropped.  Every offset the band
 * computes is reached by some path of cost d and is at most the full
 * recurrence's offset (the three-way maximum and the extend are both
 * monotone), so the first step at which the band's cell (d, kt) reaches the
 * end is an upper bound on the edit distance: bound[pi] is that step, or -1
 * if the band has not reached it after max(p_len, t_len) + 1 steps.  On the
 * synthetic workloads the bound equals the distance for all but a handful
 * of pairs; the long tiers then compute only the target's cone (about half
 * of the cells), and a bound that is not one costs a second pass, never a
 * wrong result.  Each warp keeps its pair as plain packed words (16 bases
 * per 32-bit word, src/kernels.cu:313-394) in shared memory, followed by
 * zero words. */

/* 16-base window of plain packed words starting at base v (words w and
 * w + 1 of v's word w) */
__device__ __forceinline__ uint32_t window_words(const uint32_t* W, int v)
{
    const int w = v >> 4;
    return __funnelshift_l(W[w + 1], W[w], (uint32_t)(v & 15) << 1);
}

/* extend_lane over plain packed words */
__device__ __forceinline__ int extend_words(const uint32_t* P, const uint32_t* T, int plen, int tlen, int k, int off)
{
    int v = off - k, h = off;
    while ((unsigned)v < (unsigned)plen && (unsigned)h < (unsigned)tlen) {
        const uint32_t x = window_words(P, v) ^ window_words(T, h);
        int n = __clz(x) >> 1;
        n = min(n, min(plen - v, tlen - h));
        v += n;
        h += n;
        if (n < 16) break;
    }
    return h;
}

/* words per sequence in the bound kernel's shared memory: the packed words
 * and at least one zero word after them, rounded to 16 bytes */
__host__ __device__ __forceinline__ uint32_t bound_words(uint32_t seq_words) { return (seq_words + 4u) & ~3u; }

__device__ __forceinline__ void route_by_bound(const AlignLaunch& A, uint32_t pi, int bound, int need, uint32_t count)
{
    const LongClasses& C = A.chain.cls;
    const int top = C.shape[C.n - 1].dlim;
    if (bound > top && need > top && A.retry) {
        /* past tier 5 (with no cap below its limit): straight on */
        A.retry[atomicAdd(A.retry_count, 1u)] = pi;
        if (A.passed_total) atomicAdd(A.passed_total, 1ull);
        return;
    }
    int c = 0, below = 0;
    while (c + 1 < C.n && (C.shape[c].dlim < need || (!A.bulk && !class_by_cta(C.shape[c].dlim, count)))) {
        if (class_by_cta(C.shape[c].dlim, count)) below = C.shape[c].dlim;
        ++c;
    }
    if (A.bulk || 2 * need >= below + C.shape[c].dlim)
        C.list[c][atomicAdd(C.counts + c, 1u)] = pi;
    else
        C.list[c][C.cap - 1u - atomicAdd(C.low_counts + c, 1u)] = pi;
}

__device__ __forceinline__ void bound_body(const AlignLaunch& A, uint32_t seq_words)
{
    extern __shared__ __align__(16) unsigned char smem[];
    /* tier 5 with classes: route every pair to a class, then start them */
    const bool route = A.tier == 5 && A.chain.cls.n > 0;
    constexpr int kW = kLongThreads / 32;
    constexpr int kHalf = 15;
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
    const uint32_t bw = bound_words(seq_words);
    uint32_t* WP = reinterpret_cast<uint32_t*>(smem) + (size_t)warp * 2u * bw;
    uint32_t* WT = WP + bw;
    const uint32_t count = A.work_count ? min(*A.work_count, A.n_work) : A.n_work;
    for (uint32_t item = blockIdx.x * kW + (uint32_t)warp; item < count; item += gridDim.x * kW) {
        const uint32_t pi = A.work ? A.work[item] : item;
        const PairRef pr = get_pair(A.L, pi);
        const uint32_t mx = max(pr.plen, pr.tlen);
        int bound = -1;
        int need = INT_MAX; /* steps the pair's class must hold */
        if (pr.in_range && mx <= A.max_len && mx <= 16u * seq_words) {
            const int plen = (int)pr.plen, tlen = (int)pr.tlen, kt = tlen - plen;
            /* words 0..bw-1 of each sequence: packed_word gives 0 past the end */
            for (uint32_t w0 = 0; w0 < bw; w0 += 32u) {
                const uint32_t wp = packed_word(pr.p, pr.plen, w0, lane);
                const uint32_t wt = packed_word(pr.t, pr.tlen, w0, lane);
                if (w0 + (uint32_t)lane < bw) {
                    WP[w0 + lane] = wp;
                    WT[w0 + lane] = wt;
                }
            }
            __syncwarp();
            int b = -kHalf;
            int O = lane == kHalf ? extend_words(WP, WT, plen, tlen, 0, 0) : -1;
            if (__ballot_sync(kFull, lane == kHalf && kt == 0 && O == tlen)) bound = 0;
            const int limit = (int)mx + 1;
            int delta_next = 0;
            for (int d = 1; bound < 0 && d <= limit; ++d) {
                /* The band's leader after step d-1 -- the cell that has
                 * consumed the most bases of both sequences (offsets past an
                 * end count the end) -- moves the band of step d+1: the
                 * reduction then runs beside step d instead of before it. */
                const int delta = delta_next;
                const int prog = O >= 0 ? min(O, tlen) + min(O - (b + lane), plen) : INT_MIN;
                const int best = __reduce_max_sync(kFull, prog);
                const int lead = __ffs((int)__ballot_sync(kFull, prog == best)) - 1 - delta;
                delta_next = (lead > kHalf + 1) - (lead < kHalf);
                b += delta;
                const int k = b + lane;
                /* diagonals k+1, k, k-1 of step d-1 were on lanes s+1, s, s-1 */
                const int s = lane + delta;
                int up = __shfl_sync(kFull, O, (s + 1) & 31);
                int self = __shfl_sync(kFull, O, s & 31);
                int dn = __shfl_sync(kFull, O, (s - 1) & 31);
                if ((unsigned)(s + 1) > 31u) up = -1;
                if ((unsigned)s > 31u) self = -1;
                if ((unsigned)(s - 1) > 31u) dn = -1;
                int N = -1;
                if (k >= -d && k <= d) {
                    const int off = piggyback_max(up, self, dn) >> 2;
                    if (off >= k) N = extend_words(WP, WT, plen, tlen, k, off);
                }
                O = N;
                if (__ballot_sync(kFull, k == kt && N == tlen)) bound = d;
            }
            if (bound >= 0) need = max(bound, abs(kt));
            if (A.max_distance > 0) need = min(need, A.max_distance);
        }
        if (lane == 0) {
            A.bound[pi] = bound;
            if (route) {
                route_by_bound(A, pi, bound, need, count);
            }
        }
        __syncwarp();
    }
    if (route) chain_next(A);
}

/* Launched from the host and from the device (a chain entering tier 5): a
 * bound on the registers for 6 resident CTAs per SM, no launch bounds (see
 * tier_kernel). */
__global__ void __maxnreg__(40) bound_kernel(const __grid_constant__ AlignLaunch A, uint32_t seq_words, uint32_t /* unused */)
{
    bound_body(A, seq_words);
}

/* Tier 5's list in order of length, longest first (kOrderBins bins of equal
 * width), for the scan and the classes that it fills: the pairs of a warp then
 * end together, and the longest do not come last.  Two launches of a few
 * microseconds: the bins' counts, then, unless the plan chooses a kernel that
 * does not want the order, every pair to its place. */
__device__ __forceinline__ int order_bin(const AlignLaunch& A, uint32_t item, uint32_t& pi)
{
    pi = A.work ? A.work[item] : item;
    const PairRef pr = get_pair(A.L, pi);
    const uint32_t len = min(max(pr.plen, pr.tlen), A.max_len);
    return kOrderBins - 1 - (int)((uint64_t)len * kOrderBins / ((uint64_t)A.max_len + 1u));
}

/* Adds the items of a CTA's share to bins, one atomic per bin and warp. */
__device__ __forceinline__ void order_tally(const AlignLaunch& A, uint32_t count, uint32_t* bins, uint32_t blk,
                                            uint32_t blks)
{
    const int lane = (int)(threadIdx.x & 31u);
    const uint32_t end = (count + 31u) & ~31u; /* whole warps iterate together */
    for (uint32_t i = blk * kOrderBins + threadIdx.x; i < end; i += blks * kOrderBins) {
        uint32_t pi;
        const int b = i < count ? order_bin(A, i, pi) : -1;
        const unsigned same = __match_any_sync(kFull, b);
        if (b >= 0 && lane == __ffs((int)same) - 1) atomicAdd(&bins[b], (uint32_t)__popc(same));
    }
}

/* The bins' counts, by CTA blk of `blks`. */
__device__ __forceinline__ void order_count(const AlignLaunch& A, uint32_t count, uint32_t blk, uint32_t blks)
{
    __shared__ uint32_t bins[kOrderBins];
    bins[threadIdx.x] = 0u;
    __syncthreads();
    order_tally(A, count, bins, blk, blks);
    __syncthreads();
    if (bins[threadIdx.x]) atomicAdd(A.chain.cls.order_count + threadIdx.x, bins[threadIdx.x]);
}

__global__ void __launch_bounds__(kOrderBins) order_count_kernel(const __grid_constant__ AlignLaunch A)
{
    order_count(A, A.work_count ? min(*A.work_count, A.n_work) : A.n_work, blockIdx.x, gridDim.x);
}

/* The first kernel of a list, from a sample of it (plan_choice), by the first
 * kPlanCtas CTAs, one pair per thread: the distance of the first
 * kPredictPrefix bases in a band of 32 diagonals, scaled to the length.  The
 * other CTAs count the bins of the order that the scan wants, meanwhile.  The
 * last of the first few starts what it chose, on the device, but for the
 * scan, which follows in the stream, and whose launches see the choice in
 * words[kPlanSums - 1].  (Batches of 20,000 pairs of 1,000 bases
 * at 10%: 190 us each without a plan, 192 with it, and 211 with every kernel
 * launched to see whether it is chosen.) */
constexpr uint32_t kPlanCtas = kPlanSample / kOrderBins;
__global__ void __launch_bounds__(kOrderBins) plan_kernel(const __grid_constant__ AlignLaunch A, uint32_t* words)
{
    const uint32_t count = A.work_count ? min(*A.work_count, A.n_work) : A.n_work;
    float* const sums = reinterpret_cast<float*>(words);
    const auto choose = [&](int mode) {
        words[kPlanSums - 1] = (uint32_t)mode;
        if (A.plan_tiers) {
            const int tier = mode == kPlanBand ? 0 : mode == kPlanRegister ? 1 : 5;
            if (A.entered) atomicAdd(A.entered + tier, (unsigned long long)count);
            if (mode == kPlanBulk && A.chain.launched) atomicAdd(A.chain.launched + 5, 1ull);
        }
        if (mode == kPlanBand) {
            const TierShape& b = A.chain.shape[0];
            tail_launch(band_kernel<false>, A, 0, max(1, min(b.grid, (int)((count + 31u) / 32u))), 32, b.smem, true,
                        b.seq_words, b.smem / 4u, 0, true);
        } else if (mode == kPlanRegister) {
            launch_on_device<T1>(A, 1, count, true);
        } else if (mode == kPlanCta) {
            launch_bound_on_device(A, count, true);
        }
    };
    if (count < (A.plan_tiers == kPlanFrom1 ? kPlanFrom1Min : kScanMin)) {
        /* an empty list (a bucket that no pair of the batch falls in) starts nothing */
        if (count > 0u && blockIdx.x == 0 && threadIdx.x == 0) choose(A.plan_tiers == kPlanFrom1 ? kPlanRegister : kPlanCta);
        return;
    }
    if (blockIdx.x >= kPlanCtas) {
        order_count(A, count, blockIdx.x - kPlanCtas, gridDim.x - kPlanCtas);
        return;
    }
    const uint32_t item = (uint32_t)((uint64_t)(blockIdx.x * kOrderBins + threadIdx.x) * count / kPlanSample);
    const PairRef pr = get_pair(A.L, A.work ? A.work[item] : item);
    float c = 0.f, len = 0.f, d = 0.f, u = 0.f;
    if (pr.in_range && max(pr.plen, pr.tlen) <= A.max_len) {
        constexpr int kWords = kPredictPrefix / 32;
        const uint32_t lp = min(pr.plen, (uint32_t)kPredictPrefix), lt = min(pr.tlen, (uint32_t)kPredictPrefix);
        uint32_t p0[kWords + 1], p1[kWords + 1], t0[kWords + 1], t1[kWords + 1];
        const auto load = [](const char* s, uint32_t n, uint32_t(&lo)[kWords + 1], uint32_t(&hi)[kWords + 1]) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(s);
            const uint32_t sh = (uint32_t)(a & 15u);
            const uint4* base = reinterpret_cast<const uint4*>(a - sh);
            const int nblk = n ? (int)((sh + n + 15u) >> 4) : 0;
            uint32_t x[2 * kWords + 1];
#pragma unroll
            for (int i = 0; i <= 2 * kWords; ++i)
                x[i] = planes16(i < nblk ? __ldg(base + i) : make_uint4(0u, 0u, 0u, 0u));
#pragma unroll
            for (int w = 0; w < kWords; ++w) planes32(x[2 * w], x[2 * w + 1], x[2 * w + 2], sh, lo[w], hi[w]);
            lo[kWords] = hi[kWords] = 0u;
        };
        load(pr.p, lp, p0, p1);
        load(pr.t, lt, t0, t1);
        const int kt = (int)lt - (int)lp, wide = abs(kt);
        int D = wide;
        if (wide <= kBandDistance) {
            const int b = kBandDistance + min(0, kt) - (kBandDistance - wide) / 2, it = b - kt;
            uint32_t vp = ~0u << b, vn = ~vp, l0 = 0u, l1 = 0u;
#pragma unroll 1
            for (int m = 0; m < kWords; ++m) {
                const uint32_t a0 = __funnelshift_l(l0, p0[0], (uint32_t)b), e0 = __funnelshift_l(p0[0], p0[1], (uint32_t)b);
                const uint32_t a1 = __funnelshift_l(l1, p1[0], (uint32_t)b), e1 = __funnelshift_l(p1[0], p1[1], (uint32_t)b);
                uint32_t on = 0;
#pragma unroll 8
                for (int j = 0; j < 32; ++j) {
                    const uint32_t x = __funnelshift_r(a0, e0, (uint32_t)j) ^ bit_mask(t0[0], j);
                    const uint32_t eq = ~(x | (__funnelshift_r(a1, e1, (uint32_t)j) ^ bit_mask(t1[0], j)));
                    on = __funnelshift_r(on, band_column(eq, vp, vn) >> it, 1u);
                }
                D += __popc(~on & low_bits(min(32, max(0, (int)lt - 32 * m))));
                l0 = p0[0];
                l1 = p1[0];
#pragma unroll
                for (int i = 0; i < kWords; ++i) {
                    p0[i] = p0[i + 1];
                    p1[i] = p1[i + 1];
                    t0[i] = t0[i + 1];
                    t1[i] = t1[i + 1];
                }
            }
        }
        c = 1.f;
        len = (float)max(pr.plen, pr.tlen);
        d = fmaxf((float)D * fmaxf(1.f, len / (float)kPredictPrefix), fabsf((float)pr.tlen - (float)pr.plen));
        /* nanoseconds: the scan, then its walk, or the class's band and walk */
        u = len * (d <= 60.f ? 2.95f : 2.45f + 0.78f * (d / 32.f + 2.5f)) / 444.f;
    }
    float v[5] = {c, len, d, d * d, u};
#pragma unroll
    for (int i = 0; i < 5; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(kFull, v[i], o);
        if ((threadIdx.x & 31u) == 0u) atomicAdd(sums + i, v[i]);
    }
    if ((threadIdx.x & 31u) == 0u) {
        __threadfence();
        if (atomicAdd(words + kPlanSums - 2, 1u) + 1u == kPlanSample / 32u) {
            __threadfence();
            choose(plan_choice(A, count, sums));
        }
    }
}

__global__ void __launch_bounds__(kOrderBins) order_place_kernel(const __grid_constant__ AlignLaunch A)
{
    __shared__ uint32_t start[kOrderBins], mine[kOrderBins], sums[kOrderBins / 32];
    const uint32_t count = A.work_count ? min(*A.work_count, A.n_work) : A.n_work;
    if (!planned(A)) return;
    const int t = (int)threadIdx.x, lane = t & 31;
    /* exclusive prefix of the bins */
    const uint32_t c = A.chain.cls.order_count[t];
    uint32_t x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sums[t >> 5] = x;
    mine[t] = 0u;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < (t >> 5); ++w) before += sums[w];
    const uint32_t first = before + x - c;
    order_tally(A, count, mine, blockIdx.x, gridDim.x);
    __syncthreads();
    start[t] = first + (mine[t] ? atomicAdd(A.chain.cls.order_next + t, mine[t]) : 0u);
    __syncthreads();
    /* neighbours of one bin stay neighbours, a warp at a time: their bytes lie together */
    const uint32_t end = (count + 31u) & ~31u;
    for (uint32_t i = blockIdx.x * kOrderBins + threadIdx.x; i < end; i += gridDim.x * kOrderBins) {
        uint32_t pi = 0;
        const int b = i < count ? order_bin(A, i, pi) : -1;
        const unsigned same = __match_any_sync(kFull, b);
        const int leader = __ffs((int)same) - 1;
        uint32_t at = 0;
        if (b >= 0 && lane == leader) at = atomicAdd(&start[b], (uint32_t)__popc(same));
        at = __shfl_sync(kFull, at, leader) + (uint32_t)__popc(same & ((1u << lane) - 1u));
        if (b >= 0) A.chain.cls.order[at] = pi;
    }
}

const TierInfo kTiers[kNumTiers] = {
    {kBandDistance, 32},
    {T1::DCAP, kWarps},
    {T2::DCAP, kWarps},
    {T3::DCAP, kWarps},
    {T4::DCAP, kWarps},
    {kLongSmemDistance, 1},
    {0x7fffffff, 1},
};

template <class T>
TierShape shape_of(uint32_t max_len, uint32_t cigar_stride, int sm_count)
{
    TierShape sh{};
    const size_t smem = cta_smem_bytes<T>(max_len, cigar_stride);
    if (smem > 227u * 1024u) return sh;
    const void* fn = (const void*)tier_kernel<T>;
    if (allow_smem(fn, smem) != cudaSuccess)
        return sh;
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, kThreads, smem) != cudaSuccess)
        return sh;
    sh.grid = std::max(1, nb) * sm_count;
    sh.smem = (uint32_t)smem;
    sh.seq_words = seq_words_for(max_len);
    sh.gbytes = (uint32_t)warp_smem_bytes<T>(max_len, cigar_stride);
    if (!T::SMEM_OPS) {
        sh.ops_warp_bytes = (uint32_t)T::store_bytes(max_len);
        sh.ops_rows = T::store_rows(max_len);
    }
    return sh;
}

template <class T>
cudaError_t launch(const AlignLaunch& a, int grid, cudaStream_t s)
{
    const uint32_t sw = seq_words_for(a.max_len);
    const size_t gb = warp_smem_bytes<T>(a.max_len, a.cigar_stride);
    const size_t smem = cta_smem_bytes<T>(a.max_len, a.cigar_stride);
    if (smem > 227u * 1024u) return cudaErrorInvalidValue;
    if (!T::SMEM_OPS) {
        const TierShape& tsh = a.chain.shape[a.tier];
        if (tsh.ops_warp_bytes == 0 || tsh.ops_rows <= 0 ||
            a.ops_scratch_bytes < (size_t)tsh.ops_warp_bytes * (size_t)grid * kWarps)
            return cudaErrorInvalidValue;
    }
    cudaError_t e = allow_smem((const void*)tier_kernel<T>, smem);
    if (e != cudaSuccess) return e;
    tier_kernel<T><<<grid, kThreads, smem, s>>>(a, sw, (uint32_t)gb);
    return cudaGetLastError();
}

TierShape band_shape(uint32_t max_len, int sm_count)
{
    TierShape sh{};
    const size_t smem = 4u * (size_t)band_smem_words(max_len);
    if (smem > 227u * 1024u || allow_smem((const void*)band_kernel<false>, smem) != cudaSuccess) return sh;
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, band_kernel<false>, 32, smem) != cudaSuccess) return sh;
    sh.grid = std::max(1, nb) * sm_count;
    sh.smem = (uint32_t)smem;
    sh.seq_words = std::max(1u, band_words(max_len));
    return sh;
}

cudaError_t launch_band(const AlignLaunch& a, int grid, cudaStream_t s)
{
    const size_t smem = 4u * (size_t)band_smem_words(a.max_len);
    if (smem > 227u * 1024u) return cudaErrorInvalidValue;
    const cudaError_t e = allow_smem((const void*)band_kernel<false>, smem);
    if (e != cudaSuccess) return e;
    band_kernel<false><<<grid, 32, smem, s>>>(a, std::max(1u, band_words(a.max_len)), (uint32_t)(smem / 4u));
    return cudaGetLastError();
}

/* ------------------------------------------------------------------------ */
/* Routing: one thread per pair.  The length bucket is the first whose
 * max_len holds max(p_len, t_len).  The tier is the bucket's first tier, or,
 * with predictions, the first tier whose distance limit covers the
 * prediction: the prefix distance scaled by max length / prefix length,
 * plus 25 % and 2, up to tier 5 (a prediction only chooses where a pair
 * starts; a pair above its tier's limit still moves up).  Appends are warp-aggregated: one
 * atomic per (bucket, tier) present in the warp. */
__global__ void __launch_bounds__(256) classify_kernel(Layout L, uint32_t n, Buckets B)
{
    const int lane = (int)(threadIdx.x & 31u);
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t lim = (n + 31u) & ~31u; /* whole warps iterate together */
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < lim; i += stride) {
        int key = -1, bucket = -1;
        if (i < n) {
            const PairRef pr = get_pair(L, i);
            const uint32_t len = max(pr.plen, pr.tlen);
            int b = B.n - 1;
            for (int j = 0; j < B.n; ++j)
                if (len <= B.max_len[j]) { b = j; break; }
            int t = B.first_tier[b];
            if (B.pred && len > 0) {
                const uint32_t pref = min(max(pr.plen, pr.tlen), (uint32_t)kPredictPrefix);
                const uint32_t pd = B.pred[i];
                if (pd != 0xffff) {
                    const float scale = (float)len / (float)max(pref, 1u);
                    const float est = ((float)pd + 1.0f) * scale * 1.25f + 2.0f;
                    /* never past tier 5: the global-wavefront tier only
                     * takes pairs that tier 5 hands on */
                    const int top = min(B.last_tier[b], 5);
                    while (t < top && (float)B.dcap[t] < est) ++t;
                }
            }
            key = (t == 5 && B.tier5_to >= 0 ? B.tier5_to : B.to[b]) * kListsPerBucket + t;
            bucket = b;
        }
        const unsigned same = __match_any_sync(kFull, key);
        const int leader = __ffs((int)same) - 1;
        uint32_t base = 0;
        if (key >= 0 && lane == leader) {
            const int b = key / kListsPerBucket, t = key % kListsPerBucket;
            base = atomicAdd(B.counts + (size_t)b * B.count_stride + t, (uint32_t)__popc(same));
        }
        const unsigned alike = __match_any_sync(kFull, bucket);
        if (bucket >= 0 && lane == __ffs((int)alike) - 1)
            atomicAdd(B.entered + B.entered_tier[bucket], (unsigned long long)__popc(alike));
        base = __shfl_sync(kFull, base, leader);
        if (key >= 0) {
            const uint32_t rank = (uint32_t)__popc(same & ((1u << lane) - 1u));
            B.lists[(size_t)key * B.stride + base + rank] = i;
        }
    }
}

/* ------------------------------------------------------------------------ */
/* Standalone packer (src/kernels.cu:313-394): one thread per kPackWords
 * output words.  Thread t writes words kPackWords*j .. kPackWords*j +
 * kPackWords-1 of sequence t / ceil(wps/kPackWords) (pattern of pair i at
 * 2i, text at 2i+1), j = t % ceil(wps/kPackWords), from the kPackWords+1
 * aligned 16-byte blocks that hold their bases, each packed once; the
 * threads of a sequence read its blocks and descriptor through L1, so the
 * ASCII is read from DRAM about once and the words are written with
 * coalesced stores.  For 2 n ceil(wps/kPackWords) < 2^32. */
constexpr int kPackWords = 4;
__global__ void __launch_bounds__(256)
pack_words_kernel(Layout L, uint32_t n, uint32_t* out, uint32_t wps)
{
    const uint32_t gps = (wps + kPackWords - 1u) / kPackWords;
    const uint32_t total = 2u * n * gps;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t sidx = t / gps, w0 = kPackWords * (t - sidx * gps);
        const PairRef pr = get_pair(L, sidx >> 1);
        const char* s = (sidx & 1u) ? pr.t : pr.p;
        const uint32_t len = (sidx & 1u) ? pr.tlen : pr.plen;
        const uint32_t nw = (len + 15u) >> 4;
        const uintptr_t a = reinterpret_cast<uintptr_t>(s);
        const uint32_t sh = (uint32_t)(a & 15u);
        const uint4* base = reinterpret_cast<const uint4*>(a - sh);
        const uint32_t nblk = (sh + len + 15u) >> 4;
        uint4 v[kPackWords + 1];
#pragma unroll
        for (int r = 0; r <= kPackWords; ++r) v[r] = w0 + r < nblk ? __ldg(base + w0 + r) : make_uint4(0u, 0u, 0u, 0u);
        uint32_t x[kPackWords + 1];
#pragma unroll
        for (int r = 0; r <= kPackWords; ++r) x[r] = pack16(v[r]);
        uint32_t* dst = out + (size_t)sidx * wps;
#pragma unroll
        for (int r = 0; r < kPackWords; ++r) {
            const uint32_t w = w0 + (uint32_t)r;
            if (w >= wps) break;
            uint32_t W = 0;
            if (w < nw) {
                W = sh ? __funnelshift_l(x[r + 1], x[r], 2u * sh) : x[r];
                const uint32_t rem = len - 16u * w;
                if (rem < 16u) W &= ~0u << (2u * (16u - rem));
            }
            dst[w] = W;
        }
    }
}

/* The same words, one warp per sequence: for outputs of 2^32 words or more. */
__global__ void __launch_bounds__(256)
pack_kernel(Layout L, uint32_t n, uint32_t* out, uint32_t wps)
{
    const int lane = (int)(threadIdx.x & 31u);
    const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarp = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t sidx = wid; sidx < 2u * n; sidx += nwarp) {
        const PairRef pr = get_pair(L, sidx >> 1);
        const char* s = (sidx & 1u) ? pr.t : pr.p;
        const uint32_t len = (sidx & 1u) ? pr.tlen : pr.plen;
        uint32_t* dst = out + (size_t)sidx * wps;
        const uint32_t nw = (len + 15u) >> 4;
        for (uint32_t w0 = 0; w0 < wps; w0 += 32u) {
            uint32_t W = 0;
            if (w0 < nw) W = packed_word(s, len, w0, lane);
            if (w0 + (uint32_t)lane < wps) dst[w0 + lane] = W;
        }
    }
}

/* ------------------------------------------------------------------------ */
/* CIGARs from 128-bit histories (src/kernels.cu:397-625): one pair per thread,
 * both sequences of a warp's 32 pairs as bit planes in shared memory.  A step
 * compares 32 bases, the next of them either after an operation or, if all
 * match, right after these.  The bytes go to the slot word by word as they
 * come.  Bound by the integer pipe (2,700 warp instructions for 32 pairs of
 * 150 bases, two thirds of them the steps) and, with 1.3 waves of warps, by
 * the latency of each wave's loads: with 80 registers, 24 warps an SM instead
 * of 32, 200,000 pairs whose inputs are not in L2 took 35 us instead of 33;
 * banks free of conflicts, CIGARs staged in shared memory and larger CTAs gave
 * nothing.  With
 * a group of four lanes per pair before, 200,000 pairs of 150 bases at 5%
 * took 78 us (now 25), of 250 bases at 10% 177 (73), 100,000 of 500 bases at
 * 1% 140 (81), 20,000 of 2,000 bases 341 (103), 30 of 100 bases 11 (9). */
constexpr int kWideSpanWords = 252; /* 16-byte blocks of a span: 8 pairs of 250 bases */
__host__ __device__ constexpr uint32_t history_smem_words(uint32_t nw, int span)
{
    return 4u * kPlaneRow * (nw + 1u) + 4u * (uint32_t)span_row(span);
}

template <int SPAN>
__global__ void __launch_bounds__(32, 32)
history_kernel(Layout L, uint32_t n, uint32_t max_len, const int32_t* dist, const uint64_t* hist, int8_t* cigar,
               uint32_t stride, uint8_t* status, uint32_t nw, uint32_t per_warp)
{
    const int lane = (int)threadIdx.x;
    const uint32_t pi = threadIdx.x < per_warp ? blockIdx.x * per_warp + threadIdx.x : n;
    const int plane = kPlaneRow * (int)(nw + 1u);
    PairRef pr{};
    uint64_t w0 = 0, w1 = 0;
    int D = 0, state = ST_IDLE;
    if (pi < n) {
        pr = get_pair(L, pi);
        D = dist[pi];
        state = max(pr.plen, pr.tlen) > max_len ? ST_TOOLONG : D < 0 || D > 63 ? ST_OVERMAX : ST_RUN;
        if (state == ST_RUN) {
            /* no operations past the distance */
            w0 = hist[2u * (size_t)pi] & (D < 32 ? (1ull << 2 * D) - 1ull : ~0ull);
            w1 = D > 32 ? hist[2u * (size_t)pi + 1u] & ((1ull << 2 * (D - 32)) - 1ull) : 0ull;
        }
    }
    const bool mine = state == ST_RUN;
    const int plen = mine ? (int)pr.plen : 0, tlen = mine ? (int)pr.tlen : 0;
    band_load<SPAN>(pr.p, (uint32_t)plen, pr.t, (uint32_t)tlen, band_smem + 4 * plane, band_smem,
                    (int)nw + 1, band_smem + 2 * plane, (int)nw + 1, lane);
    if (pi >= n) return;

    const uint32_t* const P = band_smem + lane;
    const uint32_t* const T = P + 2 * plane;
    int8_t* const dst = cigar + (size_t)pi * stride;
    const bool aligned = (stride & 3u) == 0u && (reinterpret_cast<uintptr_t>(cigar) & 3u) == 0u;
    uint32_t len = 0;
    uint64_t acc = 0; /* the len % 4 bytes that are not written yet */
    /* bytes [len & ~3, end) of the slot */
    const auto put = [&](uint32_t end) {
        const uint32_t at = len & ~3u;
        if (aligned) {
            if (at < min(end, stride)) *reinterpret_cast<uint32_t*>(dst + at) = (uint32_t)acc;
        } else {
            for (uint32_t j = 0; j < 4u && at + j < min(end, stride); ++j) dst[at + j] = (int8_t)(acc >> (8u * j));
        }
    };
    const auto push = [&](uint32_t two, uint32_t k) { /* up to two bytes */
        acc |= (uint64_t)two << (8u * (len & 3u));
        if ((len & 3u) + k >= 4u) {
            put(len + 4u);
            acc >>= 32;
        }
        len += k;
    };
    uint32_t o0 = (uint32_t)w0, o1 = (uint32_t)(w0 >> 32), o2 = (uint32_t)w1, o3 = (uint32_t)(w1 >> 32);
    int v = 0, h = 0, d = 0;
    uint32_t run = 0;
    /* every lane goes through the whole of a step, whether its run of matches
     * ends in it or not: the warp takes as many as its longest pair */
    while (state == ST_RUN) {
        const int rem = min(plen - v, tlen - h);
        uint32_t x = 1u;
        if (rem > 0) {
            const uint32_t* p = P + kPlaneRow * (v >> 5);
            const uint32_t* t = T + kPlaneRow * (h >> 5);
            x = __funnelshift_r(p[0], p[kPlaneRow], (uint32_t)v) ^ __funnelshift_r(t[0], t[kPlaneRow], (uint32_t)h);
            x |= __funnelshift_r(p[plane], p[plane + kPlaneRow], (uint32_t)v) ^
                 __funnelshift_r(t[plane], t[plane + kPlaneRow], (uint32_t)h);
            if (rem < 32) x |= 1u << rem;
        }
        const uint32_t k = x ? (uint32_t)__ffs((int)x) - 1u : 32u;
        const bool ends = x != 0u;
        run += k;
        if (run >= 127u && ends)
            for (; run >= 127u; run -= 127u) push(256u - 127u, 1u);
        const uint32_t op = ends ? o0 & 3u : 0u;
        const uint32_t letter = (0x44584900u >> (8u * op)) & 0xffu; /* I, X, D */
        const uint32_t r = ends ? run : 0u;
        push(r ? (256u - r) | letter << 8 : letter, (r ? 1u : 0u) + (op ? 1u : 0u));
        v += (int)(k + (op >> 1));
        h += (int)(k + ((op >> 1) ^ (op & 1u)));
        if (ends) {
            run = 0;
            o0 = __funnelshift_r(o0, o1, 2u);
            o1 = __funnelshift_r(o1, o2, 2u);
            o2 = __funnelshift_r(o2, o3, 2u);
            o3 >>= 2;
            if (op == 0u) state = ST_DONE; /* the end, or a code that is no operation */
            else ++d;
        }
    }
    const bool bad = d < D;
    if (stride && state == ST_DONE) {
        if (len < stride || (len & 3u)) put(len + 1u); /* with the terminator, when it fits */
    } else if (stride) {
        dst[0] = 0;
    }
    if (status)
        status[pi] = state == ST_TOOLONG   ? (uint8_t)WFE_PAIR_TOO_LONG
                     : state == ST_OVERMAX ? (uint8_t)WFE_PAIR_OVER_MAX_DISTANCE
                     : bad                 ? (uint8_t)WFE_PAIR_BAD_HISTORY
                     : len > stride        ? (uint8_t)WFE_PAIR_CIGAR_TRUNCATED
                                           : (uint8_t)WFE_PAIR_OK;
}

}  // namespace

const TierInfo& tier_info(int t) { return kTiers[t]; }

size_t tier_scratch_bytes(int tier, int grid, uint32_t max_len)
{
    switch (tier) {
    case 2: return T2::store_bytes(max_len) * (size_t)grid * kWarps;
    case 3: return T3::store_bytes(max_len) * (size_t)grid * kWarps;
    case 4: return T4::store_bytes(max_len) * (size_t)grid * kWarps;
    default: return 0;
    }
}

uint64_t long_slab_bytes(int dlim, bool global_wavefront)
{
    uint64_t b = long_row(dlim + 1) * 8u;              /* backtrace store */
    b += (uint64_t)((dlim + 16) & ~15);                 /* chain */
    b += 4u * (uint64_t)((dlim + 4) & ~3);              /* runs */
    if (global_wavefront) b += 8u * (uint64_t)(2 * dlim + 5); /* two wavefront buffers */
    return (b + 255u) & ~uint64_t(255);
}

namespace {

/* Shape of a CTA-per-pair launch of NT threads for sequences up to max_len
 * and distances up to dlim (global wavefront: GWF). */
template <bool GWF, int NT>
TierShape long_shape_for(uint32_t max_len, int dlim, int sm_count)
{
    TierShape sh{};
    const uint32_t sw = seq_words_for(max_len);
    const size_t smem = 16u * (size_t)sw + (GWF ? 0u : 8u * (size_t)(2 * dlim + 5));
    if (smem > 227u * 1024u) return sh;
    if (allow_smem((const void*)long_kernel<GWF, NT>, smem) != cudaSuccess)
        return sh;
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, long_kernel<GWF, NT>, NT, smem) != cudaSuccess)
        return sh;
    sh.grid = std::max(1, nb) * sm_count;
    sh.smem = (uint32_t)smem;
    sh.seq_words = sw;
    sh.dlim = dlim;
    sh.slab = long_slab_bytes(dlim, GWF);
    sh.threads = NT;
    return sh;
}

template <bool GWF>
TierShape long_shape_of(uint32_t max_len, int sm_count)
{
    const int dlim = GWF ? (int)max_len : (int)std::min<uint32_t>(max_len, kLongSmemDistance);
    return long_shape_for<GWF, kLongThreads>(max_len, dlim, sm_count);
}

template <bool GWF>
cudaError_t launch_long(const AlignLaunch& a, int grid, cudaStream_t s)
{
    const TierShape& sh = a.chain.shape[a.tier];
    if (!sh.scratch || sh.smem == 0) return cudaErrorInvalidValue;
    cudaError_t e = allow_smem((const void*)long_kernel<GWF, kLongThreads>, sh.smem);
    if (e != cudaSuccess) return e;
    long_kernel<GWF, kLongThreads><<<grid, kLongThreads, sh.smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace

namespace {

TierShape compute_tier_shape(int tier, uint32_t max_len, uint32_t cigar_stride, int sm_count)
{
    switch (tier) {
    case 0: return band_shape(max_len, sm_count);
    case 1: return shape_of<T1>(max_len, cigar_stride, sm_count);
    case 2: return shape_of<T2>(max_len, cigar_stride, sm_count);
    case 3: return shape_of<T3>(max_len, cigar_stride, sm_count);
    case 4: return shape_of<T4>(max_len, cigar_stride, sm_count);
    case 5: return long_shape_of<false>(max_len, sm_count);
    case 6: return max_len > (uint32_t)kLongSmemDistance ? long_shape_of<true>(max_len, sm_count) : TierShape{};
    default: return TierShape{};
    }
}

}  // namespace

/* Shapes depend only on the device and the arguments; each occupancy query
 * costs tens of microseconds the first time, and a context asks for every
 * tier's shape at creation and again for its first bucket, so results are
 * kept per device for the life of the process. */
TierShape tier_shape(int tier, uint32_t max_len, uint32_t cigar_stride, int sm_count)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return TierShape{};
    static std::mutex mu;
    static std::map<std::tuple<int, int, uint32_t, uint32_t, int>, TierShape> known;
    const auto key = std::make_tuple(dev, tier, max_len, cigar_stride, sm_count);
    std::lock_guard<std::mutex> lock(mu);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    const TierShape sh = compute_tier_shape(tier, max_len, cigar_stride, sm_count);
    known.emplace(key, sh);
    return sh;
}

/* cached per (device, max_len, SMs), as tier_shape */
TierShape bound_shape(uint32_t max_len, int sm_count)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return TierShape{};
    static std::mutex mu;
    static std::map<std::tuple<int, uint32_t, int>, TierShape> known;
    const auto key = std::make_tuple(dev, max_len, sm_count);
    std::lock_guard<std::mutex> lock(mu);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    TierShape sh{};
    const uint32_t sw = seq_words_for(max_len);
    const size_t smem = (size_t)(kLongThreads / 32) * 2u * bound_words(sw) * sizeof(uint32_t);
    int nb = 0;
    if (smem <= 227u * 1024u && allow_smem((const void*)bound_kernel, smem) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, bound_kernel, kLongThreads, smem) == cudaSuccess) {
        sh.grid = std::max(1, nb) * sm_count;
        sh.smem = (uint32_t)smem;
        sh.seq_words = sw;
        sh.threads = kLongThreads;
    }
    cudaGetLastError();
    known.emplace(key, sh);
    return sh;
}

namespace {
int order_grid(const AlignLaunch& a) { return (int)std::min<uint32_t>((a.n_work + 4u * kOrderBins - 1u) / (4u * kOrderBins), 4u * kSms); }
}  // namespace

cudaError_t launch_order(const AlignLaunch& a, cudaStream_t s)
{
    order_count_kernel<<<order_grid(a), kOrderBins, 0, s>>>(a);
    order_place_kernel<<<order_grid(a), kOrderBins, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_planned(const AlignLaunch& a, cudaStream_t s)
{
    if (a.chain.bound_shape.grid <= 0 || !a.bound || a.chain.cls.scan.grid <= 0) return cudaErrorInvalidValue;
    plan_kernel<<<order_grid(a) + (int)kPlanCtas, kOrderBins, 0, s>>>(a, const_cast<uint32_t*>(a.plan) - (kPlanSums - 1));
    AlignLaunch w = a;
    w.bulk = 1;
    order_place_kernel<<<order_grid(w), kOrderBins, 0, s>>>(w);
    w.work = w.chain.cls.order;
    wide_kernel<2, true><<<std::max(1, std::min(w.chain.cls.scan.grid, (int)((w.n_work + 31u) / 32u))), 32, 0, s>>>(w);
    return cudaGetLastError();
}

cudaError_t launch_bound(const AlignLaunch& a, cudaStream_t s, uint64_t* launches)
{
    const TierShape& sh = a.chain.bound_shape;
    if (sh.grid <= 0 || !a.bound || sh.seq_words != seq_words_for(a.max_len)) return cudaErrorInvalidValue;
    cudaError_t e = allow_smem((const void*)bound_kernel, sh.smem);
    if (e != cudaSuccess) return e;
    if (a.tier == 5 && a.chain.cls.n > 0 && a.chain.cls.scan.grid > 0 && a.n_work >= kScanMin) {
        *launches += 3;
        return launch_planned(a, s);
    }
    AlignLaunch w = a;
    w.plan = nullptr;
    const uint32_t per_cta = (uint32_t)sh.threads / 32u;
    const int grid = (int)std::min<uint64_t>((uint64_t)sh.grid, ((uint64_t)a.n_work + per_cta - 1) / per_cta);
    ++*launches;
    bound_kernel<<<std::max(grid, 1), sh.threads, sh.smem, s>>>(w, sh.seq_words, 0u);
    return cudaGetLastError();
}

namespace {

/* Launch shape of a wide kernel within the tier-5 scratch: as many warps as
 * fit both (grid 0: too few to be worth it). */
template <int NW, bool SCAN>
TierShape wide_shape(uint32_t max_len, int sm_count, uint64_t scratch_bytes)
{
    TierShape sh{};
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, wide_kernel<NW, SCAN>, 32, 0) != cudaSuccess) return sh;
    sh.slab = 4u * (uint64_t)wide_slab<NW>(max_len).words;
    const uint64_t grid = std::min<uint64_t>((uint64_t)std::max(nb, 0) * (uint64_t)sm_count, scratch_bytes / sh.slab);
    if (grid < (uint64_t)sm_count / 2u) return TierShape{};
    sh.grid = (int)grid;
    sh.threads = 32;
    sh.dlim = 32 * NW - 1;
    return sh;
}

/* Launch shape of the tile kernel, its slabs sized for the widest of the first n classes. */
TierShape tile_shape(uint32_t max_len, const int* dlim, int n, int sm_count, uint64_t scratch_bytes)
{
    TierShape sh{};
    int nb = 0;
    if (n < 1 || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, tile_kernel, kTileThreads, 0) != cudaSuccess)
        return sh;
    for (int c = 0; c < n; ++c) sh.slab = std::max<uint64_t>(sh.slab, 4u * tile_slab(max_len, dlim[c]).words);
    const uint64_t grid = std::min<uint64_t>((uint64_t)std::max(nb, 0) * (uint64_t)sm_count, scratch_bytes / sh.slab);
    if (grid < (uint64_t)sm_count / 2u) return TierShape{};
    sh.grid = (int)grid;
    sh.threads = kTileThreads;
    return sh;
}

LongClasses compute_long_classes(uint32_t max_len, int sm_count, uint64_t scratch_bytes)
{
    LongClasses C{};
    const int top = (int)std::min<uint32_t>(max_len, kLongSmemDistance);
    int lim[kLongClasses];
    int n = 0;
    for (int c = 0; c < kLongClasses - 1; ++c)
        if (kLongClassLimit[c] < top) lim[n++] = kLongClassLimit[c];
    lim[n++] = top;
    for (int c = 0; c < n; ++c) {
        TierShape sh = lim[c] <= kLongTinyDistance    ? long_shape_for<false, kLongTinyThreads>(max_len, lim[c], sm_count)
                     : lim[c] <= kLongSmallDistance ? long_shape_for<false, kLongSmallThreads>(max_len, lim[c], sm_count)
                                                    : long_shape_for<false, kLongThreads>(max_len, lim[c], sm_count);
        if (sh.grid <= 0) return LongClasses{};
        /* the class's slabs share tier 5's scratch: one class runs at a time */
        const uint64_t fit = sh.slab ? scratch_bytes / sh.slab : 0u;
        if (fit == 0) return LongClasses{};
        sh.grid = (int)std::min<uint64_t>((uint64_t)sh.grid, fit);
        C.shape[c] = sh;
    }
    C.n = n;
    C.scan = wide_shape<2, true>(max_len, sm_count, scratch_bytes);
    for (int c = 0; c + 1 < n; ++c) {
        C.wide[c] = lim[c] <= 127   ? wide_shape<4, false>(max_len, sm_count, scratch_bytes)
                    : lim[c] <= 255 ? wide_shape<8, false>(max_len, sm_count, scratch_bytes)
                    : lim[c] <= 511 ? wide_shape<16, false>(max_len, sm_count, scratch_bytes)
                    : lim[c] <= 1023 ? wide_shape<32, false>(max_len, sm_count, scratch_bytes) : TierShape{};
    }
    C.tile = tile_shape(max_len, lim, n - 1, sm_count, scratch_bytes);
    return C;
}

}  // namespace

/* cached per (device, max_len, SMs, scratch), as tier_shape */
LongClasses long_classes(uint32_t max_len, int sm_count, uint64_t scratch_bytes)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return LongClasses{};
    static std::mutex mu;
    static std::map<std::tuple<int, uint32_t, int, uint64_t>, LongClasses> known;
    const auto key = std::make_tuple(dev, max_len, sm_count, scratch_bytes);
    std::lock_guard<std::mutex> lock(mu);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    const LongClasses C = compute_long_classes(max_len, sm_count, scratch_bytes);
    cudaGetLastError();
    known.emplace(key, C);
    return C;
}

cudaError_t launch_tier(int tier, const AlignLaunch& a, int grid, cudaStream_t s)
{
    if (grid <= 0) return cudaErrorInvalidConfiguration;
    switch (tier) {
    case 0: return launch_band(a, grid, s);
    case 1: return launch<T1>(a, grid, s);
    case 2: return launch<T2>(a, grid, s);
    case 3: return launch<T3>(a, grid, s);
    case 4: return launch<T4>(a, grid, s);
    case 5: return launch_long<false>(a, grid, s);
    case 6: return launch_long<true>(a, grid, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_classify(const Layout& L, uint32_t n, const Buckets& B, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    const uint32_t blocks = std::min<uint32_t>((n + 255u) / 256u, 4096u);
    classify_kernel<<<blocks, 256, 0, s>>>(L, n, B);
    return cudaGetLastError();
}

cudaError_t launch_predict(const Layout& L, uint32_t n, uint32_t max_len, uint16_t* pred, int grid, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    const size_t smem = 4u * (size_t)band_smem_words((uint32_t)kPredictPrefix);
    cudaError_t e = allow_smem((const void*)band_kernel<true>, smem);
    if (e != cudaSuccess) return e;
    AlignLaunch a{};
    a.L = L;
    a.n_work = n;
    a.max_len = max_len;
    a.pred = pred;
    a.tier = 0;
    grid = std::max(1, std::min(grid, (int)((n + 31u) / 32u)));
    band_kernel<true><<<grid, 32, smem, s>>>(a, band_words((uint32_t)kPredictPrefix), (uint32_t)(smem / 4u));
    return cudaGetLastError();
}

cudaError_t launch_pack(const Layout& L, uint32_t n, uint32_t* words, uint32_t wps, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    const uint64_t total = 2ull * n * ((wps + kPackWords - 1u) / kPackWords);
    if (total < (1ull << 32)) {
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
                                                      cudaSuccess)
            return cudaErrorInvalidValue;
        /* 8 blocks of 256 per SM, each thread looping over words */
        const uint32_t blocks = (uint32_t)std::max<uint64_t>(
            1u, std::min<uint64_t>((total + 255u) / 256u, (uint64_t)sms * 8u));
        pack_words_kernel<<<blocks, 256, 0, s>>>(L, n, words, wps);
        return cudaGetLastError();
    }
    const uint32_t warps = 2u * n;
    const uint32_t blocks = std::min<uint32_t>((warps + 7u) / 8u, 65535u * 16u);
    pack_kernel<<<blocks, 256, 0, s>>>(L, n, words, wps);
    return cudaGetLastError();
}

cudaError_t launch_cigar_from_history(const Layout& L, uint32_t n, uint32_t max_len,
                                      const int32_t* dist, const uint64_t* hist, int8_t* cigar,
                                      uint32_t stride, uint8_t* status, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    /* long sequences and slots have always been refused together */
    if (16u * (size_t)seq_words_for(max_len) + 320u + round16(stride) > 227u * 32u) return cudaErrorInvalidValue;
    const uint32_t nw = std::max(1u, band_words(max_len));
    /* Few pairs: eight a warp, which read one span and take as many steps as the
     * longest of eight (4,000 pairs of 250 bases at 10% 20.9 -> 15.0 us, 2,000 of
     * 1,000 bases 45.7 -> 25.2; 16,384 of 150 bases 10.0 -> 13.1). */
    const uint32_t per_warp = n <= 8192u ? 8u : 32u;
    const auto launch_as = [&](auto kernel, int span) {
        const size_t smem = 4u * (size_t)history_smem_words(nw, span);
        const cudaError_t e = allow_smem((const void*)kernel, smem);
        if (e != cudaSuccess) return e;
        kernel<<<n / per_warp + (n % per_warp != 0u), 32, smem, s>>>(L, n, max_len, dist, hist, cigar, stride, status,
                                                                     nw, per_warp);
        return cudaGetLastError();
    };
    /* spans of 8 pairs that do not fit the narrower ones (250 bases: 40 us
     * against 52; 150 bases: 29 against 25) */
    const bool wide = max_len > (uint32_t)kSpanWords && max_len <= (uint32_t)kWideSpanWords;
    return wide ? launch_as(history_kernel<kWideSpanWords>, kWideSpanWords)
                : launch_as(history_kernel<kSpanWords>, kSpanWords);
}

}  // namespace wfe
