/*
 * wfe_band.cuh -- bit-parallel banded alignment, one pair per thread.
 *
 * The edit-distance matrix DP(v, h) (v pattern bases against h text bases)
 * is computed column by column over a band of diagonals k = h - v, a bit
 * per diagonal (Myers 1999; the diagonal form of Hyyro 2003).  Bit i of
 * column h is row v = h - b + i, where b is the highest diagonal of the band:
 * bit 0 is diagonal b, bit i diagonal b - i.  Per column, with VP/VN the
 * vertical differences of the previous column (+1 / -1) at the rows of this
 * one and Eq the matching rows:
 *   D0 = (((Eq & VP) + VP) ^ VP) | Eq | VN     DP(v,h) == DP(v-1,h-1)
 *   HP = VN | ~(D0 | VP),  HN = VP & D0         DP(v,h) - DP(v,h-1) = +1 / -1
 *   VP' = HN | ~((D0 >> 1) | HP),  VN' = (D0 >> 1) & HP
 * Rows v <= 0 are virtual, DP(v, h) = h - v: they satisfy the recurrence, so
 * column 0 needs only VP = rows v >= 1, VN = the others, and no row is
 * masked.  Rows past the pattern's end never reach the rows before it.
 *
 * A value of the band is never below the matrix's, and equals it on every
 * cell of every optimal path that stays in the band.  A path that leaves a
 * band of W diagonals holding 0 and kt (both ends of the alignment, centred)
 * costs at least W, so a banded distance of W - 1 or less is the edit
 * distance, and every optimal path lies in the band.
 *
 * The wavefront's CIGAR (furthest-reaching offsets, ties DEL > SUB > INS,
 * src/kernels.cu:136-171) is read back from the increments along the
 * diagonals.  Along diagonal k the matrix is monotone, and the furthest
 * offset F(s, k) that score s reaches is the last h with DP <= s on it: the
 * position of an increment (D0 bit 0).  A path cell is some F(s, k); its
 * source is the largest of F(s-1, k+1) (deletion), F(s-1, k) + 1 (mismatch)
 * and F(s-1, k-1) + 1 (insertion).  So the walk needs, per diagonal, the
 * increments as a bit string over the columns: D0 of 32 columns, transposed.
 * Scores on neighbouring diagonals are compared through the vertical
 * differences at the block's first column plus a population count each.
 */
#ifndef WFE_BAND_CUH
#define WFE_BAND_CUH

#include "wfe_device.cuh"

namespace wfe {

constexpr int kBandBits = 32;
constexpr int kBandDistance = kBandBits - 1; /* largest distance a band of 32 diagonals certifies */

/* Sixteen ASCII bytes -> their 2-bit codes as two bit planes, base i at bit
 * i (low code bits) and bit 16 + i (high code bits).  A multiply gathers the
 * four flags of a word, which sit 8 bits apart, into four consecutive bits:
 * the partial products never meet in one bit, so nothing carries. */
__device__ __forceinline__ uint32_t planes16(uint4 b)
{
    constexpr uint32_t M = 0x01020408u;
    const uint32_t a0 = ((b.x & 0x02020202u) * M) >> 25, a1 = ((b.y & 0x02020202u) * M) >> 25;
    const uint32_t a2 = ((b.z & 0x02020202u) * M) >> 25, a3 = ((b.w & 0x02020202u) * M) >> 25;
    const uint32_t c0 = ((b.x & 0x04040404u) * M) >> 26, c1 = ((b.y & 0x04040404u) * M) >> 26;
    const uint32_t c2 = ((b.z & 0x04040404u) * M) >> 26, c3 = ((b.w & 0x04040404u) * M) >> 26;
    const uint32_t lo = a0 + a1 * 16u + a2 * 256u + a3 * 4096u;
    const uint32_t hi = c0 + c1 * 16u + c2 * 256u + c3 * 4096u;
    return lo + hi * 65536u;
}

/* 32 bases of a sequence that starts sh bytes into a 16-byte block, from the
 * planes of the three blocks x0, x1, x2 that hold them */
__device__ __forceinline__ void planes32(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t sh, uint32_t& lo,
                                         uint32_t& hi)
{
    lo = __funnelshift_r(__byte_perm(x0, x1, 0x5410), x2 & 0xffffu, sh);
    hi = __funnelshift_r(__byte_perm(x0, x1, 0x7632), x2 >> 16, sh);
}

/* One column of a band of 32 diagonals; returns D0. */
__device__ __forceinline__ uint32_t band_column(uint32_t eq, uint32_t& vp, uint32_t& vn)
{
    const uint32_t d0 = (((eq & vp) + vp) ^ vp) | eq | vn;
    const uint32_t hp = vn | ~(d0 | vp);
    const uint32_t hn = vp & d0;
    const uint32_t x = d0 >> 1;
    vp = hn | ~(x | hp);
    vn = x & hp;
    return d0;
}

/* The same column, and the operation by which the wavefront's path leaves each
 * of its cells, going back (a match leaves by none): the first that fits of a
 * deletion (the row above has one less), a mismatch (the diagonal before has)
 * and an insertion (the column before has).  One of the two bits of the
 * operation codes, `high` or low; bit 0's deletion is not known here. */
__device__ __forceinline__ uint32_t band_column_ops(uint32_t eq, uint32_t& vp, uint32_t& vn, bool high)
{
    const uint32_t d0 = (((eq & vp) + vp) ^ vp) | eq | vn;
    const uint32_t hp = vn | ~(d0 | vp);
    const uint32_t hn = vp & d0;
    const uint32_t x = d0 >> 1;
    vp = hn | ~(x | hp);
    vn = x & hp;
    const uint32_t del = vp << 1;
    return high ? del | ~d0 : del | (d0 & hp);
}

/* all ones when bit j of w is set */
__device__ __forceinline__ uint32_t bit_mask(uint32_t w, int j)
{
    return (uint32_t)((int32_t)(w << (31 - j)) >> 31);
}

template <int S, int N>
__device__ __forceinline__ void transpose_step(uint32_t (&a)[N], uint32_t m)
{
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        const int k = ((i & ~(S - 1)) << 1) | (i & (S - 1));
        const uint32_t x = a[k], y = a[k + S];
        a[k] = (x & m) | ((y << S) & ~m);
        a[k + S] = ((x >> S) & m) | (y & ~m);
    }
}

/* Transpose a 32 x 32 bit matrix: bit j of a[i] <-> bit i of a[j]. */
__device__ __forceinline__ void transpose32(uint32_t (&a)[32])
{
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const uint32_t x = a[i], y = a[i + 16];
        a[i] = __byte_perm(x, y, 0x5410);
        a[i + 16] = __byte_perm(x, y, 0x7632);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int k = ((i & 8) << 1) | (i & 7);
        const uint32_t x = a[k], y = a[k + 8];
        a[k] = __byte_perm(x, y, 0x6240);
        a[k + 8] = __byte_perm(x, y, 0x7351);
    }
    transpose_step<4>(a, 0x0f0f0f0fu);
    transpose_step<2>(a, 0x33333333u);
    transpose_step<1>(a, 0x55555555u);
}

/* The same with only bits first .. first + 15 of every a[i], into 16 words:
 * bit i of out[r] is bit first + r of a[i]. */
__device__ __forceinline__ void transpose16(const uint32_t (&a)[32], int first, uint32_t (&out)[16])
{
#pragma unroll
    for (int i = 0; i < 16; ++i) out[i] = __byte_perm(a[i] >> first, a[i + 16] >> first, 0x5410);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t x = out[i], y = out[i + 8];
        out[i] = __byte_perm(x, y, 0x6240);
        out[i + 8] = __byte_perm(x, y, 0x7351);
    }
    transpose_step<4>(out, 0x0f0f0f0fu);
    transpose_step<2>(out, 0x33333333u);
    transpose_step<1>(out, 0x55555555u);
}

/* The lowest n bits, n in [0, 32]. */
__device__ __forceinline__ uint32_t low_bits(int n) { return __funnelshift_rc(~0u, 0u, 32u - (uint32_t)n); }

/* CIGAR bytes written from the last to the first: words of four bytes, the
 * first pushed byte highest, to words top-1, top-2, ... of a lane's column
 * of `buf` (stride words apart).  The string then lies in order at the end
 * of the column. */
struct BackBytes {
    uint32_t* buf; /* the lane's column */
    uint32_t acc;
    int n;         /* bytes pushed */
    int top;       /* words in the column */
    __device__ __forceinline__ void push(uint32_t byte, int stride)
    {
        acc = acc * 256u + (byte & 0xffu);
        ++n;
        if ((n & 3) == 0) {
            const int w = top - (n >> 2);
            if (w >= 0) buf[w * stride] = acc;
        }
    }
    /* a run of matches: -(run % 127), then -127s (backwards) */
    __device__ __forceinline__ void push_run(int run, int stride)
    {
        if (run <= 0) return;
        const int r = run % 127;
        if (r) push((uint32_t)(256 - r), stride);
        for (int j = run / 127; j > 0; --j) push(256u - 127u, stride);
    }
    __device__ __forceinline__ void finish(int stride)
    {
        if (n & 3) {
            const int w = top - (n >> 2) - 1;
            if (w >= 0) buf[w * stride] = acc << (8 * (4 - (n & 3)));
        }
    }
};

/* One step of the walk back through a block of 32 columns: from the cell on
 * the band's bit q, hb columns into the block (hb >= 1, or 0 in the first
 * block), the path cell of its score.  wq, wu, wd: increments of bits q, q-1
 * (diagonal k+1) and q+1 (diagonal k-1) over the block's columns; vp, vn:
 * vertical differences at the block's first column (bit i: between band bits
 * i+1 and i).  Returns 4 * x + op for the source candidate x = the cell's
 * first offset after the operation (relative to the block), or -1 when every
 * candidate lies before the block.  q == 0 has no deletion and q == last no
 * insertion (a certified path takes neither). */
__device__ __forceinline__ int walk_step(uint32_t wq, uint32_t wu, uint32_t wd, uint32_t vp, uint32_t vn, int q,
                                         int last, int hb)
{
    const uint32_t below = low_bits(hb);
    const uint32_t a = wq & below, u = wu & below, d = wd & (below >> 1);
    const int na = __popc(a);
    /* 31 - clz is the last set bit, -1 for none */
    const int xs = 32 - __clz((int)a); /* 0: no increment in the block */
    /* deletion: steps back on diagonal k+1 to score s-1 */
    const int du = (int)((vp >> ((q - 1) & 31)) & 1u) - (int)((vn >> ((q - 1) & 31)) & 1u);
    const int ru = 1 - du + __popc(u) - na;
    const int lu = 31 - __clz((int)u);
    const uint32_t u2 = u & ~(1u << (lu & 31)); /* lu == -1: u is 0 anyway */
    int xu = ru <= 0 ? hb : (ru == 1 ? lu : 31 - __clz((int)u2));
    if (q == 0) xu = -1;
    /* insertion: steps back from h-1 on diagonal k-1 to score s-1 */
    const int dd = (int)((vp >> q) & 1u) - (int)((vn >> q) & 1u);
    const int rd = 1 + dd + __popc(d) - na;
    const int ld = 31 - __clz((int)d);
    const uint32_t d2 = d & ~(1u << (ld & 31));
    int xd = rd <= 0 ? hb - 1 : (rd == 1 ? ld : 31 - __clz((int)d2));
    if (q >= last || hb == 0) xd = -1;
    const int kd = 4 * xu + kOpDel;
    const int ks = xs ? 4 * xs + kOpSub : -1;
    const int ki = xd >= 0 ? 4 * (xd + 1) + kOpIns : -1;
    const int best = __vimax3_s32(kd, ks, ki);
    return best;
}

/* ---- bands of NW words of 32 diagonals ------------------------------------ */

/* t += v over NW words, with carries */
template <int NW>
__device__ __forceinline__ void add_words(uint32_t (&t)[NW], const uint32_t (&v)[NW])
{
#ifdef __CUDA_ARCH__
    asm volatile("add.cc.u32 %0, %0, %1;" : "+r"(t[0]) : "r"(v[0]));
#pragma unroll
    for (int i = 1; i < NW - 1; ++i) asm volatile("addc.cc.u32 %0, %0, %1;" : "+r"(t[i]) : "r"(v[i]));
    asm volatile("addc.u32 %0, %0, %1;" : "+r"(t[NW - 1]) : "r"(v[NW - 1]));
#else
    uint64_t c = 0;
    for (int i = 0; i < NW; ++i) {
        c += (uint64_t)t[i] + v[i];
        t[i] = (uint32_t)c;
        c >>= 32;
    }
#endif
}

/* One column of a band of NW words (see band_column): column j of a block,
 * a0/a1 the bit planes of the pattern rows of the block's first column and
 * of the 32 rows after them, t0/t1 the block's text planes. */
template <int NW>
__device__ __forceinline__ void wide_column(const uint32_t (&a0)[NW + 1], const uint32_t (&a1)[NW + 1], uint32_t t0,
                                            uint32_t t1, int j, uint32_t (&vp)[NW], uint32_t (&vn)[NW],
                                            uint32_t (&d0)[NW])
{
    static_assert(NW >= 2, "one word: band_column");
    const uint32_t c0 = bit_mask(t0, j), c1 = bit_mask(t1, j);
    uint32_t eq[NW];
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        const uint32_t x = __funnelshift_r(a0[i], a0[i + 1], (uint32_t)j) ^ c0;
        eq[i] = ~(x | (__funnelshift_r(a1[i], a1[i + 1], (uint32_t)j) ^ c1));
        d0[i] = eq[i] & vp[i];
    }
    add_words<NW>(d0, vp);
#pragma unroll
    for (int i = 0; i < NW; ++i) d0[i] = (d0[i] ^ vp[i]) | eq[i] | vn[i];
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        const uint32_t hp = vn[i] | ~(d0[i] | vp[i]), hn = vp[i] & d0[i];
        const uint32_t x = __funnelshift_r(d0[i], i + 1 < NW ? d0[i + 1] : 0u, 1u);
        vp[i] = hn | ~(x | hp);
        vn[i] = x & hp;
    }
}

/* One column of a tile of 32 rows (eq: the rows that match it), with the
 * horizontal differences that come in above it, at the highest bits of hp_in
 * and hn_in, and those that leave below, collected in hp_out and hn_out
 * (first column highest). */
__device__ __forceinline__ void tile_column(uint32_t eq, uint32_t hp_in, uint32_t hn_in, uint32_t& vp, uint32_t& vn,
                                            uint32_t& hp_out, uint32_t& hn_out)
{
    const uint32_t t = hn_in >> 31;
    const uint32_t a = (eq | t) & vp;
    const uint32_t d0 = ((a + vp) ^ vp) | (eq | t | vn);
    const uint32_t hp = vn | ~(d0 | vp), hn = vp & d0;
    hp_out = __funnelshift_l(hp, hp_out, 1u);
    hn_out = __funnelshift_l(hn, hn_out, 1u);
    const uint32_t sp = __funnelshift_l(hp_in, hp, 1u), sn = __funnelshift_l(hn_in, hn, 1u);
    vp = sn | ~(d0 | sp);
    vn = sp & d0;
}

/* Words of a bit plane of the pattern that start at base r (negative: virtual
 * rows, any bits), from the lane's column of plane words, n of them, `row`
 * words apart. */
template <int N>
__device__ __forceinline__ void plane_window(const uint32_t* plane, int row, int n, int r, uint32_t (&a)[N])
{
    const int w0 = r >> 5;
    uint32_t x = (unsigned)w0 < (unsigned)n ? plane[(size_t)w0 * row] : 0u;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const int w = w0 + k + 1;
        const uint32_t y = (unsigned)w < (unsigned)n ? plane[(size_t)w * row] : 0u;
        a[k] = __funnelshift_r(x, y, (uint32_t)(r & 31));
        x = y;
    }
}

/* Move a band of 64 diagonals by `by` (16 or -16) diagonals, downwards for
 * by > 0: bit i becomes bit i - by.  Rows that enter count one more than
 * their neighbour in the band (an upper bound, as every value of a band);
 * returns the change of the value on bit 0. */
__device__ __forceinline__ int move_band(uint32_t (&vp)[2], uint32_t (&vn)[2], int by)
{
    if (by > 0) {
        const int top = __popc(vp[0] & 0xffffu) - __popc(vn[0] & 0xffffu);
        vp[0] = __funnelshift_r(vp[0], vp[1], 16u);
        vn[0] = __funnelshift_r(vn[0], vn[1], 16u);
        vp[1] = (vp[1] >> 16) | 0xffff0000u;
        vn[1] >>= 16;
        return top;
    }
    vp[1] = __funnelshift_l(vp[0], vp[1], 16u);
    vn[1] = __funnelshift_l(vn[0], vn[1], 16u);
    vp[0] <<= 16;
    vn[0] = (vn[0] << 16) | 0xffffu;
    return 16;
}

}  // namespace wfe

#endif
