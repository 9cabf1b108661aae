// GGUF mat-vec on the integer tensor-core instruction (mma.sync s8): dense calls from five batch rows
// on, in passes of eight, and grouped calls, in segments of one to eight rows.
//
// With more batch rows the mat-vec of mmvq.cuh is bound by its dp4a arithmetic (eight rows of
// Q6_K: a quarter of the copy bandwidth; 28672 x 4096 54.3 us there and 36.4 here, Q4_K 40.0 and
// 25.2; the MoE layer of 64 tokens 307 and 134), so here a warp multiplies 16 weight rows by eight
// batch rows: one mma.m16n8k32 (k16 for Q6_K, whose scales cover 16 values) replaces 32 dp4a per
// lane, and with the magic number 1.5 * 2^23 as the initial accumulator its integer result is
// read as a float with one subtraction.  The sums of a scale group are the same exact integers
// as before; the products with the scales keep their terms, and their fp32 sums are made in an order
// of their own (mma_add_tiles).
//
// mma.sync and not tcgen05: the sums have to be rescaled every 16 or 32 values of K, and an
// accumulator in tensor memory would be drained as often.  At eight columns the instruction is
// not the limit either (the scale arithmetic around it is).
//
//   * The K of an operand fragment may be permuted as long as both operands agree.  Lane (g, t)
//     of the warp takes bytes 8t..8t+7 of the packed 32 bytes of rows g and g + 8 (one 8-byte
//     load, low nibbles = one scale group, high nibbles = the next) and the activation image
//     keeps a block of eight columns x 32 codes so that the matching operand is one 8-byte load.
//   * Every warp streams the blocks it multiplies itself: cp.async of 16-byte pieces into a ring of
//     its own, two to four 16-row blocks deep, so nothing is synchronised between warps on the way
//     in.  The rows' pitch is chosen so that the eight rows of a fragment load hit different banks.
//     (One bulk copy per row and stage, as first written, took the copy engine 80 to 110 cycles
//     each: 66 MB of Q4_K in 20 us with the arithmetic left out.)
//   * `wpg` warps share a row group, warp i taking blocks i, i + wpg, ..; their partial 16 x 8
//     tiles are added through shared memory, in a fixed order.  16 / wpg groups are in work at a time.
//   * Long rows are split along K over the CTAs of a cluster (4096 values each): a CTA then
//     quantizes and holds only its part of the activations, and the cluster has more rows.
//     The CTAs add their sums in a fixed order through distributed shared memory, in as many pieces
//     (`chunk` row groups) as the sums of the cluster's rows take beside the image and the rings.
// Whether a call comes here depends on its type, K and batch rows alone, and how K is cut on the
// type and K, so a result does not depend on the number of weight rows, on what shares the launch,
// or on the launch geometry.
#pragma once

#include "mmvq_grouped.cuh"

namespace lsg {

constexpr int kMmaWarps = 16;
constexpr int kMmaThreads = kMmaWarps * 32;
constexpr int kMmaCols = 8;                           // batch rows of one launch
constexpr int kMmaSliceBlocks = 16;                   // 256-value blocks of one CTA's share of K, at most
constexpr int kMmaGroupedBlocks = 16;                 // .. of a row in a grouped call, which has no clusters
constexpr int kMmaMaxDepth = 4;

// How a row is cut and where things lie in shared memory.
struct MmaCut {
    int sb_bytes;        // bytes of 256 packed values
    int nsb;             // 256-value blocks of a row
    int ksplit, slice;   // CTAs of a cluster along K, blocks of each
    int wpg;             // warps of a row group
    int depth;           // 16-row blocks of a warp's ring
    int chunk;           // row groups between two cluster sums
    int ring_off, part_off, sum_off;   // image (at 0), rings, partial tiles, cluster sums
};

struct MmaArgs {
    MmvqArgs v;          // operands, joined matrices (CTA numbers count clusters), waits
    MmaCut c;
};

struct MmaGroupedArgs {
    GroupedArgs v;
    MmaCut c;
};

// The types this kernel is built for (the ones with byte-sized scale groups that are in use; the
// others keep the dp4a kernel).
template <int T> struct MmaDec { static constexpr bool kHas = false; };

#if defined(__CUDACC__)

// d = a * b + c; a start of its own, and not the result's registers, so that none is copied.
__device__ __forceinline__ void mma_u8s8_k32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1, int c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c));
}
__device__ __forceinline__ void mma_s8s8_k32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1, int c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c));
}
__device__ __forceinline__ void mma_u8s8_k16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, const uint4& c) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(c.x), "r"(c.y), "r"(c.z), "r"(c.w));
}

// An integer of magnitude below 2^22 added to this bit pattern is that integer as a float, offset
// by kMmaBias; the largest sum here is 32 * 128 * 127.
constexpr int kMmaBiasBits = 0x4B400000;
constexpr float kMmaBias = 12582912.0f;
// (c - bias) * s with ns = -bias * s: the product of a sum below 2^22 and a scale below 2^8 in
// magnitude is an integer of at most 24 bits here, so the one rounding of the fma is exact.
__device__ __forceinline__ float mma_scaled(int c, float s, float ns) { return fmaf(__int_as_float(c), s, ns); }
// Byte k of w as a float (unsigned; or signed after its sign bit has been flipped).
__device__ __forceinline__ float byte_f(uint32_t w, int k) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7550u | k)) - 8388608.0f;
}
__device__ __forceinline__ float sbyte_f(uint32_t w_flipped, int k) {
    return __uint_as_float(__byte_perm(w_flipped, 0x4B000000u, 0x7550u | k)) - 8388736.0f;
}
// Unaligned words at constant distances (multiples of 4) from one address: the alignment is worked
// out once.
struct MmaWords {
    uint32_t base, sh;
    __device__ __forceinline__ explicit MmaWords(uint32_t addr) : base(addr & ~3u), sh((addr & 3u) * 8u) {}
    __device__ __forceinline__ uint32_t at(int off) const { return __funnelshift_r(lds32(base + off), lds32(base + off + 4), sh); }
};

// tile(): acc[i] += the products of one 256-value block: rows r0 (accumulators 0, 1) and r1 (2, 3)
// with columns 2t and 2t + 1 (types with a scale per 32 values: in four sets of accumulators, by turns).
//   r0, r1  shared addresses of the block in rows g and g + 8
//   xq      codes of this lane's column g: block j of the 256 values at xq + 256 j, lane offset in
//   xs      scales of columns 2t, 2t + 1 (and what kKind says): block j at xs + j * kScaleBytes
// ODD false: the odd columns hold nothing (their accumulators are left alone).
// kHalves: the words of a block's two 16-value halves alternate in the image.
// kKind: 0 scales {d}; 1 {d, d * sum of the codes}; 2 {d} and, behind the scales of all blocks, the
// accumulator starts of the block's two halves, bias - 32 * sum of the half's codes, for columns
// 2t, 2t + 1 twice over (Q6_K: the offset of its codes is in the sums before they are scaled).
template <bool FIVE> struct MmaDecK45 {   // Q4_K, Q5_K
    static constexpr bool kHas = true;
    static constexpr int kKind = 1, kScaleBytes = 64;
    static constexpr bool kHalves = false;
    static constexpr int kBytes = FIVE ? 176 : 144;
    static constexpr int kPitch = FIVE ? 176 : 160;   // 8-byte loads of four rows: no bank twice with 160 (224 would not fit)

    template <bool ODD>
    __device__ static __forceinline__ void tile(uint32_t r0, uint32_t r1, int t, uint32_t xq, uint32_t xs, uint32_t,
                                                float (&acc)[16]) {
        constexpr int QS = FIVE ? 48 : 16;
        const uint4 h0 = lds128(r0), h1 = lds128(r1);
        uint32_t sc0[2], mn0[2], sc1[2], mn1[2];
        k4_unpack_all(h0.y, h0.z, h0.w, sc0, mn0);
        k4_unpack_all(h1.y, h1.z, h1.w, sc1, mn1);
        uint2 f0 = make_uint2(0, 0), f1 = f0;   // fifth bits
        if (FIVE) {
            f0 = lds64(r0 + 16 + 8 * t);
            f1 = lds64(r1 + 16 + 8 * t);
        }
        const float d0 = fp16_bits_to_float(h0.x), e0 = fp16_bits_to_float(h0.x >> 16);
        const float d1 = fp16_bits_to_float(h1.x), e1 = fp16_bits_to_float(h1.x >> 16);
        float sum1[2][4] = {}, sum2[2][4] = {};   // of each half block: sums of four sub-blocks
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            float (&s1)[4] = sum1[p >> 1], (&s2)[4] = sum2[p >> 1];
            const uint2 q0 = lds64(r0 + QS + 32 * p + 8 * t), q1 = lds64(r1 + QS + 32 * p + 8 * t);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int j = 2 * p + hf;
                uint32_t a0 = (q0.x >> (4 * hf)) & 0x0F0F0F0Fu, a2 = (q0.y >> (4 * hf)) & 0x0F0F0F0Fu;
                uint32_t a1 = (q1.x >> (4 * hf)) & 0x0F0F0F0Fu, a3 = (q1.y >> (4 * hf)) & 0x0F0F0F0Fu;
                if (FIVE) {
                    a0 |= ((f0.x >> j) & 0x01010101u) << 4;
                    a2 |= ((f0.y >> j) & 0x01010101u) << 4;
                    a1 |= ((f1.x >> j) & 0x01010101u) << 4;
                    a3 |= ((f1.y >> j) & 0x01010101u) << 4;
                }
                const uint2 xb = lds64(xq + 256 * j);
                uint4 xv = make_uint4(0, 0, 0, 0);
                if (ODD) {
                    xv = lds128(xs + 64 * j);
                } else {
                    const uint2 e = lds64(xs + 64 * j);
                    xv.x = e.x;
                    xv.y = e.y;
                }
                const float dx0 = __uint_as_float(xv.x), sx0 = __uint_as_float(xv.y);
                const float dx1 = __uint_as_float(xv.z), sx1 = __uint_as_float(xv.w);
                int c[4];
                mma_u8s8_k32(c, a0, a1, a2, a3, xb.x, xb.y, kMmaBiasBits);
                const float c0 = byte_f(sc0[j >> 2], j & 3), c1 = byte_f(sc1[j >> 2], j & 3);
                const float m0 = byte_f(mn0[j >> 2], j & 3), m1 = byte_f(mn1[j >> 2], j & 3);
                const float n0 = -kMmaBias * c0, n1 = -kMmaBias * c1;
                s1[0] = fmaf(dx0, mma_scaled(c[0], c0, n0), s1[0]);
                s1[2] = fmaf(dx0, mma_scaled(c[2], c1, n1), s1[2]);
                s2[0] = fmaf(m0, sx0, s2[0]);
                s2[2] = fmaf(m1, sx0, s2[2]);
                if (ODD) {
                    s1[1] = fmaf(dx1, mma_scaled(c[1], c0, n0), s1[1]);
                    s1[3] = fmaf(dx1, mma_scaled(c[3], c1, n1), s1[3]);
                    s2[1] = fmaf(m0, sx1, s2[1]);
                    s2[3] = fmaf(m1, sx1, s2[3]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i += ODD ? 1 : 2)
            acc[i] += (i < 2 ? d0 : d1) * (sum1[0][i] + sum1[1][i]) - (i < 2 ? e0 : e1) * (sum2[0][i] + sum2[1][i]);
    }
};
template <> struct MmaDec<LSG_GGUF_Q4_K> : MmaDecK45<false> {};
template <> struct MmaDec<LSG_GGUF_Q5_K> : MmaDecK45<true> {};

template <> struct MmaDec<LSG_GGUF_Q6_K> {
    static constexpr bool kHas = true;
    static constexpr int kKind = 2, kScaleBytes = 32;
    static constexpr bool kHalves = true;
    static constexpr int kBytes = 210;
    static constexpr int kPitch = 240;   // 4-byte loads of eight rows: no bank twice

    template <bool ODD>
    __device__ static __forceinline__ void tile(uint32_t r0, uint32_t r1, int t, uint32_t xq, uint32_t xs, uint32_t xi,
                                                float (&acc)[16]) {
        const MmaWords w[2] = {MmaWords(r0), MmaWords(r1)};
        uint32_t scw[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 4; ++i) scw[r][i] = w[r].at(192 + 4 * i) ^ 0x80808080u;
        const MmaWords v[2] = {MmaWords(r0 + 4 * t), MmaWords(r1 + 4 * t)};
        // rows keep the offset that their matrix has in memory, odd ones too: no 2-byte loads
        const float d0 = fp16_bits_to_float(w[0].at(208)), d1 = fp16_bits_to_float(w[1].at(208));
#pragma unroll
        for (int ip = 0; ip < 2; ++ip) {
            float s[4] = {0.f, 0.f, 0.f, 0.f};   // of half a block, as the dp4a kernel's units
            uint32_t la[2][2], lb[2][2], qh[2][2];   // [row][16-value half]
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int hs = 0; hs < 2; ++hs) {
                    la[r][hs] = v[r].at(64 * ip + 16 * hs);
                    lb[r][hs] = v[r].at(64 * ip + 32 + 16 * hs);
                    qh[r][hs] = v[r].at(128 + 32 * ip + 16 * hs);
                }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = 4 * ip + q;
                const uint2 xb = lds64(xq + 256 * j);
                const uint2 xv = lds64(xs + 32 * j);
                int c[2][4];
#pragma unroll
                for (int hs = 0; hs < 2; ++hs) {
                    uint32_t a[2];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const uint32_t lo = ((q & 1) ? lb[r][hs] : la[r][hs]) >> (4 * (q >> 1));
                        const uint32_t hi = q == 0 ? qh[r][hs] << 4 : (q == 1 ? qh[r][hs] << 2 : (q == 2 ? qh[r][hs] : qh[r][hs] >> 2));
                        a[r] = (lo & 0x0F0F0F0Fu) | (hi & 0x30303030u);
                    }
                    mma_u8s8_k16(c[hs], a[0], a[1], hs ? xb.y : xb.x, lds128(xi + 128 * j + 64 * hs));
                }
                const int e = 8 * ip + 2 * q;
                const float dx0 = __uint_as_float(xv.x), dx1 = __uint_as_float(xv.y);
                // both halves' integer products together stay below 2^24: exact
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float sa = sbyte_f(scw[r][e >> 2], e & 3), sb = sbyte_f(scw[r][(e + 1) >> 2], (e + 1) & 3);
                    const float na = -kMmaBias * sa, nb = -kMmaBias * sb;
                    s[2 * r] = fmaf(dx0, mma_scaled(c[0][2 * r], sa, na) + mma_scaled(c[1][2 * r], sb, nb), s[2 * r]);
                    if (ODD)
                        s[2 * r + 1] = fmaf(dx1, mma_scaled(c[0][2 * r + 1], sa, na) + mma_scaled(c[1][2 * r + 1], sb, nb), s[2 * r + 1]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i += ODD ? 1 : 2) acc[i] += (i < 2 ? d0 : d1) * s[i];
        }
    }
};

template <> struct MmaDec<LSG_GGUF_Q8_0> {   // eight 34-byte blocks
    static constexpr bool kHas = true;
    static constexpr int kKind = 0, kScaleBytes = 32;
    static constexpr bool kHalves = false;
    static constexpr int kBytes = 272;
    static constexpr int kPitch = 272;

    template <bool ODD>
    __device__ static __forceinline__ void tile(uint32_t r0, uint32_t r1, int t, uint32_t xq, uint32_t xs, uint32_t,
                                                float (&acc)[16]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            // rows start on 16-byte boundaries: every second block's codes are a half word off
            const uint32_t p0 = r0 + 8 * t + ((34 * j + 2) & ~3), p1 = r1 + 8 * t + ((34 * j + 2) & ~3);
            uint32_t w0[3], w1[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                w0[i] = (i < 2 || j % 2 == 0) ? lds32(p0 + 4 * i) : 0u;
                w1[i] = (i < 2 || j % 2 == 0) ? lds32(p1 + 4 * i) : 0u;
            }
            if (j % 2 == 0) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    w0[i] = __byte_perm(w0[i], w0[i + 1], 0x5432);
                    w1[i] = __byte_perm(w1[i], w1[i + 1], 0x5432);
                }
            }
            const uint2 xb = lds64(xq + 256 * j);
            const uint2 xv = lds64(xs + 32 * j);
            int c[4];
            mma_s8s8_k32(c, w0[0], w1[0], w0[1], w1[1], xb.x, xb.y, kMmaBiasBits);
            const float d0 = fp16_bits_to_float(lds16(r0 + 34 * j)), d1 = fp16_bits_to_float(lds16(r1 + 34 * j));
            const float dx0 = __uint_as_float(xv.x), dx1 = __uint_as_float(xv.y);
            float* const s = acc + 4 * (j & 3);
            s[0] = fmaf(d0 * dx0, __int_as_float(c[0]) - kMmaBias, s[0]);
            s[2] = fmaf(d1 * dx0, __int_as_float(c[2]) - kMmaBias, s[2]);
            if (ODD) {
                s[1] = fmaf(d0 * dx1, __int_as_float(c[1]) - kMmaBias, s[1]);
                s[3] = fmaf(d1 * dx1, __int_as_float(c[3]) - kMmaBias, s[3]);
            }
        }
    }
};

template <> struct MmaDec<LSG_GGUF_Q4_0> {   // eight 18-byte blocks; byte i: values i and i + 16
    static constexpr bool kHas = true;
    static constexpr int kKind = 0, kScaleBytes = 32;
    static constexpr bool kHalves = true;
    static constexpr int kBytes = 144;
    static constexpr int kPitch = 144;

    // four nibbles 0..15 -> value - 8 as signed bytes
    __device__ static __forceinline__ uint32_t sext4(uint32_t v) {
        const uint32_t x = v ^ 0x08080808u;
        return x | ((x & 0x08080808u) * 30u);
    }
    template <bool ODD>
    __device__ static __forceinline__ void tile(uint32_t r0, uint32_t r1, int t, uint32_t xq, uint32_t xs, uint32_t,
                                                float (&acc)[16]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            // rows start on 16-byte boundaries: every second block's codes are a half word off
            const uint32_t p0 = r0 + 4 * t + ((18 * j + 2) & ~3), p1 = r1 + 4 * t + ((18 * j + 2) & ~3);
            const uint32_t w0 = j % 2 ? lds32(p0) : __byte_perm(lds32(p0), lds32(p0 + 4), 0x5432);
            const uint32_t w1 = j % 2 ? lds32(p1) : __byte_perm(lds32(p1), lds32(p1 + 4), 0x5432);
            const uint2 xb = lds64(xq + 256 * j);
            const uint2 xv = lds64(xs + 32 * j);
            int c[4];
            mma_s8s8_k32(c, sext4(w0 & 0x0F0F0F0Fu), sext4(w1 & 0x0F0F0F0Fu), sext4((w0 >> 4) & 0x0F0F0F0Fu),
                         sext4((w1 >> 4) & 0x0F0F0F0Fu), xb.x, xb.y, kMmaBiasBits);
            const float d0 = fp16_bits_to_float(lds16(r0 + 18 * j)), d1 = fp16_bits_to_float(lds16(r1 + 18 * j));
            const float dx0 = __uint_as_float(xv.x), dx1 = __uint_as_float(xv.y);
            float* const s = acc + 4 * (j & 3);
            s[0] = fmaf(d0 * dx0, __int_as_float(c[0]) - kMmaBias, s[0]);
            s[2] = fmaf(d1 * dx0, __int_as_float(c[2]) - kMmaBias, s[2]);
            if (ODD) {
                s[1] = fmaf(d0 * dx1, __int_as_float(c[1]) - kMmaBias, s[1]);
                s[3] = fmaf(d1 * dx1, __int_as_float(c[3]) - kMmaBias, s[3]);
            }
        }
    }
};

// ---------------------------------------------------------------------------
// Activation image of `nblk` 32-value blocks from block b0 on: codes [block][column][32], then the
// scales and accumulator starts of D::kKind.  Batch row m is column m, or column 2m where there are
// at most four (mma_step): every lane then has one column with a row, and does the scale arithmetic
// of one instead of two - with one row per expert 64 x (768 x 2048) of Q4_K took the grouped kernel
// longer than dp4a.  Columns without a batch row keep what was there: it stays in their own sums.
// ---------------------------------------------------------------------------
template <class D>
__device__ __forceinline__ void mma_put_half(uint8_t* img, int b, int col, int half, const uint4& q) {
    uint8_t* at = img + b * 256 + col * 32;
    if (D::kHalves) {   // words of the two halves alternate
        uint32_t* w = reinterpret_cast<uint32_t*>(at) + half;
        w[0] = q.x;
        w[2] = q.y;
        w[4] = q.z;
        w[6] = q.w;
    } else {
        *reinterpret_cast<uint4*>(at + 16 * half) = q;
    }
}
__device__ __forceinline__ int mma_step(int M) { return M <= kMmaCols / 2 ? 2 : 1; }
template <class D> __host__ __device__ constexpr int mma_image_bytes(int nblk) {
    return nblk * (256 + D::kScaleBytes + (D::kKind == 2 ? 128 : 0));
}
// sum: of the 32 codes; with kKind 2 of the 16 of half `half` (called once per half then)
template <class D>
__device__ __forceinline__ void mma_put_scale(uint8_t* img, int nblk, int b, int col, int half, float d, int sum) {
    float* s = reinterpret_cast<float*>(img + nblk * 256);
    if (D::kKind == 1) {
        *reinterpret_cast<float2*>(s + (b * 8 + col) * 2) = make_float2(d, d * static_cast<float>(sum));
    } else {
        if (half == 0) s[b * 8 + col] = d;
        if (D::kKind == 2) {
            int* start = reinterpret_cast<int*>(img + nblk * (256 + D::kScaleBytes)) + (b * 2 + half) * 16 + (col >> 1) * 4 + (col & 1);
            start[0] = start[2] = kMmaBiasBits - 32 * sum;
        }
    }
}

template <class D>
__device__ __forceinline__ void mma_image_q8_1(uint8_t* img, const uint8_t* __restrict__ xq, int M, int row_blocks,
                                               int b0, int nblk, int tid, int nthreads) {
    for (int idx = tid; idx < M * nblk; idx += nthreads) {
        const int m = idx / nblk, b = idx - m * nblk, col = m * mma_step(M);
        uint32_t w[9];
        const uint32_t* src = reinterpret_cast<const uint32_t*>(xq + (static_cast<size_t>(m) * row_blocks + b0 + b) * kQ8_1Bytes);
#pragma unroll
        for (int i = 0; i < 9; ++i) w[i] = __ldg(src + i);
        int sum[2] = {0, 0};
#pragma unroll
        for (int i = 1; i < 9; ++i) sum[(i - 1) >> 2] = __dp4a(static_cast<int>(w[i]), 0x01010101, sum[(i - 1) >> 2]);
        mma_put_half<D>(img, b, col, 0, make_uint4(w[1], w[2], w[3], w[4]));
        mma_put_half<D>(img, b, col, 1, make_uint4(w[5], w[6], w[7], w[8]));
        const float d = fp16_bits_to_float(w[0]);
        if (D::kKind == 2) {
            mma_put_scale<D>(img, nblk, b, col, 0, d, sum[0]);
            mma_put_scale<D>(img, nblk, b, col, 1, d, sum[1]);
        } else {
            mma_put_scale<D>(img, nblk, b, col, 0, d, sum[0] + sum[1]);
        }
    }
}

// The same from bf16 activations, two lanes per block (the quantizer of build_x_image_bf16).
template <class D>
__device__ __forceinline__ void mma_image_bf16(uint8_t* img, const __nv_bfloat16* __restrict__ A, int M, int K, int b0,
                                               int nblk, int tid, int nthreads) {
    const int total = M * nblk * 2;
    for (int base = tid & ~31; base < total; base += nthreads) {   // whole warps: the two lanes of a block exchange values
        const int idx = min(base + (tid & 31), total - 1);
        const bool live = base + (tid & 31) < total;
        const int half = idx & 1, task = idx >> 1;
        const int m = task / nblk, b = task - m * nblk;
        const uint4* src = reinterpret_cast<const uint4*>(A + static_cast<size_t>(m) * K + static_cast<size_t>(b0 + b) * 32 + 16 * half);
        const uint4 r0 = __ldg(src), r1 = __ldg(src + 1);
        const uint32_t w[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
        float x[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            x[2 * i] = __uint_as_float(w[i] << 16);
            x[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
        }
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(x[i]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        const float d = amax / 127.0f;
        const float rcp = (amax == 0.0f) ? 0.0f : 1.0f / d;
        uint4 q;
        q8_round8(x, d, rcp, q.x, q.y);
        q8_round8(x + 8, d, rcp, q.z, q.w);
        int sum = __dp4a(static_cast<int>(q.x), 0x01010101,
                  __dp4a(static_cast<int>(q.y), 0x01010101,
                  __dp4a(static_cast<int>(q.z), 0x01010101,
                  __dp4a(static_cast<int>(q.w), 0x01010101, 0))));
        if (D::kKind != 2) sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        if (live) {
            const int col = m * mma_step(M);
            mma_put_half<D>(img, b, col, half, q);
            if (D::kKind == 2 || half == 0) mma_put_scale<D>(img, nblk, b, col, half, __half2float(__float2half(d)), sum);
        }
    }
}

__device__ __forceinline__ void mma_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float mma_ld_cluster(uint32_t local_addr, uint32_t rank) {
    uint32_t addr;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local_addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// A warp's weight stream: 16-row blocks through its ring.  A block's rows are copied as 16-byte
// pieces; where blocks are not whole pieces (kShifted), those that meet the row, which keeps its
// offset from a 16-byte boundary.  The bytes behind the last whole piece of a matrix, and all of a
// matrix that is not 16-byte aligned (w_end = 0), are moved one by one.
template <class D>
struct MmaStream {
    static constexpr bool kShifted = D::kBytes % 16 != 0;
    static constexpr int kPieces = kShifted ? (D::kBytes + 15 + 15) / 16 : D::kBytes / 16;
    // kShifted: sixteen lanes per row, two rows per issue; otherwise the pieces of all rows in turn
    static constexpr int kIssues = kShifted ? 8 : (16 * kPieces + 31) / 32;
    static_assert(kPieces <= 16 || !kShifted, "sixteen lanes cover a row");
    static_assert(kPieces * 16 <= D::kPitch, "a row's pieces fit its pitch");
    uint32_t goff[kShifted ? 1 : kIssues], soff[kShifted ? 1 : kIssues];   // this lane's pieces, from the block's first row
    uint32_t row_bytes;
    int lane;

    __device__ __forceinline__ MmaStream(uint32_t rb, int l) : row_bytes(rb), lane(l) {
        if (kShifted) {
            goff[0] = static_cast<uint32_t>(lane >> 4) * rb;
            soff[0] = static_cast<uint32_t>((lane >> 4) * D::kPitch + 16 * (lane & 15));
        } else {
#pragma unroll
            for (int i = 0; i < kIssues; ++i) {
                const int p = lane + 32 * i, row = p / kPieces, k = p - row * kPieces;
                goff[i] = static_cast<uint32_t>(row) * rb + 16 * k;
                soff[i] = static_cast<uint32_t>(row * D::kPitch + 16 * k);
            }
        }
    }
    __device__ static __forceinline__ void copy16(uint32_t dst, uintptr_t src, uint64_t policy) {
        asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
    }
    // src: first row of the group at the block, of which nrows rows are left
    __device__ __forceinline__ void issue(uint32_t slot, uintptr_t src, int nrows, uintptr_t w_end, uint64_t policy) const {
        nrows = min(nrows, 16);
        const uintptr_t last = src + static_cast<uintptr_t>(static_cast<uint32_t>(nrows - 1) * row_bytes) + D::kBytes;
        if (((last + 15) & ~uintptr_t(15)) <= w_end) {
            if (kShifted) {
                const uint32_t k16 = 16 * (lane & 15);
                uintptr_t b = src + goff[0];
                uint32_t dst = slot + soff[0];
#pragma unroll
                for (int i = 0; i < kIssues; ++i) {
                    const uint32_t off = static_cast<uint32_t>(b) & 15u;
                    if (2 * i + (lane >> 4) < nrows && k16 < off + D::kBytes) copy16(dst, b - off + k16, policy);
                    b += 2 * row_bytes;
                    dst += 2 * D::kPitch;
                }
            } else {
#pragma unroll
                for (int i = 0; i < kIssues; ++i)
                    if (lane + 32 * i < nrows * kPieces) copy16(slot + soff[i], src + goff[i], policy);
            }
            return;
        }
        for (int p = lane; p < nrows * kPieces; p += 32) {
            const int row = p / kPieces, k = p - row * kPieces;
            const uintptr_t b = src + static_cast<uintptr_t>(static_cast<uint32_t>(row) * row_bytes);
            const uintptr_t at = (kShifted ? b & ~uintptr_t(15) : b) + 16 * k;
            const uint32_t dst = slot + static_cast<uint32_t>(row * D::kPitch + 16 * k);
            if (at + 16 <= w_end) {
                copy16(dst, at, policy);
            } else {
                for (uintptr_t q = at < b ? b : at; q < at + 16 && q < b + D::kBytes; ++q)
                    asm volatile("st.shared.u8 [%0], %1;" ::"r"(dst + static_cast<uint32_t>(q - at)),
                                 "r"(static_cast<uint32_t>(*reinterpret_cast<const uint8_t*>(q)))
                                 : "memory");
            }
        }
    }
};

// Waits until all but the youngest depth - 1 blocks of this thread's copies have landed.
__device__ __forceinline__ void mma_wait_block(int depth) {
    if (depth == 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
    else if (depth == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else asm volatile("cp.async.wait_group 1;" ::: "memory");
}

// What a warp needs of the image and its ring.
template <class D>
struct MmaWarp {
    uint32_t xq, xs, xi, ring;
    int lane, wi, set, depth;
    __device__ __forceinline__ MmaWarp(const MmaCut& g, uint8_t* smem, int nblk) {
        lane = threadIdx.x & 31;
        const int warp = threadIdx.x >> 5;
        set = warp / g.wpg;
        wi = warp - set * g.wpg;
        depth = g.depth;
        const uint32_t img = smem_u32(smem);
        xq = img + (lane >> 2) * 32 + 8 * (lane & 3);
        xs = img + nblk * 256 + (lane & 3) * (D::kScaleBytes / 4);
        xi = img + nblk * (256 + D::kScaleBytes) + (lane & 3) * 16;
        ring = img + g.ring_off + static_cast<uint32_t>(warp * depth * 16 * D::kPitch);
    }
    __device__ __forceinline__ uint32_t slot(int i) const { return ring + static_cast<uint32_t>(i * 16 * D::kPitch); }
    // The block in slot i times the columns; lo: low bits of the address of its first row.
    template <bool ODD> __device__ __forceinline__ void multiply(int i, int sb, uint32_t lo, uint32_t row_bytes, float (&acc)[16]) const {
        const int gl = lane >> 2;
        uint32_t p0 = slot(i) + static_cast<uint32_t>(gl * D::kPitch), p1 = p0 + 8 * D::kPitch;
        if (MmaStream<D>::kShifted) {
            const uint32_t a = lo + static_cast<uint32_t>(gl) * row_bytes;
            p0 += a & 15u;
            p1 += (a + 8u * row_bytes) & 15u;
        }
        D::template tile<ODD>(p0, p1, lane & 3, xq + sb * 2048, xs + sb * 8 * D::kScaleBytes, xi + sb * 1024, acc);
    }
};

// at(0) + .. + at(n - 1), n <= 8 a power of two: neighbours first, then neighbours of those.
template <class At>
__device__ __forceinline__ float mma_sum8(int n, At at) {
    float p[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) p[i] = i < n ? at(i) : 0.0f;
    return ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
}

// The orders of the fp32 sums are chosen so that the error of a result against 64 bits is no larger
// than the dp4a kernel's (2-norm, relative, K of 768 to 28672; dp4a / here): Q4_K and Q5_K 1.65e-7 to
// 1.84e-7 / 1.64e-7 to 1.79e-7 (sums of four sub-blocks), Q6_K 7.5e-8 to 9.6e-8 / 6.2e-8 to 9.3e-8,
// Q8_0 and Q4_0 6.4e-8 to 1.14e-7 / 6.1e-8 to 7.7e-8 (four accumulators per lane; what the additions
// of the warps' tiles lose is carried along).
//
// The partial tiles of a row group's warps, added in a fixed order.  sink(row, column, value) takes
// each sum of a batch row's column once (column: the batch row).  Tiles alternate between two buffers:
// the one being read is not written before every warp of the group has passed the next barrier.
template <class D, bool ODD, class Sink>
__device__ __forceinline__ void mma_add_tiles(const MmaCut& g, float* part, int set, int buf, int wi, int lane, const float (&acc)[16],
                                              Sink sink) {
    float* all = part + (set * 2 + buf) * g.wpg * 128;
    float* mine = all + wi * 128;
    const int gl = lane >> 2, t = lane & 3;
    const auto sum = [&](int i) { return (acc[i] + acc[4 + i]) + (acc[8 + i] + acc[12 + i]); };   // zeros where a type has one accumulator
    if (ODD) {
        *reinterpret_cast<float2*>(mine + gl * 8 + 2 * t) = make_float2(sum(0), sum(1));
        *reinterpret_cast<float2*>(mine + (gl + 8) * 8 + 2 * t) = make_float2(sum(2), sum(3));
    } else {
        mine[gl * 8 + t] = sum(0);
        mine[(gl + 8) * 8 + t] = sum(2);
    }
    if (g.wpg == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(2 + set), "r"(g.wpg * 32) : "memory");
    for (int i = wi * 32 + lane; i < (ODD ? 128 : 64); i += g.wpg * 32) {
        const int col = i >> 4, r = i & 15;
        const float* p = all + r * 8 + col;
        float v = p[0], low = 0.0f;
        for (int w = 1; w < g.wpg; ++w) {
            const float x = p[w * 128], t = v + x;
            if (D::kKind == 0) {   // what the addition lost (exact)
                const float b = t - v;
                low += (v - (t - b)) + (x - b);
            }
            v = t;
        }
        sink(r, col, low == low ? v + low : v);   // an infinite sum loses NaN
    }
}

template <bool B> struct MmaFlag { static constexpr bool value = B; };

template <int T>
__global__ void __launch_bounds__(kMmaThreads, 1) mmvq_mma_kernel(const MmaArgs args) {
    using D = MmaDec<T>;
    const MmvqArgs& a = args.v;
    const MmaCut& g = args.c;
    extern __shared__ __align__(128) uint8_t smem[];
    float* part = reinterpret_cast<float*>(smem + g.part_off);     // [set][2][wpg][16 rows][8]
    float* sums = reinterpret_cast<float*>(smem + g.sum_off);      // [row of the chunk][8], with ksplit > 1

    const int tid = threadIdx.x;
    const int rank = static_cast<int>(blockIdx.x) % g.ksplit;
    int bx = static_cast<int>(blockIdx.x) / g.ksplit;
    const uint8_t* Wm = a.W;
    const __nv_bfloat16* Am = a.A;
    const uint8_t* xqm = a.xq;
    void* Cm = a.C;
    int Mm = a.M, Nm = a.N, ldcm = a.ldc, rows_q = a.rows_q, rows_r = a.rows_r;
    if (a.n_extra > 0) {
        const int b = bx;
        int jm = -1;
#pragma unroll
        for (int j = 0; j < kMmvqMaxExtra; ++j)
            if (j < a.n_extra && b >= a.cta0x[j]) jm = j;
        if (jm >= 0) {
            Wm = a.Wx[jm];
            Am = a.Ax[jm];
            xqm = a.xqx[jm];
            Cm = a.Cx[jm];
            Mm = a.Mx[jm];
            Nm = ldcm = a.Nx[jm];
            rows_q = a.rows_qx[jm];
            rows_r = a.rows_rx[jm];
            bx = b - a.cta0x[jm];
        }
    }
    const int row_begin = bx * rows_q + min(bx, rows_r);
    const int row_end = row_begin + rows_q + (bx < rows_r ? 1 : 0);
    const int groups = (row_end - row_begin + 15) >> 4;
    const int sb0 = rank * g.slice;
    const int nsb = min(g.slice, g.nsb - sb0);   // blocks of this CTA's part of K

    // dep_mode 1: nothing behind this launch runs before the work in front of the batch is done
    if (a.dep_mode != 1) pdl_launch_dependents();

    const MmaWarp<D> w(g, smem, nsb * 8);
    const int nsets = kMmaWarps / g.wpg;
    const uint32_t row_bytes = static_cast<uint32_t>(a.row_bytes);
    const MmaStream<D> stream(row_bytes, w.lane);
    const uintptr_t w_base = reinterpret_cast<uintptr_t>(Wm) + static_cast<uintptr_t>(sb0) * D::kBytes;
    const uintptr_t w_end = (reinterpret_cast<uintptr_t>(Wm) + static_cast<uintptr_t>(Nm) * row_bytes) & ~uintptr_t(15);
    const uint64_t policy = l2_policy_evict_first();

    // The stream's cursor: the next block to be copied and the slot it goes to.  Weights are
    // constants of the model, so the ring fills before the wait for the kernel in front.
    int pg = w.wi < nsb ? w.set : groups, psb = w.wi, pslot = 0;
    auto prefetch = [&]() {
        if (pg < groups) {
            const int r0 = row_begin + pg * 16;
            stream.issue(w.slot(pslot), w_base + static_cast<uintptr_t>(r0) * row_bytes + static_cast<uint32_t>(psb * D::kBytes), row_end - r0,
                         w_end, policy);
            psb += g.wpg;
            if (psb >= nsb) {
                psb = w.wi;
                pg += nsets;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (++pslot == w.depth) pslot = 0;
    };
    for (int i = 0; i + 1 < w.depth; ++i) prefetch();

    if (a.dep_mode != 2) pdl_wait_prior();
    if (a.dep_mode == 1) pdl_launch_dependents();
    if (Am) mma_image_bf16<D>(smem, Am, Mm, a.K, sb0 * 8, nsb * 8, tid, kMmaThreads);
    else mma_image_q8_1<D>(smem, xqm, Mm, a.K / 32, sb0 * 8, nsb * 8, tid, kMmaThreads);
    __syncthreads();

    auto run = [&](auto odd) {
        constexpr bool ODD = decltype(odd)::value;
        int slot = 0, buf = 0, gi = w.set;
        for (int c0 = 0; c0 < groups; c0 += g.chunk) {   // the same chunks in every CTA of the cluster
            const int c1 = min(groups, c0 + g.chunk);
            for (; gi < c1; gi += nsets, buf ^= 1) {
                const int r0 = row_begin + gi * 16;
                float acc[16] = {};
                for (int sb = w.wi; sb < nsb; sb += g.wpg) {
                    prefetch();
                    mma_wait_block(w.depth);
                    __syncwarp();
                    w.template multiply<ODD>(slot, sb, static_cast<uint32_t>(w_base) + static_cast<uint32_t>(r0) * row_bytes + static_cast<uint32_t>(sb * D::kBytes),
                                             row_bytes, acc);
                    __syncwarp();   // every lane has read the slot before it is filled again
                    if (++slot == w.depth) slot = 0;
                }
                mma_add_tiles<D, ODD>(g, part, w.set, buf, w.wi, w.lane, acc, [&](int r, int m, float v) {
                    if (g.ksplit > 1) sums[((gi - c0) * 16 + r) * 8 + m] = v;
                    else if (m < Mm && r0 + r < row_end) store_out(Cm, a.out_f32, static_cast<size_t>(m) * ldcm + r0 + r, v);
                });
            }
            if (g.ksplit > 1) {
                __syncwarp();
                mma_cluster_sync();
                const uint32_t base = smem_u32(sums);
                const int first = row_begin + c0 * 16, rows = min(row_end - first, (c1 - c0) * 16);
                for (int i = rank * kMmaThreads + tid; i < rows * Mm; i += g.ksplit * kMmaThreads) {
                    const int m = i / rows, r = i - m * rows;
                    const uint32_t at = base + static_cast<uint32_t>(r * 8 + m) * 4u;
                    const float v = mma_sum8(g.ksplit, [&](int k) { return mma_ld_cluster(at, k); });
                    store_out(Cm, a.out_f32, static_cast<size_t>(m) * ldcm + first + r, v);
                }
                __syncwarp();
                mma_cluster_sync();   // no CTA leaves, or writes the next chunk, while a peer still reads its sums
            }
        }
    };
    if (mma_step(Mm) == 2) run(MmaFlag<false>{});
    else run(MmaFlag<true>{});
    if (a.dep_mode == 2) pdl_wait_prior();
}

// Grouped (MoE) form: the segments of the device-built list (expert, first row, up to eight rows)
// times the expert's row groups are one virtual space, cut into equal contiguous ranges of row
// groups, one per persistent CTA.  A CTA rebuilds its activation image where its range crosses
// into another segment, while the copies of the next blocks are under way; row groups go to the
// sets round robin across segments.  K fits one CTA (no clusters).
template <int T>
__global__ void __launch_bounds__(kMmaThreads, 1) mmvq_mma_grouped_kernel(const MmaGroupedArgs args) {
    using D = MmaDec<T>;
    const GroupedArgs& a = args.v;
    const MmaCut& g = args.c;
    extern __shared__ __align__(128) uint8_t smem[];
    float* part = reinterpret_cast<float*>(smem + g.part_off);
    pdl_launch_dependents();
    pdl_wait_prior();   // the segment list and the activations come from earlier kernels

    const int gn = (a.N + 15) >> 4;   // row groups of an expert
    // CTA b: quotient row groups, and one of the remainder.  Divisions in 32 bits where that is enough:
    // four of 64 bits in a row stand in front of the first load.
    const auto div = [](unsigned long long n, uint32_t d) {
        return (n >> 32) == 0 ? static_cast<unsigned long long>(static_cast<uint32_t>(n) / d) : n / d;
    };
    const unsigned long long V = static_cast<unsigned long long>(a.seg[0]) * gn;
    const unsigned long long vq = div(V, gridDim.x);
    const uint32_t vr = static_cast<uint32_t>(V - vq * gridDim.x);
    const unsigned long long vb = vq * blockIdx.x + min(blockIdx.x, vr);
    const int total = static_cast<int>(vq) + (blockIdx.x < vr ? 1 : 0);   // row groups of this CTA
    if (total == 0) return;
    const int sg0 = static_cast<int>(div(vb, gn)), first0 = static_cast<int>(vb - static_cast<unsigned long long>(sg0) * gn);

    const MmaWarp<D> w(g, smem, g.nsb * 8);
    const int nsets = kMmaWarps / g.wpg;
    const uint32_t row_bytes = static_cast<uint32_t>(a.row_bytes);
    const MmaStream<D> stream(row_bytes, w.lane);
    const uint64_t policy = l2_policy_evict_first();

    // The stream's cursor: row group pn of the range (pgi of segment psg, whose matrix is at base),
    // block psb of it.
    int pn = w.wi < g.nsb ? w.set : total, psg = sg0, pgi = first0 + w.set, psb = w.wi, pslot = 0;
    uintptr_t base = 0;
    auto locate = [&]() {
        while (pgi >= gn) {
            pgi -= gn;
            ++psg;
        }
        base = reinterpret_cast<uintptr_t>(a.B_ptrs[a.seg[1 + 3 * psg]]);
    };
    if (pn < total) locate();
    auto prefetch = [&]() {
        if (pn < total) {
            // a matrix off a 16-byte boundary is moved byte by byte rather than read before its start
            const uintptr_t end = (base & 15) ? 0 : (base + static_cast<uintptr_t>(a.N) * row_bytes) & ~uintptr_t(15);
            stream.issue(w.slot(pslot), base + static_cast<uintptr_t>(pgi * 16) * row_bytes + static_cast<uint32_t>(psb * D::kBytes),
                         a.N - pgi * 16, end, policy);
            psb += g.wpg;
            if (psb >= g.nsb) {
                psb = w.wi;
                pn += nsets;
                pgi += nsets;
                if (pgi >= gn && pn < total) locate();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (++pslot == w.depth) pslot = 0;
    };
    for (int i = 0; i + 1 < w.depth; ++i) prefetch();

    int slot = 0, buf = 0, next = w.set;   // next: this set's next row group of the range
    int done = 0;                          // row groups of the segments before this one
    for (int sg = sg0, first = first0; done < total; ++sg, first = 0) {
        const int last = min(gn, first + total - done);
        const int arow0 = a.seg[2 + 3 * sg], mcount = a.seg[3 + 3 * sg];
        const uint32_t w_lo = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(a.B_ptrs[a.seg[1 + 3 * sg]]));
        if (done > 0) __syncthreads();   // the previous image is no longer read
        mma_image_q8_1<D>(smem, a.xq + static_cast<size_t>(arow0) * (a.K / 32) * kQ8_1Bytes, mcount, a.K / 32, 0, g.nsb * 8, threadIdx.x,
                          kMmaThreads);
        __syncthreads();
        auto run = [&](auto odd) {
            constexpr bool ODD = decltype(odd)::value;
            for (; next < done + last - first; next += nsets, buf ^= 1) {
                const int r0 = (first + next - done) * 16;
                float acc[16] = {};
                for (int sb = w.wi; sb < g.nsb; sb += g.wpg) {
                    prefetch();
                    mma_wait_block(w.depth);
                    __syncwarp();
                    w.template multiply<ODD>(slot, sb, w_lo + static_cast<uint32_t>(r0) * row_bytes + static_cast<uint32_t>(sb * D::kBytes), row_bytes, acc);
                    __syncwarp();
                    if (++slot == w.depth) slot = 0;
                }
                mma_add_tiles<D, ODD>(g, part, w.set, buf, w.wi, w.lane, acc, [&](int r, int m, float v) {
                    if (m < mcount && r0 + r < a.N) store_out(a.D, a.out_f32, static_cast<size_t>(arow0 + m) * a.N + r0 + r, v);
                });
            }
        };
        if (mma_step(mcount) == 2) run(MmaFlag<false>{});
        else run(MmaFlag<true>{});
        done += last - first;
    }
}

#endif  // __CUDACC__

}  // namespace lsg
