// GGUF mat-vec for 2 to 8 batch rows on the integer tensor-core instruction (mma.sync s8).
//
// From two batch rows on the mat-vec of mmvq.cuh is bound by its dp4a arithmetic (eight rows of
// Q6_K: a quarter of the copy bandwidth), so here a warp multiplies 16 weight rows by eight
// batch rows: one mma.m16n8k32 (k16 for Q6_K, whose scales cover 16 values) replaces 32 dp4a per
// lane, and with the magic number 1.5 * 2^23 as the initial accumulator its integer result is
// read as a float with one subtraction.  The sums of a scale group are the same exact integers
// as before; the products with the scales and their fp32 sums keep the same terms.
//
// mma.sync and not tcgen05: the sums have to be rescaled every 16 or 32 values of K, and an
// accumulator in tensor memory would be drained as often.  At eight columns the instruction is
// not the limit either (the scale arithmetic around it is).
//
//   * The K of an operand fragment may be permuted as long as both operands agree.  Lane (g, t)
//     of the warp takes bytes 8t..8t+7 of the packed 32 bytes of rows g and g + 8 (one 8-byte
//     load, low nibbles = one scale group, high nibbles = the next) and the activation image
//     keeps a block of eight columns x 32 codes so that the matching operand is one 8-byte load.
//   * A stage of the ring holds 16 rows x up to eight super-blocks, one bulk copy per row.  The
//     rows' pitch is chosen so that the eight rows of a fragment load hit different banks; that
//     is why the rows are copied one by one.
//   * `wpg` warps share a row group, warp i taking super-block i of every stage; their partial
//     16 x 8 tiles are added in warp order through shared memory.  16 / wpg groups are in work at
//     a time, each with a ring of its own, so a warp meets every lap of the ring it waits on.
//   * Long rows are split along K over the CTAs of a cluster (4096 values each): a CTA then
//     quantizes and holds only its part of the activations, and the cluster has more rows.
//     The CTAs add their sums in rank order through distributed shared memory.
// How K is cut depends on K and the type alone, so a result does not depend on the number of
// weight rows, on what shares the launch, or on the launch geometry.
#pragma once

#include "mmvq_grouped.cuh"

namespace lsg {

constexpr int kMmaWarps = 16;                         // consumer warps
constexpr int kMmaThreads = (kMmaWarps + 1) * 32;
constexpr int kMmaCols = 8;                           // batch rows of one launch
constexpr int kMmaSliceBlocks = 16;                   // super-blocks of one CTA's share of K, at most
constexpr int kMmaMaxRing = 8;                        // stages of one row group's ring

// How a row is cut and where things lie in shared memory.
struct MmaCut {
    int sb_bytes;        // bytes of 256 packed values
    int nsb;             // 256-value blocks of a row
    int ksplit, slice;   // CTAs of a cluster along K, blocks of each
    int nc, chunk;       // stages per row group, blocks of a stage
    int wpg;             // warps of a row group
    int ring;            // stages of a row group's ring
    int pitch;           // bytes between the rows of a stage
    int img_bytes, part_off, sum_off, bar_off;   // image, ring, partial tiles, cluster sums, barriers
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

__device__ __forceinline__ void mma_u8s8_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_s8s8_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_s8s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0));
}

// An integer of magnitude below 2^22 added to this bit pattern is that integer as a float, offset
// by kMmaBias; the largest sum here is 32 * 128 * 127.
constexpr int kMmaBiasBits = 0x4B400000;
constexpr float kMmaBias = 12582912.0f;
__device__ __forceinline__ void mma_zero(int (&c)[4]) { c[0] = c[1] = c[2] = c[3] = kMmaBiasBits; }
__device__ __forceinline__ float mma_val(int c) { return __int_as_float(c) - kMmaBias; }
// Byte k of w as a float (unsigned; or signed after its sign bit has been flipped).
__device__ __forceinline__ float byte_f(uint32_t w, int k) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7550u | k)) - 8388608.0f;
}
__device__ __forceinline__ float sbyte_f(uint32_t w_flipped, int k) {
    return __uint_as_float(__byte_perm(w_flipped, 0x4B000000u, 0x7550u | k)) - 8388736.0f;
}
__device__ __forceinline__ uint32_t lds_word_unaligned(uint32_t addr) {
    const uint32_t b = addr & ~3u;
    return __funnelshift_r(lds32(b), lds32(b + 4), (addr & 3u) * 8u);
}

// tile(): acc[i] += the products of one 256-value block: rows r0 (accumulators 0, 1) and r1 (2, 3)
// with columns 2t and 2t + 1.
//   r0, r1  shared addresses of the block in rows g and g + 8
//   xq      codes of this lane's column g: block j of the 256 values at xq + 256 j, lane offset in
//   xs      scales (with the block sum where kSums) of columns 2t, 2t + 1: block j at xs + j * 64 or 32
// kHalves: the words of a block's two 16-value halves alternate in the image.
template <bool FIVE> struct MmaDecK45 {   // Q4_K, Q5_K
    static constexpr bool kHas = true;
    static constexpr bool kSums = true, kHalves = false;
    static constexpr int kBytes = FIVE ? 176 : 144;
    static constexpr int kPitchMod = 64, kPitchRem = 32;   // 8-byte loads of eight rows: no bank twice

    __device__ static __forceinline__ void tile(uint32_t r0, uint32_t r1, int t, uint32_t xq, uint32_t xs,
                                                float (&acc)[4]) {
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
        float s1[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
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
                const uint4 xv = lds128(xs + 64 * j);
                const float dx0 = __uint_as_float(xv.x), sx0 = __uint_as_float(xv.y);
                const float dx1 = __uint_as_float(xv.z), sx1 = __uint_as_float(xv.w);
                int c[4];
                mma_zero(c);
                mma_u8s8_k32(c, a0, a1, a2, a3, xb.x, xb.y);
                const float c0 = byte_f(sc0[j >> 2], j & 3), c1 = byte_f(sc1[j >> 2], j & 3);
                const float m0 = byte_f(mn0[j >> 2], j & 3), m1 = byte_f(mn1[j >> 2], j & 3);
                s1[0] = fmaf(dx0, mma_val(c[0]) * c0, s1[0]);   // integer products below 2^24: exact
                s1[1] = fmaf(dx1, mma_val(c[1]) * c0, s1[1]);
                s1[2] = fmaf(dx0, mma_val(c[2]) * c1, s1[2]);
                s1[3] = fmaf(dx1, mma_val(c[3]) * c1, s1[3]);
                s2[0] = fmaf(m0, sx0, s2[0]);
                s2[1] = fmaf(m0, sx1, s2[1]);
                s2[2] = fmaf(m1, sx0, s2[2]);
                s2[3] = fmaf(m1, sx1, s2[3]);
            }
        }
        const float d0 = fp16_bits_to_float(h0.x), e0 = fp16_bits_to_float(h0.x >> 16);
        const float d1 = fp16_bits_to_float(h1.x), e1 = fp16_bits_to_float(h1.x >> 16);
        acc[0] += d0 * s1[0] - e0 * s2[0];
        acc[1] += d0 * s1[1] - e0 * s2[1];
        acc[2] += d1 * s1[2] - e1 * s2[2];
        acc[3] += d1 * s1[3] - e1 * s2[3];
    }
};
template <> struct MmaDec<LSG_GGUF_Q4_K> : MmaDecK45<false> {};
template <> struct MmaDec<LSG_GGUF_Q5_K> : MmaDecK45<true> {};

template <> struct MmaDec<LSG_GGUF_Q6_K> {
    static constexpr bool kHas = true;
    static constexpr bool kSums = false, kHalves = true;
    static constexpr int kBytes = 210;
    static constexpr int kPitchMod = 32, kPitchRem = 16;   // 4-byte loads of eight rows

    // four 6-bit values 0..63 -> value - 32 as signed bytes
    __device__ static __forceinline__ uint32_t sext6(uint32_t v) {
        const uint32_t x = v ^ 0x20202020u;
        return x | ((x & 0x20202020u) * 6u);
    }
    __device__ static __forceinline__ void tile(uint32_t r0, uint32_t r1, int t, uint32_t xq, uint32_t xs,
                                                float (&acc)[4]) {
        const uint32_t row[2] = {r0, r1};
        uint32_t scw[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            lds_words_unaligned<4>(row[r] + 192, scw[r]);
#pragma unroll
            for (int i = 0; i < 4; ++i) scw[r][i] ^= 0x80808080u;
        }
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ip = 0; ip < 2; ++ip) {
            uint32_t la[2][2], lb[2][2], qh[2][2];   // [row][16-value half]
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int hs = 0; hs < 2; ++hs) {
                    la[r][hs] = lds_word_unaligned(row[r] + 64 * ip + 16 * hs + 4 * t);
                    lb[r][hs] = lds_word_unaligned(row[r] + 64 * ip + 32 + 16 * hs + 4 * t);
                    qh[r][hs] = lds_word_unaligned(row[r] + 128 + 32 * ip + 16 * hs + 4 * t);
                }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint2 xb = lds64(xq + 256 * (4 * ip + q));
                const uint2 xv = lds64(xs + 32 * (4 * ip + q));
                float f[2][4];
#pragma unroll
                for (int hs = 0; hs < 2; ++hs) {
                    uint32_t a[2];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const uint32_t lo = ((q & 1) ? lb[r][hs] : la[r][hs]) >> (4 * (q >> 1));
                        const uint32_t hi = q == 0 ? qh[r][hs] << 4 : (q == 1 ? qh[r][hs] << 2 : (q == 2 ? qh[r][hs] : qh[r][hs] >> 2));
                        a[r] = sext6((lo & 0x0F0F0F0Fu) | (hi & 0x30303030u));
                    }
                    int c[4];
                    mma_zero(c);
                    mma_s8s8_k16(c, a[0], a[1], hs ? xb.y : xb.x);
#pragma unroll
                    for (int i = 0; i < 4; ++i) f[hs][i] = mma_val(c[i]);
                }
                const int e = 8 * ip + 2 * q;
                const float dx0 = __uint_as_float(xv.x), dx1 = __uint_as_float(xv.y);
                // both halves' integer products together stay below 2^24: exact
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float sa = sbyte_f(scw[r][e >> 2], e & 3), sb = sbyte_f(scw[r][(e + 1) >> 2], (e + 1) & 3);
                    s[2 * r] = fmaf(dx0, fmaf(f[1][2 * r], sb, f[0][2 * r] * sa), s[2 * r]);
                    s[2 * r + 1] = fmaf(dx1, fmaf(f[1][2 * r + 1], sb, f[0][2 * r + 1] * sa), s[2 * r + 1]);
                }
            }
        }
        const float d0 = fp16_bits_to_float(lds16(r0 + 208)), d1 = fp16_bits_to_float(lds16(r1 + 208));
        acc[0] += d0 * s[0];
        acc[1] += d0 * s[1];
        acc[2] += d1 * s[2];
        acc[3] += d1 * s[3];
    }
};

template <> struct MmaDec<LSG_GGUF_Q8_0> {   // eight 34-byte blocks
    static constexpr bool kHas = true;
    static constexpr bool kSums = false, kHalves = false;
    static constexpr int kBytes = 272;
    static constexpr int kPitchMod = 64, kPitchRem = 32;

    __device__ static __forceinline__ void tile(uint32_t r0, uint32_t r1, int t, uint32_t xq, uint32_t xs,
                                                float (&acc)[4]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            uint32_t w0[2], w1[2];
            lds_words_unaligned<2>(r0 + 34 * j + 2 + 8 * t, w0);
            lds_words_unaligned<2>(r1 + 34 * j + 2 + 8 * t, w1);
            const uint2 xb = lds64(xq + 256 * j);
            const uint2 xv = lds64(xs + 32 * j);
            int c[4];
            mma_zero(c);
            mma_s8s8_k32(c, w0[0], w1[0], w0[1], w1[1], xb.x, xb.y);
            const float d0 = fp16_bits_to_float(lds16(r0 + 34 * j)), d1 = fp16_bits_to_float(lds16(r1 + 34 * j));
            const float dx0 = __uint_as_float(xv.x), dx1 = __uint_as_float(xv.y);
            acc[0] = fmaf(d0 * dx0, mma_val(c[0]), acc[0]);
            acc[1] = fmaf(d0 * dx1, mma_val(c[1]), acc[1]);
            acc[2] = fmaf(d1 * dx0, mma_val(c[2]), acc[2]);
            acc[3] = fmaf(d1 * dx1, mma_val(c[3]), acc[3]);
        }
    }
};

template <> struct MmaDec<LSG_GGUF_Q4_0> {   // eight 18-byte blocks; byte i: values i and i + 16
    static constexpr bool kHas = true;
    static constexpr bool kSums = false, kHalves = true;
    static constexpr int kBytes = 144;
    static constexpr int kPitchMod = 32, kPitchRem = 16;

    // four nibbles 0..15 -> value - 8 as signed bytes
    __device__ static __forceinline__ uint32_t sext4(uint32_t v) {
        const uint32_t x = v ^ 0x08080808u;
        return x | ((x & 0x08080808u) * 30u);
    }
    __device__ static __forceinline__ void tile(uint32_t r0, uint32_t r1, int t, uint32_t xq, uint32_t xs,
                                                float (&acc)[4]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t w0 = lds_word_unaligned(r0 + 18 * j + 2 + 4 * t);
            const uint32_t w1 = lds_word_unaligned(r1 + 18 * j + 2 + 4 * t);
            const uint2 xb = lds64(xq + 256 * j);
            const uint2 xv = lds64(xs + 32 * j);
            int c[4];
            mma_zero(c);
            mma_s8s8_k32(c, sext4(w0 & 0x0F0F0F0Fu), sext4(w1 & 0x0F0F0F0Fu), sext4((w0 >> 4) & 0x0F0F0F0Fu),
                         sext4((w1 >> 4) & 0x0F0F0F0Fu), xb.x, xb.y);
            const float d0 = fp16_bits_to_float(lds16(r0 + 18 * j)), d1 = fp16_bits_to_float(lds16(r1 + 18 * j));
            const float dx0 = __uint_as_float(xv.x), dx1 = __uint_as_float(xv.y);
            acc[0] = fmaf(d0 * dx0, mma_val(c[0]), acc[0]);
            acc[1] = fmaf(d0 * dx1, mma_val(c[1]), acc[1]);
            acc[2] = fmaf(d1 * dx0, mma_val(c[2]), acc[2]);
            acc[3] = fmaf(d1 * dx1, mma_val(c[3]), acc[3]);
        }
    }
};

// ---------------------------------------------------------------------------
// Activation image of `nblk` 32-value blocks from block b0 on, eight columns (batch rows from M
// on are zeros):  codes [block][column][32], then scales [block][column]{d} or {d, d * sum}.
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
template <class D>
__device__ __forceinline__ void mma_put_scale(uint8_t* img, int nblk, int b, int col, float d, int sum) {
    float* s = reinterpret_cast<float*>(img + nblk * 256);
    if (D::kSums) {
        *reinterpret_cast<float2*>(s + (b * 8 + col) * 2) = make_float2(d, d * static_cast<float>(sum));
    } else {
        s[b * 8 + col] = d;
    }
}

template <class D>
__device__ __forceinline__ void mma_image_q8_1(uint8_t* img, const uint8_t* __restrict__ xq, int M, int row_blocks,
                                               int b0, int nblk, int tid, int nthreads) {
    for (int idx = tid; idx < kMmaCols * nblk; idx += nthreads) {
        const int m = idx / nblk, b = idx - m * nblk;
        uint32_t w[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if (m < M) {
            const uint32_t* src = reinterpret_cast<const uint32_t*>(xq + (static_cast<size_t>(m) * row_blocks + b0 + b) * kQ8_1Bytes);
#pragma unroll
            for (int i = 0; i < 9; ++i) w[i] = __ldg(src + i);
        }
        int sum = 0;
#pragma unroll
        for (int i = 1; i < 9; ++i) sum = __dp4a(static_cast<int>(w[i]), 0x01010101, sum);
        mma_put_half<D>(img, b, m, 0, make_uint4(w[1], w[2], w[3], w[4]));
        mma_put_half<D>(img, b, m, 1, make_uint4(w[5], w[6], w[7], w[8]));
        mma_put_scale<D>(img, nblk, b, m, fp16_bits_to_float(w[0]), sum);
    }
}

// The same from bf16 activations, two lanes per block (the quantizer of build_x_image_bf16).
template <class D>
__device__ __forceinline__ void mma_image_bf16(uint8_t* img, const __nv_bfloat16* __restrict__ A, int M, int K, int b0,
                                               int nblk, int tid, int nthreads) {
    const int total = kMmaCols * nblk * 2;   // a multiple of 32, as nthreads: no warp is split by the loop
    for (int idx = tid; idx < total; idx += nthreads) {
        const int half = idx & 1, task = idx >> 1;
        const int m = task / nblk, b = task - m * nblk;
        uint4 r0 = make_uint4(0, 0, 0, 0), r1 = r0;
        if (m < M) {
            const uint4* src = reinterpret_cast<const uint4*>(A + static_cast<size_t>(m) * K + static_cast<size_t>(b0 + b) * 32 + 16 * half);
            r0 = __ldg(src);
            r1 = __ldg(src + 1);
        }
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
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        mma_put_half<D>(img, b, m, half, q);
        if (half == 0) mma_put_scale<D>(img, nblk, b, m, __half2float(__float2half(d)), sum);
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

// One stage: `nrows` rows of `bytes` packed bytes each, row r at src + r * row_bytes, into the
// stage at `pitch`.  `shifted`: a row keeps its offset from a 16-byte boundary (the types whose
// blocks are not whole 16-byte pieces).  Bulk copies take whole 16-byte pieces; what a row holds
// behind the last whole piece of the matrix (w_end_al), and all of it when the matrix itself is
// not 16-byte aligned (w_end_al = 0), is moved with byte loads.  Called by a converged warp.
__device__ __forceinline__ void mma_copy_stage(uint8_t* dst, uintptr_t src, int nrows, long long row_bytes, int bytes,
                                               int pitch, uintptr_t w_end_al, bool shifted, uint64_t* bar, uint64_t policy) {
    const int lane = threadIdx.x & 31;
    const uintptr_t my_b = src + static_cast<uintptr_t>(lane < nrows ? lane : 0) * row_bytes, my_e = my_b + bytes;
    const uintptr_t at_b = shifted ? my_b & ~uintptr_t(15) : my_b;   // what the row's place in the stage stands for
    uintptr_t cp_e = (my_e + 15) & ~uintptr_t(15);
    if (cp_e > w_end_al) cp_e = w_end_al > at_b ? w_end_al : at_b;
    const uint32_t mine = lane < nrows ? static_cast<uint32_t>(cp_e - at_b) : 0u;
    const uint32_t all = __reduce_add_sync(0xffffffffu, mine);
    if (lane < nrows)
        for (uintptr_t p = mine > 0 ? cp_e : my_b; p < my_e; ++p)
            dst[lane * pitch + (p - at_b)] = *reinterpret_cast<const uint8_t*>(p);
    __syncwarp();
    if (elect_one_lane()) mbar_arrive_expect_tx(bar, all);
    __syncwarp();
    if (mine > 0) bulk_g2s_hint(dst + lane * pitch, reinterpret_cast<const void*>(at_b), mine, bar, policy);
    __syncwarp();
}

// One warp's part of a row group: block `wi` of each of its stages, the partial tile left in
// mine[16 rows][8 columns].  lo0: low bits of the address of the group's first row, at this CTA's
// first block.  s, phase: the warp's position in its set's ring.
template <class D>
__device__ __forceinline__ void mma_row_group(const MmaCut& g, int lane, int wi, uint32_t lo0, uint32_t row_bytes, int nsb,
                                              uint32_t xq0, uint32_t xs0, uint32_t ring0, uint64_t* full, uint64_t* empty,
                                              int& s, uint32_t& phase, volatile int* abort_flag, unsigned int* status,
                                              long long wait_limit, float* mine) {
    constexpr int kScaleBytes = D::kSums ? 64 : 32;
    const int gl = lane >> 2, t = lane & 3;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < g.nc; ++c) {
        // After a wait has run out the warps keep walking (the barriers of their set need every
        // warp) but neither wait nor compute.
        bool ok = *abort_flag == 0;
        ok = __all_sync(0xffffffffu, ok && mbar_wait_bounded(&full[s], phase, status, kDevWaitFull, 2000u, wait_limit));
        if (!ok) *abort_flag = 1;
        const int sb = c * g.chunk + wi;
        if (ok && wi < g.chunk && sb < nsb) {
            uint32_t p0 = ring0 + static_cast<uint32_t>(s * 16 + gl) * g.pitch + wi * D::kBytes, p1 = p0 + 8 * g.pitch;
            if (D::kBytes % 16 != 0) {   // rows may start off a 16-byte boundary
                const uint32_t lo = lo0 + static_cast<uint32_t>(gl) * row_bytes + static_cast<uint32_t>(c * g.chunk) * D::kBytes;
                p0 += lo & 15u;
                p1 += (lo + 8u * row_bytes) & 15u;
            }
            D::tile(p0, p1, t, xq0 + sb * 2048, xs0 + sb * 8 * kScaleBytes, acc);
        }
        __syncwarp();
        if (elect_one_lane()) mbar_arrive(&empty[s]);
        if (++s == g.ring) {
            s = 0;
            phase ^= 1;
        }
    }
    *reinterpret_cast<float2*>(mine + gl * 8 + 2 * t) = make_float2(acc[0], acc[1]);
    *reinterpret_cast<float2*>(mine + (gl + 8) * 8 + 2 * t) = make_float2(acc[2], acc[3]);
}

template <int T>
__global__ void __launch_bounds__(kMmaThreads, 1) mmvq_mma_kernel(const MmaArgs args) {
    using D = MmaDec<T>;
    const MmvqArgs& a = args.v;
    const MmaCut& g = args.c;
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* ring = smem + g.img_bytes;
    float* part = reinterpret_cast<float*>(smem + g.part_off);     // [set][2][wpg][16 rows][8]
    float* sums = reinterpret_cast<float*>(smem + g.sum_off);      // [row][8], with ksplit > 1
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + g.bar_off);
    const int nsets = kMmaWarps / g.wpg;
    uint64_t* empty = full + nsets * g.ring;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + nsets * g.ring);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = static_cast<int>(blockIdx.x) % g.ksplit;
    int bx = static_cast<int>(blockIdx.x) / g.ksplit;
    const uint8_t* Wm = a.W;
    const __nv_bfloat16* Am = a.A;
    const uint8_t* xqm = a.xq;
    void* Cm = a.C;
    int Nm = a.N, ldcm = a.ldc, rows_q = a.rows_q, rows_r = a.rows_r;
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
    const int stage_bytes = 16 * g.pitch;

    if (tid < nsets * g.ring) {
        mbar_init(&full[tid], 1);
        mbar_init(&empty[tid], g.wpg);
        mbar_fence_init();
    }
    if (tid == 0) *abort_flag = 0;
    __syncthreads();
    if (a.dep_mode != 1) pdl_launch_dependents();

    const uintptr_t w_base = reinterpret_cast<uintptr_t>(Wm);
    if (warp == kMmaWarps) {
        // ------------------------------ producer ------------------------------
        const uint64_t policy = l2_policy_evict_first();
        const uintptr_t w_end_al = (w_base + static_cast<uintptr_t>(Nm) * a.row_bytes) & ~uintptr_t(15);
        bool released = a.dep_mode != 1;
        bool ok = true;
        int slot = 0;        // ring position, the same in every set's ring
        uint32_t lap = 0;
        for (int g0 = 0; g0 < groups && ok; g0 += nsets) {
            for (int c = 0; c < g.nc && ok; ++c) {
                const int cb = min(g.chunk, nsb - c * g.chunk);   // blocks of the stage, may be 0 or less
                for (int h = 0; h < nsets && g0 + h < groups; ++h) {
                    const int s = h * g.ring + slot;
                    if (lap > 0) {
                        // first launch of a batch whose later launches do not wait: release them once
                        // the ring is full and the work in front of the batch has completed
                        if (!released) {
                            pdl_wait_prior();
                            pdl_launch_dependents();
                            released = true;
                        }
                        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty[s], (lap - 1) & 1, a.status, kDevWaitEmpty, 2000u, a.wait_limit));
                        if (!ok) break;
                    }
                    const int r0 = row_begin + (g0 + h) * 16;
                    const int nrows = min(16, row_end - r0);
                    if (cb > 0)
                        mma_copy_stage(ring + static_cast<size_t>(s) * stage_bytes,
                                       w_base + static_cast<uintptr_t>(r0) * a.row_bytes + static_cast<uintptr_t>(sb0 + c * g.chunk) * g.sb_bytes,
                                       nrows, a.row_bytes, cb * g.sb_bytes, g.pitch, w_end_al, D::kBytes % 16 != 0, &full[s], policy);
                    else if (elect_one_lane())
                        mbar_arrive(&full[s]);
                    __syncwarp();
                }
                if (++slot == g.ring) {
                    slot = 0;
                    ++lap;
                }
            }
        }
        if (!ok) *abort_flag = 1;
        if (!released) {
            pdl_wait_prior();
            pdl_launch_dependents();
        }
    } else {
        // ------------------------------ consumers ------------------------------
        const int n_cons = kMmaWarps * 32;
        if (a.dep_mode != 2) pdl_wait_prior();
        if (a.dep_mode == 1) pdl_launch_dependents();
        const int nblk = nsb * 8;
        if (Am) mma_image_bf16<D>(smem, Am, a.M, a.K, sb0 * 8, nblk, tid, n_cons);
        else mma_image_q8_1<D>(smem, xqm, a.M, a.K / 32, sb0 * 8, nblk, tid, n_cons);
        asm volatile("bar.sync 1, %0;" ::"r"(n_cons) : "memory");

        const int set = warp / g.wpg, wi = warp - set * g.wpg;
        const int set_tid = wi * 32 + lane;
        const uint32_t img = smem_u32(smem);
        const uint32_t xq0 = img + (lane >> 2) * 32 + 8 * (lane & 3);
        const uint32_t xs0 = img + nblk * 256 + (lane & 3) * (D::kSums ? 16 : 8);
        const uint32_t ring0 = smem_u32(ring) + static_cast<uint32_t>(set * g.ring) * stage_bytes;
        int s = 0, buf = 0;
        uint32_t phase = 0;
        for (int gi = set; gi < groups; gi += nsets, buf ^= 1) {
            const int r0 = row_begin + gi * 16;
            mma_row_group<D>(g, lane, wi, static_cast<uint32_t>(w_base) + static_cast<uint32_t>(r0) * static_cast<uint32_t>(a.row_bytes) +
                                              static_cast<uint32_t>(sb0) * D::kBytes,
                             static_cast<uint32_t>(a.row_bytes), nsb, xq0, xs0, ring0, full + set * g.ring, empty + set * g.ring, s,
                             phase, abort_flag, a.status, a.wait_limit, part + ((set * 2 + buf) * g.wpg + wi) * 128);
            asm volatile("bar.sync %0, %1;" ::"r"(2 + set), "r"(g.wpg * 32) : "memory");
            const float* all = part + (set * 2 + buf) * g.wpg * 128;
            for (int i = set_tid; i < 128; i += g.wpg * 32) {
                const int col = i >> 4, r = i & 15;
                float v = all[r * 8 + col];
                for (int w = 1; w < g.wpg; ++w) v += all[w * 128 + r * 8 + col];
                if (g.ksplit > 1) sums[(gi * 16 + r) * 8 + col] = v;
                else if (col < a.M && r0 + r < row_end) store_out(Cm, a.out_f32, static_cast<size_t>(col) * ldcm + r0 + r, v);
            }
        }
    }
    if (g.ksplit > 1) {
        __syncwarp();
        mma_cluster_sync();
        const uint32_t base = smem_u32(sums);
        const int rows = row_end - row_begin;
        for (int i = rank * kMmaThreads + tid; i < rows * a.M; i += g.ksplit * kMmaThreads) {
            const int col = i / rows, r = i - col * rows;
            const uint32_t at = base + static_cast<uint32_t>(r * 8 + col) * 4u;
            float v = mma_ld_cluster(at, 0);
            for (int k = 1; k < g.ksplit; ++k) v += mma_ld_cluster(at, k);
            store_out(Cm, a.out_f32, static_cast<size_t>(col) * ldcm + row_begin + r, v);
        }
        __syncwarp();
        mma_cluster_sync();   // no CTA leaves while a peer still reads its sums
    }
    if (a.dep_mode == 2) pdl_wait_prior();
}

// Grouped (MoE) form: the segments of the device-built list (expert, first row, up to eight rows)
// times the expert's row groups are one virtual space, cut into equal contiguous ranges of row
// groups, one per persistent CTA.  A CTA rebuilds its activation image where its range crosses
// into another segment; row groups go to the sets round robin across segments, so every set's
// ring is one sequence.  K fits one CTA's share (no clusters).
template <int T>
__global__ void __launch_bounds__(kMmaThreads, 1) mmvq_mma_grouped_kernel(const MmaGroupedArgs args) {
    using D = MmaDec<T>;
    const GroupedArgs& a = args.v;
    const MmaCut& g = args.c;
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* ring = smem + g.img_bytes;
    float* part = reinterpret_cast<float*>(smem + g.part_off);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + g.bar_off);
    const int nsets = kMmaWarps / g.wpg;
    uint64_t* empty = full + nsets * g.ring;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + nsets * g.ring);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int stage_bytes = 16 * g.pitch;
    if (tid < nsets * g.ring) {
        mbar_init(&full[tid], 1);
        mbar_init(&empty[tid], g.wpg);
        mbar_fence_init();
    }
    if (tid == 0) *abort_flag = 0;
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait_prior();   // the segment list and the activations come from earlier kernels

    const int gn = (a.N + 15) >> 4;   // row groups of an expert
    const long long V = static_cast<long long>(a.seg[0]) * gn;
    const long long vb = V * blockIdx.x / gridDim.x, ve = V * (blockIdx.x + 1) / gridDim.x;

    if (warp == kMmaWarps) {
        const uint64_t policy = l2_policy_evict_first();
        bool ok = true;
        int slot0 = 0, set = 0;   // ring position of the round's first stage, set of the next row group
        uint32_t lap0 = 0;
        for (long long cur = vb; cur < ve && ok;) {
            const int sg = static_cast<int>(cur / gn);
            const int first = static_cast<int>(cur - static_cast<long long>(sg) * gn);
            const int last = static_cast<int>(min(static_cast<long long>(gn), first + (ve - cur)));
            const uintptr_t w_base = reinterpret_cast<uintptr_t>(a.B_ptrs[a.seg[1 + 3 * sg]]);
            // a matrix off a 16-byte boundary is moved with byte loads rather than read before its start
            const uintptr_t w_end_al = (w_base & 15) ? 0 : (w_base + static_cast<uintptr_t>(a.N) * a.row_bytes) & ~uintptr_t(15);
            for (int gi = first; gi < last && ok; ++gi) {
                int slot = slot0;
                uint32_t lap = lap0;
                for (int c = 0; c < g.nc && ok; ++c) {
                    const int s = set * g.ring + slot;
                    if (lap > 0) {
                        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty[s], (lap - 1) & 1, a.status, kDevWaitEmpty));
                        if (!ok) break;
                    }
                    mma_copy_stage(ring + static_cast<size_t>(s) * stage_bytes,
                                   w_base + static_cast<uintptr_t>(gi * 16) * a.row_bytes + static_cast<uintptr_t>(c * g.chunk) * g.sb_bytes,
                                   min(16, a.N - gi * 16), a.row_bytes, min(g.chunk, g.nsb - c * g.chunk) * g.sb_bytes, g.pitch,
                                   w_end_al, D::kBytes % 16 != 0, &full[s], policy);
                    if (++slot == g.ring) {
                        slot = 0;
                        ++lap;
                    }
                }
                if (++set == nsets) {
                    set = 0;
                    slot0 = slot;
                    lap0 = lap;
                }
            }
            cur += last - first;
        }
        if (!ok) *abort_flag = 1;
        return;
    }

    const int n_cons = kMmaWarps * 32;
    const int set = warp / g.wpg, wi = warp - set * g.wpg;
    const int set_tid = wi * 32 + lane;
    const int nblk = g.nsb * 8;
    const uint32_t img = smem_u32(smem);
    const uint32_t xq0 = img + (lane >> 2) * 32 + 8 * (lane & 3);
    const uint32_t xs0 = img + nblk * 256 + (lane & 3) * (D::kSums ? 16 : 8);
    const uint32_t ring0 = smem_u32(ring) + static_cast<uint32_t>(set * g.ring) * stage_bytes;
    int s = 0, buf = 0, next = set;   // next: this set's next row group, counted from the range's first
    uint32_t phase = 0;
    int done = 0;                     // row groups of the segments before this one
    for (long long cur = vb; cur < ve;) {
        const int sg = static_cast<int>(cur / gn);
        const int first = static_cast<int>(cur - static_cast<long long>(sg) * gn);
        const int last = static_cast<int>(min(static_cast<long long>(gn), first + (ve - cur)));
        const int arow0 = a.seg[2 + 3 * sg], mcount = a.seg[3 + 3 * sg];
        const uint32_t w_lo = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(a.B_ptrs[a.seg[1 + 3 * sg]]));
        if (done > 0) asm volatile("bar.sync 1, %0;" ::"r"(n_cons) : "memory");   // the previous image is no longer read
        mma_image_q8_1<D>(smem, a.xq + static_cast<size_t>(arow0) * (a.K / 32) * kQ8_1Bytes, mcount, a.K / 32, 0, nblk, tid, n_cons);
        asm volatile("bar.sync 1, %0;" ::"r"(n_cons) : "memory");
        for (; next < done + last - first; next += nsets, buf ^= 1) {
            const int r0 = (first + next - done) * 16;
            mma_row_group<D>(g, lane, wi, w_lo + static_cast<uint32_t>(r0) * static_cast<uint32_t>(a.row_bytes),
                             static_cast<uint32_t>(a.row_bytes), g.nsb, xq0, xs0, ring0, full + set * g.ring, empty + set * g.ring, s,
                             phase, abort_flag, a.status, kWaitLimitCycles, part + ((set * 2 + buf) * g.wpg + wi) * 128);
            asm volatile("bar.sync %0, %1;" ::"r"(2 + set), "r"(g.wpg * 32) : "memory");
            const float* all = part + (set * 2 + buf) * g.wpg * 128;
            for (int i = set_tid; i < 128; i += g.wpg * 32) {
                const int col = i >> 4, r = i & 15;
                float v = all[r * 8 + col];
                for (int w = 1; w < g.wpg; ++w) v += all[w * 128 + r * 8 + col];
                if (col < mcount && r0 + r < a.N) store_out(a.D, a.out_f32, static_cast<size_t>(arow0 + col) * a.N + r0 + r, v);
            }
        }
        done += last - first;
        cur += last - first;
    }
}

#endif  // __CUDACC__

}  // namespace lsg
