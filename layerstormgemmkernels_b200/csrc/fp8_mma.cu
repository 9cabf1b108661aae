// Block-scaled FP8 GEMM on tcgen05.mma.kind::f8f6f4:
//   D[m,n] = sum over 128-wide K blocks kb of  sA[m,kb] * sB[n/128,kb] * sum_{k in kb} a[m,k] * b[n,k]
// a, b e4m3 bytes, the products of one K block summed in fp32 in tensor memory, the scales applied
// in fp32 registers (operand contract: fp8_gemm.cu, launch_fp8_gemm of the reference,
// csrc/sm120/gemm/fp8/fp8_gemm.h:18-44).
//
// The operands are multiplied as they are; the route this replaces for M > 4 first expanded both
// into fp16 with their scales applied (three bytes of extra traffic per value, and one rounding
// per operand) and then ran the fp16 GEMM at half the rate: 2048 x 4096 x 4096 with its activation
// quantizer 98.0 -> 55.1 us.
//
// The scales change every 128 values of K, so the accumulator is drained once per K block: eight
// warps read it out of tensor memory and add it, times its scale, to fp32 accumulators of their
// own, while the tensor core fills the other of two accumulators.  The GEMM alone takes 48 us at
// that size, 39 with the drain left out: the bytes that come out of L2 bound it first (48 KB per K
// block of a 128 x 256 tile at about 42 B/clk and SM, against 512 cycles of tensor time), which is
// why 256 columns are the tile (a narrower one moves more bytes per product), the drain second.
// Sixteen drain warps with half the columns each: 57 us.  K is not split, so few rows leave most SMs
// idle: 5 to 128 x 1024 x 14336 are 8 CTAs and 53 us (84 to 88 on the route this replaced).
//   warps 0-7   drain and epilogue: warp w owns tensor-memory lanes 32 (w % 4).. (= token rows)
//               and column half w / 4; output rows are stored as 16-byte pieces
//   warp 8      TMA producer: one box of 128 tokens x 128 bytes, one of NC weight rows
//   warp 9      MMA issuer: 4 x tcgen05.mma (M = 128, N = NC, K = 32) per K block
// Persistent, one CTA per SM; every wait is time-limited.
#include "common.cuh"
#include "host.h"
#include "tcgen05.cuh"

#include <atomic>

namespace lsg {

using namespace tc;

namespace {

constexpr int kM = 128;                      // token rows of a tile
constexpr int kKB = 128;                     // values (= bytes) of a K block
constexpr int kDrainWarps = 8;
constexpr int kThreads = (kDrainWarps + 2) * 32;

template <int NC> struct Tile {              // NC output columns: 256, or 128
    static constexpr int kStageBytes = (kM + NC) * kKB;
    static constexpr int kStages = NC == 256 ? 4 : 6;
    static constexpr int kSmem = kStages * kStageBytes + 1024 + 256;
};

struct Fp8Args {
    void* D;
    int out_dtype;
    const float* sA;   // [K blocks][M]
    const float* sB;   // [N / 128][K blocks]
    int M, N, kblocks;
    int m_tiles, n_tiles;
    unsigned int* status;
};

__device__ __forceinline__ void tc_mma_f8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Sixteen columns of this thread's tensor-memory lane: thirty-two beside 128 accumulators spill.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

template <int NC>
__global__ void __launch_bounds__(kThreads, 1)
fp8_mma_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Fp8Args a) {
    using L = Tile<NC>;
    constexpr int kStages = L::kStages, kStageBytes = L::kStageBytes;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
    uint64_t* empty = full + kStages;
    uint64_t* acc_full = empty + kStages;    // [2]
    uint64_t* acc_empty = acc_full + 2;      // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], kDrainWarps);
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == kDrainWarps + 1) tmem_alloc(tmem_slot, 2 * NC);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    pdl_wait_prior();

    const int total = a.m_tiles * a.n_tiles;

    if (warp == kDrainWarps) {
        // ------------------------------ TMA producer ------------------------------
        int s = 0;
        uint32_t lap = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < total && ok && !*abort_flag; w += gridDim.x) {
            const int m0 = (w % a.m_tiles) * kM, n0 = (w / a.m_tiles) * NC;
            for (int kb = 0; kb < a.kblocks; ++kb) {
                if (lap > 0)
                    ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty[s], (lap - 1) & 1, a.status, kDevWaitEmpty));
                if (!ok) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&full[s], kStageBytes);
                    tma_load_2d(smem + s * kStageBytes, &tmA, kb * kKB, m0, &full[s]);
                    tma_load_2d(smem + s * kStageBytes + kM * kKB, &tmB, kb * kKB, n0, &full[s]);
                }
                __syncwarp();
                if (++s == kStages) {
                    s = 0;
                    ++lap;
                }
            }
        }
        if (!ok) *abort_flag = 1;
    } else if (warp == kDrainWarps + 1) {
        // ------------------------------ MMA issuer --------------------------------
        // E4M3 is format 0 of this kind, so the descriptor of the fp16 kind serves as it is.
        constexpr uint32_t idesc = idesc_f16(kM, NC);
        int s = 0, ab = 0;
        uint32_t lap = 0, acc_lap = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < total && ok && !*abort_flag; w += gridDim.x) {
            for (int kb = 0; kb < a.kblocks; ++kb) {
                if (acc_lap > 0)
                    ok = __all_sync(0xffffffffu, mbar_wait_bounded(&acc_empty[ab], (acc_lap - 1) & 1, a.status, kDevWaitTmem));
                if (!ok) break;
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[s], lap & 1, a.status, kDevWaitFull));
                if (!ok) break;
                tc_fence_after();
                const uint64_t adesc = smem_desc_sw128(smem_u32(smem + s * kStageBytes));
                const uint64_t bdesc = smem_desc_sw128(smem_u32(smem + s * kStageBytes + kM * kKB));
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < kKB / 32; ++k)   // 32 values = 32 bytes along K inside the swizzle atom
                        tc_mma_f8(tmem_base + ab * NC, adesc + 2 * k, bdesc + 2 * k, idesc, k != 0 ? 1u : 0u);
                    tc_commit(&empty[s]);
                    tc_commit(&acc_full[ab]);
                }
                __syncwarp();
                if (++s == kStages) {
                    s = 0;
                    ++lap;
                }
                ab ^= 1;
                acc_lap += ab == 0;
            }
        }
        if (!ok) *abort_flag = 1;
    } else {
        // ------------------------------ drain (warps 0-7) -------------------------
        constexpr int CW = NC / 2;   // columns of a warp
        const int half = warp >> 2;
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + half * CW;
        int ab = 0;
        uint32_t acc_lap = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < total && ok && !*abort_flag; w += gridDim.x) {
            const int row = (w % a.m_tiles) * kM + (warp & 3) * 32 + lane;
            const int n0 = (w / a.m_tiles) * NC + half * CW;
            const float* sa = a.sA + min(row, a.M - 1);
            const float* sb = a.sB + static_cast<size_t>(min(n0, a.N - 1) >> 7) * a.kblocks;
            float acc[CW];
#pragma unroll
            for (int i = 0; i < CW; ++i) acc[i] = 0.0f;
            float scale = __ldg(sa) * __ldg(sb);
            for (int kb = 0; kb < a.kblocks; ++kb) {
                // the next block's scales are fetched while this one's products are summed
                const int nk = min(kb + 1, a.kblocks - 1);
                const float sa_next = __ldg(sa + static_cast<size_t>(nk) * a.M), sb_next = __ldg(sb + nk);
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(&acc_full[ab], acc_lap & 1, a.status, kDevWaitMma));
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < CW; c += 16) {
                    uint32_t r[16];
                    tmem_ld16(t_lane + ab * NC + c, r);
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[c + i] = fmaf(__uint_as_float(r[i]), scale, acc[c + i]);
                }
                tc_fence_before();
                __syncwarp();
                if (elect_one()) mbar_arrive(&acc_empty[ab]);
                ab ^= 1;
                acc_lap += ab == 0;
                scale = sa_next * sb_next;
            }
            if (!ok) break;
            if (row < a.M && n0 < a.N) {
                const size_t o = static_cast<size_t>(row) * a.N + n0;
                const int ncols = min(CW, a.N - n0);
                const bool vec = ncols == CW && (a.N & 7) == 0 && (reinterpret_cast<uintptr_t>(a.D) & 15) == 0;
                if (a.out_dtype == LSG_DTYPE_F32) {
                    float* dst = static_cast<float*>(a.D) + o;
                    if (vec) {
#pragma unroll
                        for (int q = 0; q < CW / 4; ++q)
                            reinterpret_cast<float4*>(dst)[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
                    } else {
#pragma unroll
                        for (int q = 0; q < CW; ++q)
                            if (q < ncols) dst[q] = acc[q];
                    }
                } else {
                    const bool f16 = a.out_dtype == LSG_DTYPE_F16;
                    uint16_t* dst = static_cast<uint16_t*>(a.D) + o;
#pragma unroll
                    for (int q = 0; q < CW / 8; ++q) {
                        uint32_t pk[4];
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            const float v0 = acc[8 * q + 2 * h], v1 = acc[8 * q + 2 * h + 1];
                            if (f16) {
                                const __half2 v = __floats2half2_rn(v0, v1);
                                pk[h] = *reinterpret_cast<const uint32_t*>(&v);
                            } else {
                                const __nv_bfloat162 v = __floats2bfloat162_rn(v0, v1);
                                pk[h] = *reinterpret_cast<const uint32_t*>(&v);
                            }
                        }
                        if (vec) {
                            reinterpret_cast<uint4*>(dst)[q] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                        } else {
#pragma unroll
                            for (int h = 0; h < 8; ++h)
                                if (8 * q + h < ncols) dst[8 * q + h] = static_cast<uint16_t>(pk[h >> 1] >> (16 * (h & 1)));
                        }
                    }
                }
            }
        }
        if (!ok) *abort_flag = 1;
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kDrainWarps + 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 2 * NC);
    }
}

// e4m3 matrix [rows, K] row-major -> tensor map with a (128 bytes x box_rows) box, 128 B swizzle.
int make_map_e4m3(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(LSG_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K)};
    const cuuint32_t box[2] = {kKB, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(LSG_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d", static_cast<int>(r));
    return LSG_OK;
}

template <int NC>
int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const Fp8Args& a, cudaStream_t s) {
    static std::atomic<bool> configured[64];
    int dev = 0;
    LSG_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_relaxed)) {
        LSG_CUDA_TRY(cudaFuncSetAttribute(fp8_mma_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<NC>::kSmem));
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_relaxed);
    }
    const long long items = static_cast<long long>(a.m_tiles) * a.n_tiles;
    const int grid = items < sm_count() ? static_cast<int>(items) : sm_count();
    LSG_CUDA_TRY(launch_kernel(fp8_mma_kernel<NC>, dim3(grid), dim3(kThreads), Tile<NC>::kSmem, s, true, tmA, tmB, a));
    return LSG_OK;
}

}  // namespace

// TMA wants both operands on 16-byte boundaries and rows that are whole 16-byte pieces.
bool fp8_mma_usable(const void* A, const void* B, int K) {
    return K > 0 && K % 16 == 0 && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) == 0;
}

int fp8_mma(const void* A, const void* B, const float* sA, const float* sB, void* D, int out_dtype, int M, int N, int K,
            cudaStream_t s) {
    Fp8Args a = {};
    a.D = D; a.out_dtype = out_dtype; a.sA = sA; a.sB = sB;
    a.M = M; a.N = N; a.kblocks = (K + kKB - 1) / kKB;
    a.m_tiles = (M + kM - 1) / kM;
    a.status = device_status_word();
    // 256 columns move fewer operand bytes per product; 128 fill more SMs.  A K block of the wide
    // tile takes 1.5 times as long (48 against 32 KB through shared memory).
    const long long wide = static_cast<long long>(a.m_tiles) * ((N + 255) / 256);
    const long long narrow = static_cast<long long>(a.m_tiles) * ((N + 127) / 128);
    const int sms = sm_count();
    const bool take_wide = 3 * ((wide + sms - 1) / sms) <= 2 * ((narrow + sms - 1) / sms);
    const int nc = take_wide ? 256 : 128;
    a.n_tiles = (N + nc - 1) / nc;
    CUtensorMap tmA, tmB;
    int rc = make_map_e4m3(&tmA, A, M, K, kM);
    if (rc != LSG_OK) return rc;
    rc = make_map_e4m3(&tmB, B, N, K, nc);
    if (rc != LSG_OK) return rc;
    return take_wide ? launch<256>(tmA, tmB, a, s) : launch<128>(tmA, tmB, a, s);
}

}  // namespace lsg
