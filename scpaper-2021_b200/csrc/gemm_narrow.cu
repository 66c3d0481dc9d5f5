// Dense fp16 GEMM for few output tiles:  Y = act(X W^T + bias)  or fp32 K-slice sums without bias.
//
// With one to a few row blocks of 128 tokens a GEMM's time is a chain of latencies and the operand
// stream of one SM (about 84 bytes per cycle however few SMs pull), so the output is cut into 128 x 32
// or 128 x 64 tiles - and, where a LayerNorm that adds up slices of K follows, into slices of tiles up
// to 128 wide - until most SMs have one.  One tile per CTA: warp 0 = TMA producer (200 KB of K blocks in flight; weights before the
// wait for the previous kernel), one elected lane of warp 1 issues tcgen05.mma (M = 128, N = BN, K = 16),
// warps 2-9 hold half a tile row each and store it with 16-byte stores, straight from registers or, for
// fp32 rows of 128 bytes and more, through the idle ring so that a warp writes whole lines (a TMA store
// would have to be waited for: 1.1 thousand cycles).  All waits are bounded.
//
// Measured on B200, one 128-token sequence (microseconds, 128 x 128 tiles -> this kernel): 768 -> 3072
// with GELU 5.5 -> 3.9; the 3072 -> 768 product with its residual and LayerNorm 12.9 as one kernel of
// six CTAs -> 7.0 as four K slices on 96 CTAs plus the LayerNorm that adds them.
#include <atomic>

#include "common.cuh"
#include "gemm_common.cuh"
#include "kernels.h"

namespace et {
namespace {

using namespace gemm;

constexpr int PARTIAL = -1;  // ACT value of the fp32 form

template <int BN>
struct NarrowCfg {
    static constexpr int B_BYTES = BN * BK * 2;
    static constexpr int STAGE = A_STAGE_BYTES + B_BYTES;
    static constexpr int STAGES = BN == 32 ? 10 : (BN == 64 ? 8 : 6);
    static constexpr int SMEM = STAGES * STAGE + 256 + 1024;
    static constexpr int TMEM_COLS = BN;
    static_assert(SMEM <= 227 * 1024 && 2 * STAGES * 8 + 16 <= 256, "shared memory budget exceeded");
};

struct NarrowArgs {
    void* Y;  // fp16 [M, ldy], or fp32 [splits][M, N]
    const __half* bias;
    int ldy, M, N, K, splits;
    int* err_word;
};

template <int BN, int ACT>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const NarrowArgs g) {
    using Cfg = NarrowCfg<BN>;
    constexpr int HC = BN / 2;  // columns of an epilogue thread
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* sA = smem;
    uint8_t* sB = smem + Cfg::STAGES * A_STAGE_BYTES;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE);
    uint64_t* empty_bar = full_bar + Cfg::STAGES;
    uint64_t* acc_full = empty_bar + Cfg::STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = uniform_warp_id();
    const int lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * BN;
    const int m0 = blockIdx.y * BM;
    const int split = blockIdx.z;
    const int nkb = (g.K + BK - 1) / BK;
    const int kb0 = nkb * split / g.splits, num_kb = nkb * (split + 1) / g.splits - kb0;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        for (int s = 0; s < Cfg::STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (elect_one()) {
            // weights do not depend on the previous kernel: fetch them before waiting for it
            const int pre = num_kb < Cfg::STAGES ? num_kb : Cfg::STAGES;
            for (int i = 0; i < pre; ++i) {
                mbar_arrive_expect_tx(&full_bar[i], Cfg::STAGE);
                tma_load_2d(sB + i * Cfg::B_BYTES, &tmB, &full_bar[i], (kb0 + i) * BK, n0);
            }
            pdl_wait();
            for (int i = 0; i < pre; ++i)
                tma_load_2d(sA + i * A_STAGE_BYTES, &tmA, &full_bar[i], (kb0 + i) * BK, m0);
            int issued = pre, s = pre == Cfg::STAGES ? 0 : pre;
            uint32_t ph = pre == Cfg::STAGES ? 1u : 0u;
            for (int i = pre; i < num_kb; ++i) {
                if (!mbar_wait_bounded(&empty_bar[s], ph ^ 1, abort_flag)) {
                    report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_PRODUCER);
                    break;
                }
                mbar_arrive_expect_tx(&full_bar[s], Cfg::STAGE);
                tma_load_2d(sA + s * A_STAGE_BYTES, &tmA, &full_bar[s], (kb0 + i) * BK, m0);
                tma_load_2d(sB + s * Cfg::B_BYTES, &tmB, &full_bar[s], (kb0 + i) * BK, n0);
                ++issued;
                if (++s == Cfg::STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            if (*abort_flag)  // let copies in flight land before the CTA's shared memory is released
                for (int i = issued > Cfg::STAGES ? issued - Cfg::STAGES : 0; i < issued; ++i)
                    for (uint32_t sp = 0; sp < ET_SPIN_LIMIT; ++sp)
                        if (mbar_try_wait(&full_bar[i % Cfg::STAGES], (i / Cfg::STAGES) & 1)) break;
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (warp-uniform, one elected lane issues) ----------------
        const bool leader = elect_one();
        constexpr uint32_t idesc = make_idesc_f16(BM, BN, 0, 0);
        const uint32_t a_base = desc_lo(smem_u32(sA)), b_base = desc_lo(smem_u32(sB));
        bool ok = true;
        int s = 0;
        uint32_t ph = 0;
        for (int i = 0; i < num_kb; ++i) {
            if (!mbar_wait_bounded_warp(&full_bar[s], ph, abort_flag)) {
                ok = false;
                break;
            }
            tc_fence_after_sync();
            const uint32_t a_lo = a_base + s * (A_STAGE_BYTES >> 4);
            const uint32_t b_lo = b_base + s * (Cfg::B_BYTES >> 4);
            if (leader) {
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    mma_f16_ss_k128(tmem_base, a_lo + k * 2, b_lo + k * 2, idesc, (i | k) != 0 ? 1u : 0u);
                mma_commit(&empty_bar[s]);
            }
            __syncwarp();
            if (++s == Cfg::STAGES) {
                s = 0;
                ph ^= 1u;
            }
        }
        if (leader) {
            if (ok) mma_commit(acc_full);
            else report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_MMA);
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: half a tile row per thread ----------------
        const int q = warp & 3;            // tensor-memory lane quadrant
        const int half = (warp - 2) >> 2;  // which HC columns of the row
        const int n = n0 + half * HC;
        const int row = m0 + q * 32 + lane;
        float b[ACT == PARTIAL ? 8 : HC];
#pragma unroll
        for (int j = 0; j < (ACT == PARTIAL ? 0 : HC); j += 8) {
            uint4 bq = make_uint4(0u, 0u, 0u, 0u);
            if (g.bias != nullptr && n + j < g.N)  // (N % 8 == 0)
                bq = __ldg(reinterpret_cast<const uint4*>(g.bias + n + j));
            const __half2* h = reinterpret_cast<const __half2*>(&bq);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = __half22float2(h[i]);
                b[j + 2 * i] = f.x;
                b[j + 2 * i + 1] = f.y;
            }
        }
        pdl_wait();  // the output may still be read by an earlier kernel
        bool ok = mbar_wait_bounded(acc_full, 0, abort_flag);
        if (!ok) report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_EPILOGUE);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            tc_fence_after_sync();
            const uint32_t addr = tmem_base + half * HC + (static_cast<uint32_t>(q * 32) << 16);
            constexpr int CH = HC < 32 ? HC : 32;  // columns per step
#pragma unroll
            for (int c = 0; c < HC; c += CH) {
                uint32_t r[CH];
                if (num_kb > 0) {
                    if (CH == 16) tmem_ld16(addr + c, *reinterpret_cast<uint32_t(*)[16]>(&r[0]));
                    else tmem_ld32(addr + c, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int j = 0; j < CH; ++j) r[j] = 0u;
                }
                if (ACT == PARTIAL) {
                    float* p = static_cast<float*>(g.Y) + static_cast<size_t>(split) * g.M * g.N;
                    if (CH == 32) {
                        uint8_t* tile = smem + (warp - 2) * 4096;  // 32 rows of 128 bytes, swizzled
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            *reinterpret_cast<uint4*>(tile + lane * 128 + ((j ^ (lane & 7)) * 16)) =
                                make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                        __syncwarp();
                        const int piece = lane & 7, nn = n + c + piece * 4;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int rr = i * 4 + (lane >> 3), m = m0 + q * 32 + rr;
                            if (m < g.M && nn < g.N)
                                *reinterpret_cast<uint4*>(p + static_cast<size_t>(m) * g.N + nn) =
                                    *reinterpret_cast<const uint4*>(tile + rr * 128 +
                                                                    ((piece ^ (rr & 7)) * 16));
                        }
                        __syncwarp();
                    } else if (row < g.M) {
#pragma unroll
                        for (int j = 0; j < CH; j += 4)
                            if (n + c + j < g.N)
                                *reinterpret_cast<uint4*>(p + static_cast<size_t>(row) * g.N + n + c + j) =
                                    make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
                    }
                } else if (row < g.M) {
                    __half* p = static_cast<__half*>(g.Y) + static_cast<size_t>(row) * g.ldy + n + c;
#pragma unroll
                    for (int j = 0; j < CH; j += 8) {
                        float v[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            v[i] = act_fn<ACT == PARTIAL ? ET_ACT_NONE : ACT>(__uint_as_float(r[j + i]) + b[ACT == PARTIAL ? 0 : c + j + i]);
                        if (n + c + j < g.N)
                            *reinterpret_cast<uint4*>(p + j) =
                                make_uint4(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]),
                                           pack_half2(v[4], v[5]), pack_half2(v[6], v[7]));
                    }
                }
            }
        }
    }

    pdl_wait();  // no CTA may retire before the kernels it depends on have completed
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
}

template <int BN, int ACT>
int launch_cfg(const CUtensorMap& tmA, const CUtensorMap& tmB, const NarrowArgs& a, cudaStream_t stream) {
    auto kern = gemm_narrow_kernel<BN, ACT>;
    static std::atomic<bool> attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, NarrowCfg<BN>::SMEM) !=
            cudaSuccess)
            return ET_ERR_CUDA;
        attr_set[dev] = true;
    }
    const dim3 grid((a.N + BN - 1) / BN, (a.M + BM - 1) / BM, a.splits);
    return launch_kernel(kern, grid, dim3(GEMM_THREADS), NarrowCfg<BN>::SMEM, stream, tmA, tmB, a) ==
                   cudaSuccess
               ? ET_OK
               : ET_ERR_CUDA;
}

template <int BN>
int launch_bn(int act, bool partial, const CUtensorMap& tmA, const CUtensorMap& tmB, const NarrowArgs& a,
              cudaStream_t stream) {
    if (partial) return launch_cfg<BN, PARTIAL>(tmA, tmB, a, stream);
    if (act == ET_ACT_GELU) return launch_cfg<BN, ET_ACT_GELU>(tmA, tmB, a, stream);
    if (act == ET_ACT_RELU) return launch_cfg<BN, ET_ACT_RELU>(tmA, tmB, a, stream);
    return launch_cfg<BN, ET_ACT_NONE>(tmA, tmB, a, stream);
}

}  // namespace

int launch_gemm_narrow(const __half* X, int ldx, const __half* W, int ldw, const __half* bias, void* Y,
                       int ldy, int M, int N, int K, int act, int bn, int splits, bool partial,
                       cudaStream_t stream) {
    CUtensorMap tmA, tmB;
    int st;
    if ((st = encode_operand(&tmA, X, ldx, M, K, BM)) != ET_OK) return st;
    if ((st = encode_operand(&tmB, W, ldw, N, K, bn)) != ET_OK) return st;
    NarrowArgs a;
    a.Y = Y;
    a.bias = bias;
    a.ldy = ldy;
    a.M = M;
    a.N = N;
    a.K = K;
    a.splits = splits;
    a.err_word = device_error_word();
    if (!a.err_word) return ET_ERR_NO_DEVICE;
    if (bn == 32) return launch_bn<32>(act, partial, tmA, tmB, a, stream);
    if (bn == 64) return launch_bn<64>(act, partial, tmA, tmB, a, stream);
    if (bn == 128 && partial) return launch_cfg<128, PARTIAL>(tmA, tmB, a, stream);
    return ET_ERR_INVALID_ARG;
}

}  // namespace et
