// Dense Linear + residual + LayerNorm in one kernel for many rows:
//   out = LayerNorm(X W^T + bias + residual) * gamma + beta          (eps 1e-5)
// (reference Encoder/Encoder.h: the O projection and FFN2, each followed by SkipLayerNorm).
//
// A cluster of N / 128 CTAs owns 256 rows over their whole width: N / 256 CTA pairs side by side, each
// pair a 256 x 256 tile with tcgen05.mma.cta_group::2 exactly as gemm_pair.cu computes it (every CTA
// fetches only its own 128 rows of X and 128 rows of W).  The clusters are persistent over the row
// blocks with two accumulators, so the epilogue of one block runs under the products of the next:
//   * a thread owns one row x 128 columns; the accumulator goes into registers at once and its tensor
//     memory is handed back,
//   * the residual arrives by TMA in the warp's staging tile while the products run, and the result
//     leaves through the same tile,
//   * the row's partial sums go to the other column tiles' CTAs with st.async, whose completion is
//     counted on the receiver's mbarrier: no cluster-wide barrier inside the loop.
// The product is never rounded to fp16 nor written: per row the separate LayerNorm pass (6 bytes an
// element, bound by HBM) and the product's own store go away.
//
// What bounds it: operand bandwidth of the pair tiles (64 B/clk/SM) and the SMs that whole clusters
// cannot cover.  All waits are bounded.
#include <atomic>

#include "common.cuh"
#include "gemm_common.cuh"
#include "kernels.h"

namespace et {
namespace {

using namespace gemm;

constexpr int PL_BN = 256;
constexpr int PL_STAGES = 4;
constexpr int PL_B_HALF = (PL_BN / 2) * BK * 2;
constexpr int PL_STAGE_BYTES = A_STAGE_BYTES + PL_B_HALF;  // per CTA
constexpr int PL_RING = PL_STAGES * PL_STAGE_BYTES;        // 128 KB
constexpr int PL_WARP_TILE = 32 * 128 * 2;                 // 32 rows x 128 fp16 columns
constexpr int PL_STAGING = EPI_WARPS * PL_WARP_TILE;       // 64 KB
constexpr int PL_MAX_COLS = 4;                             // column tiles (pairs) per cluster
constexpr int PL_STATS = 2 * PL_MAX_COLS * 2 * BM * 8;     // [parity][column tile][half][row]
constexpr int PL_MISC = 256 + 3 * PL_BN * 4 + PL_STATS;
constexpr int PL_SMEM = PL_RING + PL_STAGING + PL_MISC + 1024;
static_assert(PL_SMEM <= 227 * 1024, "shared memory budget exceeded");

struct PairLnArgs {
    const __half* bias;   // [N] or null
    const __half* gamma;  // [N]
    const __half* beta;   // [N]
    int M, N, K;
    float eps;
    int* err_word;
};

__device__ __forceinline__ void st_async_f32x2(uint32_t cluster_addr, float a, float b, uint32_t cluster_bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(
                     cluster_addr),
                 "f"(a), "f"(b), "r"(cluster_bar)
                 : "memory");
}

// Bounded wait on a barrier of this CTA that st.async of other CTAs complete: acquires at cluster scope.
__device__ __forceinline__ bool mbar_wait_bounded_cluster(uint64_t* bar, uint32_t parity,
                                                          volatile int* abort_flag) {
    for (uint32_t it = 0; it < ET_SPIN_LIMIT; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t"
            ".reg .pred P;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, P;\n\t"
            "}\n"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 255u) == 255u && *abort_flag) return false;
    }
    return false;
}

__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_pair_ln_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmR, const __grid_constant__ CUtensorMap tmY,
                    const PairLnArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* sA = smem;
    uint8_t* sB = smem + PL_STAGES * A_STAGE_BYTES;
    uint8_t* sStage = smem + PL_RING;
    uint8_t* misc = sStage + PL_STAGING;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(misc);  // used in the pair's leader
    uint64_t* empty_bar = full_bar + PL_STAGES;
    uint64_t* acc_full = empty_bar + PL_STAGES;  // [2]
    uint64_t* acc_empty = acc_full + 2;          // [2], in the leader: both CTAs' epilogue warps
    uint64_t* stat_full = acc_empty + 2;         // [2]
    uint64_t* res_full = stat_full + 2;          // [EPI_WARPS]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(res_full + EPI_WARPS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* s_bias = reinterpret_cast<float*>(misc + 256);
    float* s_gamma = s_bias + PL_BN;
    float* s_beta = s_gamma + PL_BN;
    float2* s_stats = reinterpret_cast<float2*>(s_beta + PL_BN);  // [2][PL_MAX_COLS][2][BM]

    const int warp = uniform_warp_id();
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const uint32_t row_half = rank & 1, leader_rank = rank & ~1u;
    const int ct = static_cast<int>(rank >> 1);  // this pair's column tile
    const int ncol = g.N / PL_BN;
    const int n0 = ct * PL_BN;
    const int cluster = blockIdx.x / (2 * ncol), nclusters = gridDim.x / (2 * ncol);
    const int tiles = (g.M + 2 * BM - 1) / (2 * BM);
    const int num_kb = (g.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        tma_prefetch_desc(&tmR);
        for (int s = 0; s < PL_STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 2 * EPI_WARPS);
            mbar_init(&stat_full[i], 1);
        }
        for (int i = 0; i < EPI_WARPS; ++i) mbar_init(&res_full[i], 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 2 * PL_BN);
        tmem_relinquish_pair();
    }
    for (int i = threadIdx.x; i < PL_BN; i += GEMM_THREADS) {
        s_bias[i] = g.bias != nullptr ? __half2float(__ldg(g.bias + n0 + i)) : 0.f;
        s_gamma[i] = __half2float(__ldg(g.gamma + n0 + i));
        s_beta[i] = __half2float(__ldg(g.beta + n0 + i));
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();  // every CTA's barriers exist before anything arrives on them
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();

    if (warp == 0) {
        // ---------------- TMA producer (every CTA: its own rows of X and W) ----------------
        if (elect_one()) {
            int s = 0, issued = 0;
            uint32_t ph = 0;
            bool ok = true, first = true;
            const int nb0 = n0 + static_cast<int>(row_half) * (PL_BN / 2);
            for (int t = cluster; ok && t < tiles; t += nclusters) {
                const int m0 = t * 2 * BM + static_cast<int>(row_half) * BM;
                int i0 = 0;
                if (first) {
                    // weights do not depend on the previous kernel: fetch them before waiting for it
                    first = false;
                    const int pre = num_kb < PL_STAGES ? num_kb : PL_STAGES;
                    for (int i = 0; i < pre; ++i) {
                        if (row_half == 0) mbar_arrive_expect_tx(&full_bar[i], 2 * PL_STAGE_BYTES);
                        tma_load_2d_pair(sB + i * PL_B_HALF, &tmB,
                                         map_to_cta(smem_u32(&full_bar[i]), leader_rank), i * BK, nb0);
                    }
                    pdl_wait();
                    for (int i = 0; i < pre; ++i)
                        tma_load_2d_pair(sA + i * A_STAGE_BYTES, &tmA,
                                         map_to_cta(smem_u32(&full_bar[i]), leader_rank), i * BK, m0);
                    issued = pre;
                    s = pre % PL_STAGES;
                    ph = (pre / PL_STAGES) & 1;
                    i0 = pre;
                }
                for (int i = i0; i < num_kb; ++i) {
                    if (!mbar_wait_bounded(&empty_bar[s], ph ^ 1, abort_flag)) {
                        report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_PRODUCER);
                        ok = false;
                        break;
                    }
                    if (row_half == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * PL_STAGE_BYTES);
                    const uint32_t lb = map_to_cta(smem_u32(&full_bar[s]), leader_rank);
                    tma_load_2d_pair(sA + s * A_STAGE_BYTES, &tmA, lb, i * BK, m0);
                    tma_load_2d_pair(sB + s * PL_B_HALF, &tmB, lb, i * BK, nb0);
                    ++issued;
                    if (++s == PL_STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (*abort_flag && row_half == 0) {
                // Let copies in flight land before shared memory is released: both CTAs' loads signal
                // the leader's barriers, and no CTA leaves before the final cluster barrier.
                for (int i = issued > PL_STAGES ? issued - PL_STAGES : 0; i < issued; ++i)
                    for (uint32_t sp = 0; sp < ET_SPIN_LIMIT; ++sp)
                        if (mbar_try_wait(&full_bar[i % PL_STAGES], (i / PL_STAGES) & 1)) break;
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the pair's leader; warp-uniform, one elected lane) --------
        if (row_half == 0) {
            const bool leader = elect_one();
            constexpr uint32_t idesc = make_idesc_f16(2 * BM, PL_BN, 0, 0);
            const uint32_t a_base = desc_lo(smem_u32(sA)), b_base = desc_lo(smem_u32(sB));
            const uint32_t eb0 = map_to_cta(smem_u32(empty_bar), leader_rank);
            const uint32_t eb1 = map_to_cta(smem_u32(empty_bar), leader_rank + 1);
            const uint32_t af0 = map_to_cta(smem_u32(acc_full), leader_rank);
            const uint32_t af1 = map_to_cta(smem_u32(acc_full), leader_rank + 1);
            int s = 0, it = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = cluster; ok && t < tiles; t += nclusters, ++it) {
                const int buf = it & 1;
                // both CTAs' epilogues must have drained this accumulator's previous tile
                if (!mbar_wait_bounded_warp(&acc_empty[buf], ((it >> 1) & 1) ^ 1, abort_flag)) {
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + buf * PL_BN;
                for (int i = 0; i < num_kb; ++i) {
                    if (!mbar_wait_bounded_warp(&full_bar[s], ph, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t a_lo = a_base + s * (A_STAGE_BYTES >> 4);
                    const uint32_t b_lo = b_base + s * (PL_B_HALF >> 4);
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)
                            mma_f16_ss_pair_k128(d_tmem, a_lo + k * 2, b_lo + k * 2, idesc,
                                                 (i | k) != 0 ? 1u : 0u);
                        // the stage is free in both CTAs once these products have read it
                        mma_commit_pair(eb0 + s * 8);
                        mma_commit_pair(eb1 + s * 8);
                    }
                    __syncwarp();
                    if (++s == PL_STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                if (ok && leader) {
                    mma_commit_pair(af0 + buf * 8);
                    mma_commit_pair(af1 + buf * 8);
                }
                __syncwarp();
            }
            if (!ok && leader) report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_MMA);
            __syncwarp();
        }
    } else {
        // ---------------- epilogue of this CTA's 128 rows x 256 columns ----------------
        const int w = warp - 2;
        const int q = warp & 3;   // tensor-memory lane quadrant
        const int half = w >> 2;  // which 128 columns of the tile
        const int r = q * 32 + lane;
        uint8_t* tile = sStage + w * PL_WARP_TILE;  // two 32 x 64 boxes, 128-byte swizzled
        uint8_t* srow = tile + lane * 128;
        const int nc0 = n0 + half * 128;
        const float* b128 = s_bias + half * 128;
        const float* g128 = s_gamma + half * 128;
        const float* e128 = s_beta + half * 128;
        const uint32_t my_empty = smem_u32(&acc_empty[0]);
        const uint32_t leader_acc_empty = map_to_cta(my_empty, leader_rank);
        const float inv_n = 1.0f / static_cast<float>(g.N);
        bool ok = true;

        auto load_residual = [&](int t) {  // one lane
            mbar_arrive_expect_tx(&res_full[w], PL_WARP_TILE);
            const int row = t * 2 * BM + static_cast<int>(row_half) * BM + q * 32;
            tma_load_2d(tile, &tmR, &res_full[w], nc0, row);
            tma_load_2d(tile + 4096, &tmR, &res_full[w], nc0 + 64, row);
        };
        pdl_wait();  // the residual and the output buffer belong to earlier kernels
        if (lane == 0 && cluster < tiles) load_residual(cluster);

        int it = 0;
        for (int t = cluster; t < tiles; t += nclusters, ++it) {
            const int buf = it & 1;
            const uint32_t use_ph = (it >> 1) & 1;
            const int m0 = t * 2 * BM + static_cast<int>(row_half) * BM;
            if (threadIdx.x == 64) mbar_arrive_expect_tx(&stat_full[buf], ncol * 2 * BM * 8);
            // the residual first: its copy has landed when this warp leaves, whatever fails later
            ok = mbar_wait_bounded(&res_full[w], it & 1, abort_flag);
            ok = mbar_wait_bounded(&acc_full[buf], use_ph, abort_flag) && ok;
            if (!ok) report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_EPILOGUE);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();

            uint32_t v[4][32];
            const uint32_t addr =
                tmem_base + buf * PL_BN + half * 128 + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(addr + c * 32, v[c]);
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld_wait_regs(v[c]);
            // this warp no longer needs the accumulator: tell the leader's MMA warp
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                if (row_half == 0)
                    mbar_arrive(&acc_empty[buf]);
                else
                    mbar_arrive_cluster(leader_acc_empty + buf * 8);
            }

            float sum = 0.f, sq = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 res = *reinterpret_cast<const uint4*>(
                        srow + (c >> 1) * 4096 + ((((c & 1) * 4 + i) ^ (lane & 7)) * 16));
                    const __half2* hp = reinterpret_cast<const __half2*>(&res);
                    const float4 b0 = *reinterpret_cast<const float4*>(b128 + c * 32 + i * 8);
                    const float4 b1 = *reinterpret_cast<const float4*>(b128 + c * 32 + i * 8 + 4);
                    const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f = __half22float2(hp[j]);
                        const float x0 = __uint_as_float(v[c][i * 8 + 2 * j]) + bb[2 * j] + f.x;
                        const float x1 = __uint_as_float(v[c][i * 8 + 2 * j + 1]) + bb[2 * j + 1] + f.y;
                        v[c][i * 8 + 2 * j] = __float_as_uint(x0);
                        v[c][i * 8 + 2 * j + 1] = __float_as_uint(x1);
                        sum += x0 + x1;
                        sq = fmaf(x0, x0, fmaf(x1, x1, sq));
                    }
                }
            // to the CTAs that hold the same rows, this one included
            {
                const uint32_t slot =
                    smem_u32(&s_stats[((buf * PL_MAX_COLS + ct) * 2 + half) * BM + r]);
                const uint32_t bar = smem_u32(&stat_full[buf]);
                for (int p = 0; p < ncol; ++p) {
                    const uint32_t to = 2 * p + row_half;
                    st_async_f32x2(map_to_cta(slot, to), sum, sq, map_to_cta(bar, to));
                }
            }
            ok = mbar_wait_bounded_cluster(&stat_full[buf], use_ph, abort_flag);
            if (!ok) report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_EPILOGUE);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            float tsum = 0.f, tsq = 0.f;
            for (int p = 0; p < 2 * ncol; ++p) {
                const float2 s2 = s_stats[(buf * PL_MAX_COLS * 2 + p) * BM + r];
                tsum += s2.x;
                tsq += s2.y;
            }
            const float mean = tsum * inv_n;
            const float var = fmaxf(tsq * inv_n - mean * mean, 0.f);
            const float rstd = rsqrtf(var + g.eps);
            const float shift = -mean * rstd;
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = c * 32 + i * 8;
                    float y[8];
#pragma unroll
                    for (int j = 0; j < 8; j += 4) {
                        const float4 gm = *reinterpret_cast<const float4*>(g128 + n + j);
                        const float4 bt = *reinterpret_cast<const float4*>(e128 + n + j);
                        y[j] = fmaf(fmaf(__uint_as_float(v[c][i * 8 + j]), rstd, shift), gm.x, bt.x);
                        y[j + 1] = fmaf(fmaf(__uint_as_float(v[c][i * 8 + j + 1]), rstd, shift), gm.y, bt.y);
                        y[j + 2] = fmaf(fmaf(__uint_as_float(v[c][i * 8 + j + 2]), rstd, shift), gm.z, bt.z);
                        y[j + 3] = fmaf(fmaf(__uint_as_float(v[c][i * 8 + j + 3]), rstd, shift), gm.w, bt.w);
                    }
                    uint4 o;
                    o.x = pack_half2(y[0], y[1]);
                    o.y = pack_half2(y[2], y[3]);
                    o.z = pack_half2(y[4], y[5]);
                    o.w = pack_half2(y[6], y[7]);
                    *reinterpret_cast<uint4*>(srow + (c >> 1) * 4096 +
                                              ((((c & 1) * 4 + i) ^ (lane & 7)) * 16)) = o;
                }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                if (m0 + q * 32 < g.M) {
                    tma_store_2d(&tmY, tile, nc0, m0 + q * 32);
                    tma_store_2d(&tmY, tile + 4096, nc0 + 64, m0 + q * 32);
                }
                tma_store_commit();
                tma_store_wait_read();
                if (t + nclusters < tiles) load_residual(t + nclusters);
            }
            __syncwarp();
        }
    }

    pdl_wait();  // no CTA may retire before the kernels it depends on have completed
    tc_fence_before_sync();
    __syncthreads();
    // no CTA may leave while another can still read its operands or write its statistics
    cluster_sync_all();
    if (warp == 1) tmem_dealloc_pair(tmem_base, 2 * PL_BN);
}

cudaError_t set_smem_attr() {
    return cudaFuncSetAttribute(gemm_pair_ln_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PL_SMEM);
}

// Clusters of `csize` CTAs the device holds at once (whole clusters inside a GPC); asked once per
// device and size, 0 if the question fails.
int resident_clusters(int csize) {
    static std::atomic<int> known[64][2 * PL_MAX_COLS + 1] = {};  // 0 = not asked, else answer + 1
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || csize < 2 || csize > 2 * PL_MAX_COLS) return 0;
    if (known[dev][csize] == 0) {
        int n = 0;
        if (set_smem_attr() == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(static_cast<unsigned>(csize));
            cfg.blockDim = dim3(GEMM_THREADS);
            cfg.dynamicSmemBytes = PL_SMEM;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = static_cast<unsigned>(csize);
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, gemm_pair_ln_kernel, &cfg) != cudaSuccess) n = 0;
        }
        cudaGetLastError();
        known[dev][csize] = (n < 0 ? 0 : n) + 1;
    }
    return known[dev][csize] - 1;
}

int g_pair_ln = -1;  // test hook: -1 = automatic, 0 = never, 1 = wherever it applies

}  // namespace

bool gemm_pair_ln_applies(int M, int N, int K) {
    if (g_pair_ln == 0 || M <= 0 || K <= 0) return false;
    if (N < 2 * PL_BN || N % PL_BN || N / PL_BN > PL_MAX_COLS) return false;
    return resident_clusters(N / 128) > 0;
}

// Whether this kernel is expected to beat the plain GEMM followed by the LayerNorm pass.  Times in
// hundredths of a microsecond, fitted to B200 runs at N = 512 / 768 / 1024, K = N .. 4 N and 1024 to 131072
// rows: a 256 x 256 pair tile costs 41 a K block in either form; here whole clusters must cover the rows
// (22 resident clusters of 6 CTAs at N = 768, 15 of 8 at N = 1024) and a tile's epilogue shows 180; there the
// pass reads and writes 6 bytes an element at 5.5 TB/s behind a launch.  Measured, here against there: 172.6
// against 235.9 us (131072 x 768 -> 768), 513 against 551 us (3072 -> 768), 274 against 386 us (1024 -> 1024), 19.3
// against 19.7 us (8192 x 768 -> 768), but 66 against 57 us where three rounds of clusters replace two of pairs
// (12288 x 3072 -> 768).  Below 8192 rows the plain GEMM has better-fitting tiles (31 against 41 us at
// 6144 x 3072 -> 768).
bool gemm_pair_ln_pays(int M, int N, int K) {
    if (!gemm_pair_ln_applies(M, N, K)) return false;
    if (g_pair_ln > 0) return true;
    if (M < 8192) return false;
    const long sms = sm_count() > 0 ? sm_count() : 148;
    const long mt = (M + 2 * BM - 1) / (2 * BM), nkb = (K + BK - 1) / BK;
    const long res = resident_clusters(N / 128);
    const long here = 450 + (mt + res - 1) / res * (nkb * 41 + 180);
    const long pairs = mt * ((N + 255) / 256);
    const long there = (pairs + sms / 2 - 1) / (sms / 2) * (nkb * 41 + 100) + 850 +
                       static_cast<long>(M) * N * 6 / 55000;
    return here < there;
}

// Arguments as launch_gemm_ln's, already checked; resid not null.
int launch_gemm_pair_ln(const __half* X, int ldx, const __half* W, int ldw, const __half* bias,
                        const __half* resid, int ldr, const __half* gamma, const __half* beta, __half* out,
                        int ldo, int M, int N, int K, cudaStream_t stream) {
    CUtensorMap tmA, tmB, tmR, tmY;
    int st;
    if ((st = encode_operand(&tmA, X, ldx, M, K, BM)) != ET_OK) return st;
    if ((st = encode_operand(&tmB, W, ldw, N, K, PL_BN / 2)) != ET_OK) return st;
    auto rows32 = [&](CUtensorMap* tm, const __half* p, int ld) {
        const uint64_t dims[2] = {static_cast<uint64_t>(N), static_cast<uint64_t>(M)};
        const uint64_t strides[1] = {static_cast<uint64_t>(ld) * 2};
        const uint32_t box[2] = {64, 32};
        return make_tensor_map_f16(tm, p, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    };
    if ((st = rows32(&tmR, resid, ldr)) != ET_OK) return st;
    if ((st = rows32(&tmY, out, ldo)) != ET_OK) return st;
    static std::atomic<bool> attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (set_smem_attr() != cudaSuccess) return ET_ERR_CUDA;
        attr_set[dev] = true;
    }
    PairLnArgs a;
    a.bias = bias;
    a.gamma = gamma;
    a.beta = beta;
    a.M = M;
    a.N = N;
    a.K = K;
    a.eps = 1e-5f;
    a.err_word = device_error_word();
    const int csize = N / 128;
    const int tiles = (M + 2 * BM - 1) / (2 * BM);
    const int resident = resident_clusters(csize);
    const int clusters = resident > 0 && resident < tiles ? resident : tiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(clusters * csize));
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = PL_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(csize);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, gemm_pair_ln_kernel, tmA, tmB, tmR, tmY, a) == cudaSuccess ? ET_OK
                                                                                             : ET_ERR_CUDA;
}

}  // namespace et

#ifdef ET_TEST_HOOKS
extern "C" {
// Test hook: dense Linear + LayerNorm on persistent clusters of CTA pairs: -1 = automatic, 0 = never,
// 1 = wherever it applies.  Returns the resident clusters for an N-wide output.
int et_debug_set_pair_ln(int mode, int N) {
    et::g_pair_ln = mode;
    return et::resident_clusters(N / 128);
}
}
#endif  // ET_TEST_HOOKS
