// Attention with the value and output projections pre-multiplied (W_VO = W_V W_O per head):
//   out[t, :] = bias_o + sum_h softmax(scale * Q_h K_h^T + mask)[t, :] . VO_h
// where VO[b][h] = X_b W_VO[h] has the full model width.
//
// A work item is 128 queries of one sequence and a chunk of up to 256 output features.  Its heads
// are dealt to the CTAs of a thread-block cluster (contiguous ranges; one CTA when the items alone
// fill the machine).  A CTA accumulates its heads' O += P_h . VO_h in tensor memory, in the order
// of the heads; at the end the cluster's partial sums meet in distributed shared memory, every CTA
// adding the ranks' contributions to its share of the rows in rank order, so the result is
// deterministic and the output needs no pre-zeroing (the reference reduces heads with half2
// atomics).  Because every head has its own softmax normaliser, probabilities are normalised
// BEFORE the second product: for sequences longer than one key block a first pass over the head's
// key blocks computes the row max and sum (scores only), a second pass recomputes the scores,
// writes P = exp2(s - m) / l as the fp16 A operand and accumulates O += P . VO_h[block].
//
// What bounds it: per head and key block the tensor core needs 1280 cycles (256 for the scores,
// 1024 for 128 x 256 x 128) and the special-function unit 1024 (128 x 128 exponentials), so the
// kernel is a pipeline of the two: two score buffers in tensor memory (S of the next task is
// computed while this task's softmax runs), probabilities held in registers until the previous
// P . VO has left the P tile, Q / K of the next task and VO in half blocks of 64 keys prefetched
// by two producer warps.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace et {
namespace {

constexpr int BQ = 128;
constexpr int BKV = 128;
constexpr int VO_KEYS = 64;                        // keys of one VO stage
constexpr int VO_STAGES = 3;
constexpr int VO_SM_WARPS = 8;                     // softmax / output warps
constexpr int VO_SM_THREADS = 32 * VO_SM_WARPS;
constexpr int VO_THREADS = 96 + VO_SM_THREADS;     // + Q/K producer, MMA issuer, VO producer
constexpr int VO_MAX_CLUSTER = 8;
constexpr int ATOM_BYTES = 128 * 128;
constexpr int VO_ATOM = VO_KEYS * 128;             // 64 keys x 64 features
constexpr int VO_QK_BYTES = 4 * ATOM_BYTES;        // two stages of 64-wide heads or one of 128-wide
// NC output features per CTA: 256, or 128 / 64 behind a test hook.  Tensor memory: two score
// buffers in columns [0, 256), the accumulator behind them.
constexpr int VO_TMEM_COLS = 512;
__host__ __device__ constexpr int vo_stage_bytes(int nc) { return (nc / 64) * VO_ATOM; }
// fp32 rows of the final exchange, padded so that a warp's 16-byte stores (one row per lane) hit
// all banks
__host__ __device__ constexpr int vo_pitch(int nc) { return nc * 4 + 16; }
__host__ __device__ constexpr int vo_exchange_bytes(int nc, int csize) {
    return csize * ((BQ + csize - 1) / csize) * vo_pitch(nc);
}
__host__ __device__ constexpr int vo_smem_bytes(int nc) {
    // the exchange overlays the operand stages once the last product is complete
    const int operands = VO_QK_BYTES + VO_STAGES * vo_stage_bytes(nc);
    int exchange = 0;
    for (int g = 1; g <= VO_MAX_CLUSTER; ++g)
        exchange = vo_exchange_bytes(nc, g) > exchange ? vo_exchange_bytes(nc, g) : exchange;
    return (operands > exchange ? (operands + 1023) / 1024 * 1024 : (exchange + 1023) / 1024 * 1024) +
           2 * ATOM_BYTES + 256 + 4 * BQ * 4 + 1024;
}
static_assert(vo_smem_bytes(256) <= 227 * 1024, "shared memory budget exceeded");

struct VoArgs {
    __half* out;
    const __half* bias_o;
    const __half* mask;
    const int* valid_len;
    int batch, seq, nhead, dh_qk, emdim;
    float scale_log2;
    int* err_word;
};

__device__ __forceinline__ uint32_t vo_cluster_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t x, uint32_t y, uint32_t z,
                                              uint32_t w) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y),
                 "r"(z), "r"(w)
                 : "memory");
}

template <int NC, int MASK>
__global__ void __launch_bounds__(VO_THREADS, 1)
attention_vo_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmVO, const VoArgs a) {
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment computed on the shared-window offset, so that the pointer keeps its
    // shared-memory provenance (plain LDS / STS instead of generic accesses)
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int nqa = (a.dh_qk + 63) >> 6;
    const int qk_stages = nqa == 1 ? 2 : 1;
    const int qk_stage_bytes = 2 * nqa * ATOM_BYTES;
    uint8_t* sQK = smem;
    uint8_t* sVO = sQK + VO_QK_BYTES;
    uint8_t* sP = smem + vo_smem_bytes(NC) - 1024 - (2 * ATOM_BYTES + 256 + 4 * BQ * 4);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sP + 2 * ATOM_BYTES);
    uint64_t* qk_full = bars;        // [2]
    uint64_t* qk_empty = bars + 2;   // [2]
    uint64_t* vo_full = bars + 4;    // [VO_STAGES]
    uint64_t* vo_empty = bars + 7;   // [VO_STAGES]
    uint64_t* s_full = bars + 10;    // [2]
    uint64_t* s_free = bars + 12;    // [2]
    uint64_t* p_full = bars + 14;
    uint64_t* pv_done = bars + 15;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* s_x = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 256);  // [2][2][128]

    const int warp = uniform_warp_id();
    const int lane = threadIdx.x & 31;
    const int csize = static_cast<int>(vo_cluster_size());
    const int rank = static_cast<int>(cluster_ctarank());
    const int q0 = static_cast<int>(blockIdx.x / csize) * BQ;
    const int e0 = blockIdx.y * NC;
    const int b = blockIdx.z;
    const int n_c = (a.emdim - e0) < NC ? (a.emdim - e0) : NC;  // multiple of 16
    const int nca = (n_c + 63) >> 6;
    const int h_begin = a.nhead * rank / csize, h_end = a.nhead * (rank + 1) / csize;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmVO);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&qk_full[i], 1);
            mbar_init(&qk_empty[i], 1);
            mbar_init(&s_full[i], 1);
            mbar_init(&s_free[i], VO_SM_THREADS);
        }
        for (int i = 0; i < VO_STAGES; ++i) {
            mbar_init(&vo_full[i], 1);
            mbar_init(&vo_empty[i], 1);
        }
        mbar_init(p_full, VO_SM_THREADS);
        mbar_init(pv_done, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, VO_TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_O = tmem_base + 256;
    pdl_launch_dependents();
    pdl_wait();  // every input is produced by earlier kernels on the stream

    int kv_len = a.seq;
    if (MASK == ET_MASK_PADDING) {
        kv_len = __ldcg(a.valid_len + b);
        kv_len = kv_len < 0 ? 0 : (kv_len > a.seq ? a.seq : kv_len);
    }
    int n_kv = (kv_len + BKV - 1) / BKV;
    if (MASK == ET_MASK_CAUSAL) {
        const int last_q = (q0 + BQ - 1 < a.seq ? q0 + BQ - 1 : a.seq - 1);
        const int lim = last_q / BKV + 1;
        n_kv = n_kv < lim ? n_kv : lim;
    }
    const int passes = n_kv > 1 ? 2 : 1;  // statistics pass only when a row spans several blocks
    // Task t of this CTA: (head, pass, key block), in that order of nesting.
    const int per_head = passes * n_kv;
    const int n_task = (h_end - h_begin) * per_head;

    if (warp == 0) {
        // ---------------- Q / K producer ----------------
        if (n_task > 0 && elect_one()) {
            int h = h_begin, in_head = 0, t = 0;
            for (; t < n_task; ++t) {
                const int s = t % qk_stages;
                if (!mbar_wait_bounded(&qk_empty[s], ((t / qk_stages) & 1) ^ 1, abort_flag)) {
                    report_error(a.err_word, abort_flag, DEV_TIMEOUT_VO_PRODUCER);
                    break;
                }
                const int j = in_head >= n_kv ? in_head - n_kv : in_head;
                uint8_t* st = sQK + s * qk_stage_bytes;
                mbar_arrive_expect_tx(&qk_full[s], qk_stage_bytes);
                for (int i = 0; i < nqa; ++i) {
                    tma_load_3d(st + i * ATOM_BYTES, &tmQ, &qk_full[s], h * a.dh_qk + i * 64, q0, b);
                    tma_load_3d(st + (nqa + i) * ATOM_BYTES, &tmK, &qk_full[s], h * a.dh_qk + i * 64,
                                j * BKV, b);
                }
                if (++in_head == per_head) {
                    in_head = 0;
                    ++h;
                }
            }
            if (*abort_flag)  // let copies in flight land before shared memory is released
                for (int i = t > qk_stages ? t - qk_stages : 0; i < t; ++i)
                    for (uint32_t it = 0; it < ET_SPIN_LIMIT; ++it)
                        if (mbar_try_wait(&qk_full[i % qk_stages], (i / qk_stages) & 1)) break;
        }
    } else if (warp == 2) {
        // ---------------- VO producer: half blocks of 64 keys ----------------
        if (n_task > 0 && elect_one()) {
            const int halves = 2 * n_kv;
            const int total = (h_end - h_begin) * halves;
            int h = h_begin, in_head = 0, i = 0;
            for (; i < total; ++i) {
                const int s = i % VO_STAGES;
                if (!mbar_wait_bounded_relaxed(&vo_empty[s], ((i / VO_STAGES) & 1) ^ 1, abort_flag)) {
                    report_error(a.err_word, abort_flag, DEV_TIMEOUT_VO_PRODUCER);
                    break;
                }
                mbar_arrive_expect_tx(&vo_full[s], nca * VO_ATOM);
                for (int c = 0; c < nca; ++c)
                    tma_load_3d(sVO + s * vo_stage_bytes(NC) + c * VO_ATOM, &tmVO, &vo_full[s],
                                e0 + c * 64, in_head * VO_KEYS, b * a.nhead + h);
                if (++in_head == halves) {
                    in_head = 0;
                    ++h;
                }
            }
            if (*abort_flag)
                for (int k = i > VO_STAGES ? i - VO_STAGES : 0; k < i; ++k)
                    for (uint32_t it = 0; it < ET_SPIN_LIMIT; ++it)
                        if (mbar_try_wait(&vo_full[k % VO_STAGES], (k / VO_STAGES) & 1)) break;
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (warp-uniform, one elected lane issues) ----------------
        if (n_task > 0) {
            const bool leader = elect_one();
            const uint32_t idesc_s = make_idesc_f16(BQ, BKV, 0, 0);
            const uint32_t idesc_o = make_idesc_f16(BQ, n_c, 0, 1);  // VO is MN-major
            const uint32_t qk_lo = desc_lo(smem_u32(sQK)), p_lo = desc_lo(smem_u32(sP));
            const uint32_t vo_lo =
                ((smem_u32(sVO) & 0x3FFFFu) >> 4) | (static_cast<uint32_t>(VO_ATOM >> 4) << 16);
            const int ksteps = a.dh_qk >> 4;
            auto issue_s = [&](int t) -> bool {
                const int s = t & (qk_stages - 1);
                if (!mbar_wait_bounded_warp(&qk_full[s], (qk_stages == 2 ? t >> 1 : t) & 1, abort_flag) ||
                    !mbar_wait_bounded_warp(&s_free[t & 1], ((t >> 1) & 1) ^ 1, abort_flag))
                    return false;
                tc_fence_after_sync();
                const uint32_t q_lo = qk_lo + s * (qk_stage_bytes >> 4);
                const uint32_t k_lo = q_lo + nqa * (ATOM_BYTES >> 4);
                if (leader) {
                    for (int kk = 0; kk < ksteps; ++kk) {
                        const uint32_t off = (kk >> 2) * (ATOM_BYTES >> 4) + (kk & 3) * 2;
                        mma_f16_ss_k128(tmem_base + (t & 1) * BKV, q_lo + off, k_lo + off, idesc_s,
                                        kk != 0 ? 1u : 0u);
                    }
                    mma_commit(&s_full[t & 1]);
                    mma_commit(&qk_empty[s]);
                }
                __syncwarp();
                return true;
            };
            bool ok = issue_s(0);
            int in_head = 0, t_b = 0, v = 0;
            uint32_t vph = 0;
            for (int t = 0; ok && t < n_task; ++t) {
                if (t + 1 < n_task) ok = issue_s(t + 1);
                if (!ok) break;
                if (in_head >= per_head - n_kv) {
                    ok = mbar_wait_bounded_warp(p_full, t_b & 1, abort_flag);
                    for (int half = 0; ok && half < 2; ++half) {
                        ok = mbar_wait_bounded_warp(&vo_full[v], vph, abort_flag);
                        if (!ok) break;
                        tc_fence_after_sync();
                        if (leader) {
#pragma unroll
                            for (int kk = 0; kk < VO_KEYS / 16; ++kk)
                                mma_f16_ss_k128(tmem_O, p_lo + half * (ATOM_BYTES >> 4) + kk * 2,
                                                vo_lo + v * (vo_stage_bytes(NC) >> 4) + kk * (2048 >> 4),
                                                idesc_o, (t_b | half | kk) != 0 ? 1u : 0u);
                            mma_commit(&vo_empty[v]);
                        }
                        __syncwarp();
                        if (++v == VO_STAGES) {
                            v = 0;
                            vph ^= 1u;
                        }
                    }
                    if (!ok) break;
                    if (leader) mma_commit(pv_done);
                    __syncwarp();
                    ++t_b;
                }
                if (++in_head == per_head) in_head = 0;
            }
            if (!ok && leader) report_error(a.err_word, abort_flag, DEV_TIMEOUT_VO_MMA);
            __syncwarp();
        }
    } else {
        // ---------------- softmax warps: two per quadrant, 64 keys of a query row each --------
        const int qd = warp & 3;
        const int hf = (warp - 3) >> 2;
        const int r = qd * 32 + lane;
        const int qrow = q0 + r;
        const uint32_t lane_off = static_cast<uint32_t>(qd * 32) << 16;
        const float NINF = -INFINITY;
        float* x_a = s_x;           // [2 halves][128 rows]: maxima
        float* x_b = s_x + 2 * BQ;  // [2 halves][128 rows]: sums
        const __half* mrow = (MASK == ET_MASK_ADDITIVE && qrow < a.seq)
                                 ? a.mask + static_cast<size_t>(qrow) * a.seq
                                 : nullptr;
        auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(2 + qd) : "memory"); };
        int t = 0, t_b = 0;
        bool ok = true;

        // this thread's 64 scores of task t, scaled and masked (log2 domain); frees the buffer
        auto fetch = [&](float (&s)[64], int kbase, int j) -> float {
            uint32_t v0[32], v1[32];
            const uint32_t addr = tmem_base + (t & 1) * BKV + lane_off + hf * 64;
            tmem_ld32(addr, v0);
            tmem_ld32(addr + 32, v1);
            tmem_ld_wait_regs(v0);
            tmem_ld_wait_regs(v1);
            tc_fence_before_sync();
            mbar_arrive(&s_free[t & 1]);
            float mx = NINF;
#pragma unroll
            for (int i = 0; i < 64; ++i)
                s[i] = __uint_as_float(i < 32 ? v0[i & 31] : v1[i & 31]) * a.scale_log2;
            const bool need_mask = (j * BKV + BKV > kv_len) || (MASK == ET_MASK_ADDITIVE) ||
                                   (MASK == ET_MASK_CAUSAL && j * BKV + BKV - 1 > q0);
            if (need_mask) {
#pragma unroll
                for (int i = 0; i < 64; ++i) {
                    const int kc = kbase + i;
                    if (kc >= kv_len || (MASK == ET_MASK_CAUSAL && kc > qrow)) s[i] = NINF;
                    else if (MASK == ET_MASK_ADDITIVE && mrow)
                        s[i] += __half2float(__ldcg(reinterpret_cast<const __half*>(mrow + kc))) *
                                1.4426950408889634f;
                }
            }
#pragma unroll
            for (int i = 0; i < 64; ++i) mx = fmaxf(mx, s[i]);
            return mx;
        };
        auto wait_scores = [&]() -> bool {
            bool good = mbar_wait_bounded(&s_full[t & 1], (t >> 1) & 1, abort_flag);
            good = __all_sync(0xffffffffu, good);
            if (good) tc_fence_after_sync();
            return good;
        };

        // A warp whose wait ran out keeps walking (every later wait is skipped), so that the pair
        // barriers match.
        for (int h = h_begin; n_kv > 0 && h < h_end; ++h) {
            float m_use = 0.f, inv = 0.f;
            if (passes == 2) {
                // each half keeps a running max and sum of its own keys; the halves meet once
                float m_run = NINF, l_run = 0.f;
                for (int j = 0; j < n_kv; ++j) {
                    ok = ok && wait_scores();
                    float s[64];
                    const float mx = fetch(s, j * BKV + hf * 64, j);
                    const float m_new = fmaxf(m_run, mx);
                    const float neg = (m_new == NINF) ? 0.f : -m_new;
                    float sum = 0.f;
#pragma unroll
                    for (int i = 0; i < 64; ++i) sum += exp2_approx(s[i] + neg);
                    l_run = l_run * exp2_approx(m_run + neg) + sum;
                    m_run = m_new;
                    ++t;
                }
                x_a[hf * BQ + r] = m_run;
                x_b[hf * BQ + r] = l_run;
                pair_sync();
                const float m_o = x_a[(hf ^ 1) * BQ + r], l_o = x_b[(hf ^ 1) * BQ + r];
                const float m_all = fmaxf(m_run, m_o);
                m_use = (m_all == NINF) ? 0.f : m_all;
                // (the same order of addition in both halves)
                const float l0 = (hf == 0 ? l_run : l_o) * exp2_approx((hf == 0 ? m_run : m_o) - m_use);
                const float l1 = (hf == 0 ? l_o : l_run) * exp2_approx((hf == 0 ? m_o : m_run) - m_use);
                const float l_all = l0 + l1;
                inv = l_all > 0.f ? 1.0f / l_all : 0.f;
                pair_sync();  // the exchange slots are free for the next head
            }
            for (int j = 0; j < n_kv; ++j) {
                ok = ok && wait_scores();
                float s[64];
                const float mx = fetch(s, j * BKV + hf * 64, j);
                if (passes == 1) {
                    x_a[hf * BQ + r] = mx;
                    pair_sync();
                    const float m_all = fmaxf(mx, x_a[(hf ^ 1) * BQ + r]);
                    m_use = (m_all == NINF) ? 0.f : m_all;
                }
                float sum = 0.f;
#pragma unroll
                for (int i = 0; i < 64; ++i) {
                    s[i] = exp2_approx(s[i] - m_use);
                    sum += s[i];
                }
                if (passes == 1) {
                    x_b[hf * BQ + r] = sum;
                    pair_sync();
                    const float l_all = x_b[r] + x_b[BQ + r];
                    inv = l_all > 0.f ? 1.0f / l_all : 0.f;
                }
                uint32_t p[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) p[i] = pack_half2(s[2 * i] * inv, s[2 * i + 1] * inv);
                if (ok && t_b > 0) {  // the previous product has read the P tile
                    ok = mbar_wait_bounded(pv_done, (t_b - 1) & 1, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                }
                uint8_t* prow = sP + hf * ATOM_BYTES + r * 128;
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    *reinterpret_cast<uint4*>(prow + ((g ^ (r & 7)) * 16)) =
                        make_uint4(p[4 * g], p[4 * g + 1], p[4 * g + 2], p[4 * g + 3]);
                fence_proxy_async_smem();
                mbar_arrive(p_full);
                ++t;
                ++t_b;
            }
        }
        if (ok && t_b > 0) {
            ok = mbar_wait_bounded(pv_done, (t_b - 1) & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
        }
        if (!ok) report_error(a.err_word, abort_flag, DEV_TIMEOUT_VO_SOFTMAX);
        tc_fence_after_sync();
    }

    // ---------------- the heads' partial sums meet, rows dealt to the ranks ----------------
    // Every product of every CTA is complete, so the operand stages may be overwritten.  (A CTA
    // whose wait ran out takes the same barriers.)
    __syncwarp();
    if (csize > 1) cluster_sync_all(); else __syncthreads();
    const int rows_per = (BQ + csize - 1) / csize;
    constexpr int pitch = vo_pitch(NC);
    if (warp >= 3 && !*abort_flag) {
        const int qd = warp & 3;
        const int hf = (warp - 3) >> 2;
        const int r = qd * 32 + lane;
        const uint32_t lane_off = static_cast<uint32_t>(qd * 32) << 16;
        const int owner = r / rows_per;
        const uint32_t local = smem_u32(smem + (rank * rows_per + (r - owner * rows_per)) * pitch);
        const uint32_t dst = csize > 1 ? map_to_cta(local, owner) : local;
        for (int c = hf; c < (n_c >> 4); c += 2) {
            uint32_t o[16];
            if (n_task > 0) {
                tmem_ld16(tmem_O + lane_off + c * 16, o);
                tmem_ld_wait();
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = 0u;
            }
#pragma unroll
            for (int g = 0; g < 4; ++g)
                st_cluster_v4(dst + c * 64 + g * 16, o[4 * g], o[4 * g + 1], o[4 * g + 2], o[4 * g + 3]);
        }
    }
    __syncwarp();
    if (csize > 1) cluster_sync_all(); else __syncthreads();
    if (!*abort_flag) {
        const int r0 = rank * rows_per;
        int nrow = BQ - r0 < rows_per ? BQ - r0 : rows_per;
        nrow = a.seq - q0 - r0 < nrow ? a.seq - q0 - r0 : nrow;
        const int pieces = n_c >> 3;
        for (int i = threadIdx.x; i < nrow * pieces; i += VO_THREADS) {
            const int rl = i / pieces, c = (i - rl * pieces) * 8;
            float f[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) f[k] = 0.f;
            for (int g = 0; g < csize; ++g) {
                const float4* src =
                    reinterpret_cast<const float4*>(smem + (g * rows_per + rl) * pitch + c * 4);
                const float4 u = src[0], w = src[1];
                f[0] += u.x; f[1] += u.y; f[2] += u.z; f[3] += u.w;
                f[4] += w.x; f[5] += w.y; f[6] += w.z; f[7] += w.w;
            }
            if (a.bias_o != nullptr) {
                const uint4 bq = __ldg(reinterpret_cast<const uint4*>(a.bias_o + e0 + c));
                const __half2* bh = reinterpret_cast<const __half2*>(&bq);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 bf = __half22float2(bh[k]);
                    f[2 * k] += bf.x;
                    f[2 * k + 1] += bf.y;
                }
            }
            uint4 w;
            w.x = pack_half2(f[0], f[1]);
            w.y = pack_half2(f[2], f[3]);
            w.z = pack_half2(f[4], f[5]);
            w.w = pack_half2(f[6], f[7]);
            *reinterpret_cast<uint4*>(a.out + (static_cast<size_t>(b) * a.seq + q0 + r0 + rl) * a.emdim +
                                      e0 + c) = w;
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, VO_TMEM_COLS);
}

}  // namespace
}  // namespace et

namespace et {

int g_vo_chunk = 0;  // test hook: 64 / 128 / 256 output features per CTA, 0 = automatic

// out[t, c] = bias[c] (0 without a bias) for every element.
__global__ void vo_fill_bias_kernel(__half* __restrict__ out, const __half* __restrict__ bias, int T,
                                    int emdim) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t total = static_cast<size_t>(T) * emdim;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x)
        out[i] = bias ? __ldg(bias + i % emdim) : __float2half_rn(0.f);
}

// out[t, col_id[k]] = comp[t, k] + bias[col_id[k]]: the kept features of a column-pruned result.
__global__ void vo_scatter_cols_kernel(const __half* __restrict__ comp, const int* __restrict__ col_id,
                                       const __half* __restrict__ bias, __half* __restrict__ out,
                                       int T, int nnz_col, int emdim) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t total = static_cast<size_t>(T) * nnz_col;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t t = i / nnz_col;
        const int c = __ldg(col_id + (i - t * nnz_col));
        if (c < 0 || c >= emdim) continue;
        const float b = bias ? __half2float(__ldg(bias + c)) : 0.f;
        out[t * emdim + c] = __float2half_rn(__half2float(__ldcg(comp + i)) + b);
    }
}

}  // namespace et

extern "C" {

int et_fused_vo_attention_fwd(const et_half* Q, const et_half* K, const et_half* VO,
                              const et_half* bias_o, et_half* out, int batch, int seq, int nhead,
                              int dh_qk, int emdim, int ldq, int ldk, int mask_kind,
                              const et_half* mask, const int32_t* valid_len, float scale,
                              et_stream stream) {
    using namespace et;
    if (!Q || !K || !VO || !out || batch <= 0 || seq <= 0 || nhead <= 0 || dh_qk <= 0 || emdim <= 0)
        return ET_ERR_INVALID_ARG;
    if (mask_kind < ET_MASK_NONE || mask_kind > ET_MASK_ADDITIVE) return ET_ERR_INVALID_ARG;
    if (mask_kind == ET_MASK_ADDITIVE && !mask) return ET_ERR_INVALID_ARG;
    if (mask_kind == ET_MASK_PADDING && !valid_len) return ET_ERR_INVALID_ARG;
    if (dh_qk % 16 || dh_qk > 128 || emdim % 16) return ET_ERR_SHAPE;
    if (ldq % 8 || ldk % 8 || ldq < nhead * dh_qk || ldk < nhead * dh_qk) return ET_ERR_SHAPE;
    if (batch > 65535 || static_cast<long>(batch) * nhead > 0x7fffffffL) return ET_ERR_SHAPE;
    if (!aligned16(Q) || !aligned16(K) || !aligned16(VO) || !aligned16(out) ||
        (bias_o && !aligned16(bias_o)))
        return ET_ERR_ALIGNMENT;
    int* err = device_error_word();
    if (!err) return ET_ERR_NO_DEVICE;

    CUtensorMap tmQ, tmK, tmVO;
    auto make = [&](CUtensorMap* m, const void* p, int ld, int width, int groups, uint32_t rows) {
        const uint32_t box[3] = {64, rows, 1};
        const uint64_t dims[3] = {static_cast<uint64_t>(width), static_cast<uint64_t>(seq),
                                  static_cast<uint64_t>(groups)};
        const uint64_t strides[2] = {static_cast<uint64_t>(ld) * 2,
                                     static_cast<uint64_t>(ld) * 2 * static_cast<uint64_t>(seq)};
        return make_tensor_map_f16(m, p, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    };
    int st;
    if ((st = make(&tmQ, Q, ldq, nhead * dh_qk, batch, BQ)) != ET_OK) return st;
    if ((st = make(&tmK, K, ldk, nhead * dh_qk, batch, BKV)) != ET_OK) return st;
    if ((st = make(&tmVO, VO, emdim, emdim, batch * nhead, VO_KEYS)) != ET_OK) return st;

    VoArgs a;
    a.out = reinterpret_cast<__half*>(out);
    a.bias_o = reinterpret_cast<const __half*>(bias_o);
    a.mask = reinterpret_cast<const __half*>(mask);
    a.valid_len = valid_len;
    a.batch = batch;
    a.seq = seq;
    a.nhead = nhead;
    a.dh_qk = dh_qk;
    a.emdim = emdim;
    a.scale_log2 = scale * 1.4426950408889634f;
    a.err_word = err;
    // Heads are dealt to as many CTAs per item (up to 8, a portable cluster) as keep the launch
    // within one CTA per SM: a CTA's time is its serial walk over its heads.  The count is taken
    // for 256-feature items whatever the chunk width, so that every width adds the heads' partial
    // sums in the same order.
    int nc = 256;
    if (g_vo_chunk == 64 || g_vo_chunk == 128) nc = g_vo_chunk;
    const int sms = sm_count() > 0 ? sm_count() : 148;
    const long qblocks = (seq + BQ - 1) / BQ;
    const long items = qblocks * ((emdim + 255) / 256) * batch;
    long csize = sms / items;
    csize = csize > VO_MAX_CLUSTER ? VO_MAX_CLUSTER : csize;
    csize = csize > nhead ? nhead : csize;
    csize = csize < 1 ? 1 : csize;
    int dev = 0;
    cudaGetDevice(&dev);
    auto go = [&](auto kern, int slot, int width) -> int {
        const int smem_bytes = vo_smem_bytes(width);
        static std::atomic<bool> attr_set[12][64] = {};
        if (dev >= 0 && dev < 64 && !attr_set[slot][dev]) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) !=
                cudaSuccess)
                return ET_ERR_CUDA;
            attr_set[slot][dev] = true;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(csize * qblocks),
                           static_cast<unsigned>((emdim + width - 1) / width), static_cast<unsigned>(batch));
        cfg.blockDim = dim3(VO_THREADS);
        cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
        cfg.stream = static_cast<cudaStream_t>(stream);
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
        return cudaLaunchKernelEx(&cfg, kern, tmQ, tmK, tmVO, a) == cudaSuccess ? ET_OK : ET_ERR_CUDA;
    };
    auto by_mask = [&](auto width) -> int {
        constexpr int W = decltype(width)::value;
        constexpr int base = W == 256 ? 0 : (W == 128 ? 4 : 8);
        switch (mask_kind) {
            case ET_MASK_CAUSAL: return go(attention_vo_kernel<W, ET_MASK_CAUSAL>, base + 1, W);
            case ET_MASK_PADDING: return go(attention_vo_kernel<W, ET_MASK_PADDING>, base + 2, W);
            case ET_MASK_ADDITIVE: return go(attention_vo_kernel<W, ET_MASK_ADDITIVE>, base + 3, W);
            default: return go(attention_vo_kernel<W, ET_MASK_NONE>, base, W);
        }
    };
    if (nc == 64) return by_mask(std::integral_constant<int, 64>{});
    if (nc == 128) return by_mask(std::integral_constant<int, 128>{});
    return by_mask(std::integral_constant<int, 256>{});
}

#ifdef ET_TEST_HOOKS
// Test hook: output features per CTA of the pre-multiplied V.O attention (64 / 128 / 256), 0 = automatic.
void et_debug_set_vo_chunk(int nc) { et::g_vo_chunk = nc; }
#endif  // ET_TEST_HOOKS

// ---- column-pruned V.O (Linear_VO_prune + Fused_prune_Multihead_attention) -----------------
// The pre-multiplied weight keeps only the output features col_id[0 .. nnz_col): VO_c is
// [batch][nhead][seq][nnz_col]; the attention runs at that width and its result is scattered
// back to the full feature dimension (pruned features carry the output bias alone).

int et_linear_vo_pruned_fwd(const et_half* X, const et_half* Wvo_c, const et_half* bias,
                            et_half* VOc, int batch, int seq, int nhead, int emdim, int nnz_col,
                            et_stream stream) {
    if (batch <= 0 || seq <= 0 || nhead <= 0 || emdim <= 0 || nnz_col <= 0) return ET_ERR_INVALID_ARG;
    if (emdim % 16 || nnz_col % 16) return ET_ERR_SHAPE;
    return et::launch_gemm_f16_grouped_kn(
        reinterpret_cast<const __half*>(X), emdim, reinterpret_cast<const __half*>(Wvo_c),
        reinterpret_cast<const __half*>(bias), reinterpret_cast<__half*>(VOc), batch * seq, nnz_col,
        emdim, nhead, seq, static_cast<cudaStream_t>(stream));
}

int et_fused_vo_attention_pruned_fwd(const et_half* Q, const et_half* K, const et_half* VOc,
                                     const int32_t* col_id, int nnz_col, const et_half* bias_o,
                                     et_half* scratch, et_half* out, int batch, int seq, int nhead,
                                     int dh_qk, int emdim, int ldq, int ldk, int mask_kind,
                                     const et_half* mask, const int32_t* valid_len, float scale,
                                     et_stream stream) {
    if (!col_id || !scratch || !out || nnz_col <= 0 || emdim <= 0) return ET_ERR_INVALID_ARG;
    if (nnz_col % 16 || emdim % 8 || nnz_col > emdim) return ET_ERR_SHAPE;
    if (!et::aligned16(out) || !et::aligned16(scratch) || (bias_o && !et::aligned16(bias_o)))
        return ET_ERR_ALIGNMENT;
    int st = et_fused_vo_attention_fwd(Q, K, VOc, nullptr, scratch, batch, seq, nhead, dh_qk, nnz_col,
                                       ldq, ldk, mask_kind, mask, valid_len, scale, stream);
    if (st != ET_OK) return st;
    const int T = batch * seq;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t total = static_cast<size_t>(T) * emdim;
    const int blocks = static_cast<int>((total + 255) / 256 < 2048 ? (total + 255) / 256 : 2048);
    if (et::launch_kernel(et::vo_fill_bias_kernel, dim3(blocks), dim3(256), 0, s,
                          reinterpret_cast<__half*>(out), reinterpret_cast<const __half*>(bias_o), T,
                          emdim) != cudaSuccess)
        return ET_ERR_CUDA;
    const size_t totc = static_cast<size_t>(T) * nnz_col;
    const int blocks2 = static_cast<int>((totc + 255) / 256 < 2048 ? (totc + 255) / 256 : 2048);
    return et::launch_kernel(et::vo_scatter_cols_kernel, dim3(blocks2), dim3(256), 0, s,
                             reinterpret_cast<const __half*>(scratch), col_id,
                             reinterpret_cast<const __half*>(bias_o), reinterpret_cast<__half*>(out),
                             T, nnz_col, emdim) == cudaSuccess
               ? ET_OK
               : ET_ERR_CUDA;
}

}  // extern "C"

