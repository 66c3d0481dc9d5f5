// On-the-fly fused self-attention for heads of up to 64 features: one query row per thread, persistent.
//
// Two CTAs share an SM and walk items of 128 queries of one (sequence, head).  Warp 0 streams Q and
// K / V blocks of 128 keys with TMA (K and V through two-stage rings), warp 1 issues S = Q.K^T and
// O += P.V, and each thread of the four softmax warps owns ONE whole query row: it walks the row's 128
// scores in tensor memory, 32 columns at a time with the next 32 in flight, for their maximum and then
// again for exp2 (the half that is still in registers first), and writes the fp16 probabilities back into
// tensor memory, where they are the A operand of P.V.  No value crosses threads, so a block costs no named
// barrier, no shared-memory exchange and no proxy fence; the scores' columns are handed back in the middle
// of the exponentials, and the next block's Q.K^T runs under the rest.  Loads and Q.K^T run ahead into the
// next item, whose first scores are there when the output of the last one has left.
//
// What bounds it: the special-function unit (16 exp2 per clock and SM: 1024 cycles a 128 x 128 block)
// and what a warp cannot hide of its own chain: clock stamps gave 2330 cycles a block to a CTA alone and
// 2740 to each of two, of which 300 are the maximum, 240 the raise decision and 1600 the exponentials,
// before these drained once instead of four times a block.  Every fourth pair of exponentials runs on the
// FMA pipe, whose issue slots are two thirds free: 1 x 4096 94.4 -> 86.9 us, 256 x 512 328 -> 309 us; 5 / 16,
// 3 / 8 and half of them measured 88.8, 92 and 99 us on the first.
// Against the kernel that splits a row over two threads (attention_body.cuh), 64-wide heads: 256 x 512
// tokens, 12 heads 430 -> 309 us; 32 x 384, 16 heads 53 -> 38.5 us; 4 x 2048 causal, 16 heads 92 -> 60 us;
// 1 x 4096 98.5 -> 86.9 us (384 items on 296 CTAs: the second round is a third full); 16 x 128, one item per
// CTA, 6.9 -> 7.2 us.
//
// Tensor memory: S in columns [0, 128), O in [128, 192), P in [192, 256): 256 columns, two CTAs' worth.
// All waits are bounded.
#include "attention_body.cuh"

namespace et {
namespace {

using namespace attn;

constexpr int AR_SM_WARPS = 4;
constexpr int AR_THREADS = 64 + 32 * AR_SM_WARPS;
constexpr int AR_KV = 2;  // K / V ring stages
constexpr int AR_SMEM = (2 + 2 * AR_KV) * ATOM_BYTES + 256 + 1024;
static_assert(2 * AR_SMEM <= 227 * 1024, "two CTAs per SM");
constexpr uint32_t AR_COL_O = 128, AR_COL_P = 192;

// D[tmem] (+)= A[tmem] . B[smem]; B's descriptor by its low word (128-byte swizzle).
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t"
        "}\n"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(DESC_HI_K128)
        : "memory");
}

// The work items: (query block, head or work unit, sequence), dealt to the persistent CTAs round by
// round, every other round backwards, so that a CTA that drew a long item draws a short one next.
struct RowsSched {
    int items, nqb, nh, batch;
    int heavy_first;  // 1: query blocks vary slowest, the last (causal: longest) ones first
};

// 2^x of both lanes on the FMA pipe, for x <= 64: x = n + r with n whole and |r| <= 1/2, 2^r by a degree-5
// polynomial (Remez fit of the relative error on [-1/2, 1/2]; 2.1e-7 at worst in fp32, as far off as
// ex2.approx may be), 2^n through the exponent field.  Below -126 it returns 2^-126, which is zero as an fp16
// probability; NaN stays NaN.
__device__ __forceinline__ uint64_t exp2_poly_f32x2(uint64_t x2) {
    float x0, x1;
    unpack_f32x2(x2, x0, x1);
    asm("max.NaN.f32 %0, %0, 0fC2FC0000;" : "+f"(x0));  // -126
    asm("max.NaN.f32 %0, %0, 0fC2FC0000;" : "+f"(x1));
    const uint64_t x = pack_f32x2(x0, x1);
    const uint64_t magic = pack_f32x2(12582912.f, 12582912.f), unmagic = pack_f32x2(-12582912.f, -12582912.f);
    const uint64_t t = add_f32x2(x, magic);  // the whole part in the low mantissa bits
    const uint64_t minus1 = pack_f32x2(-1.f, -1.f);
    const uint64_t r = fma_f32x2(add_f32x2(t, unmagic), minus1, x);
    auto both = [](float c) { return pack_f32x2(c, c); };
    uint64_t p = fma_f32x2(both(0.0013276472f), r, both(0.009675541f));
    p = fma_f32x2(p, r, both(0.05550713f));
    p = fma_f32x2(p, r, both(0.2402212f));
    p = fma_f32x2(p, r, both(0.69314694f));
    p = fma_f32x2(p, r, both(1.0000001f));
    float t0, t1;
    unpack_f32x2(t, t0, t1);
    const float s0 = __uint_as_float((__float_as_uint(t0) << 23) + 0x3f800000u);
    const float s1 = __uint_as_float((__float_as_uint(t1) << 23) + 0x3f800000u);
    return mul_f32x2(p, pack_f32x2(s0, s1));
}

template <int MASK>
__global__ void __launch_bounds__(AR_THREADS, 2)
attention_rows_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmZ,
                      const AttnArgs a, const RowsSched sched) {
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment computed on the shared-window offset, so that the pointer keeps its
    // shared-memory provenance (plain LDS / STS instead of generic accesses)
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + ATOM_BYTES;
    uint8_t* sV = sK + AR_KV * ATOM_BYTES;
    uint8_t* sZ = sV + AR_KV * ATOM_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sZ + ATOM_BYTES);
    uint64_t* k_full = bars;             // [2]
    uint64_t* k_empty = k_full + AR_KV;  // [2]
    uint64_t* v_full = k_empty + AR_KV;  // [2]
    uint64_t* v_empty = v_full + AR_KV;  // [2]
    uint64_t* q_full = v_empty + AR_KV;
    uint64_t* q_empty = q_full + 1;
    uint64_t* s_full = q_empty + 1;
    uint64_t* s_free = s_full + 1;
    uint64_t* p_full = s_free + 1;
    uint64_t* o_full = p_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = uniform_warp_id();
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        for (int s = 0; s < AR_KV; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        mbar_init(q_full, 1);
        mbar_init(q_empty, 1);
        mbar_init(s_full, 1);
        mbar_init(s_free, AR_SM_WARPS);
        mbar_init(p_full, AR_SM_WARPS);
        mbar_init(o_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TMEM_COLS_ATT);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();
    pdl_wait();  // Q, K, V come from the previous kernel; Z may still be read by an earlier one

    // One item: 128 queries from q0 of head h of sequence b against n_kv blocks of keys.
    struct Item {
        int q0, h, b, kv_len, n_kv;
    };
    // Moves `round` on to this CTA's next item (any, or one with keys) and describes it; false at the end.
    auto seek = [&](int& round, Item& w, bool with_keys) -> bool {
        for (;; ++round) {
            const int base = round * static_cast<int>(gridDim.x);
            if (base >= sched.items) return false;
            const int t = base + static_cast<int>((round & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
            if (t >= sched.items) continue;
            int qb, hh;
            if (sched.heavy_first) {
                const int per = sched.nh * sched.batch, rest = t % per;
                qb = sched.nqb - 1 - t / per;
                hh = rest % sched.nh;
                w.b = rest / sched.nh;
            } else {
                const int rest = t / sched.nqb;
                qb = t - rest * sched.nqb;
                hh = rest % sched.nh;
                w.b = rest / sched.nh;
            }
            w.q0 = ((a.n_units > 0 ? a.unit_first[hh] : 0) + qb) * BQ;
            w.h = a.n_units > 0 ? a.unit_head[hh] : hh;
            w.kv_len = a.seq;
            if (MASK == ET_MASK_PADDING) {
                const int len = a.valid_len[w.b];
                w.kv_len = len < 0 ? 0 : (len > a.seq ? a.seq : len);
            }
            w.n_kv = (w.kv_len + BKV - 1) / BKV;
            if (MASK == ET_MASK_CAUSAL) {
                const int last_q = (w.q0 + BQ - 1 < a.seq ? w.q0 + BQ - 1 : a.seq - 1);
                const int lim = last_q / BKV + 1;
                w.n_kv = w.n_kv < lim ? w.n_kv : lim;
            }
            if (w.n_kv > 0 || !with_keys) return true;
        }
    };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (elect_one()) {
            Item w;
            int n_items = 0, k_issued = 0, v_issued = 0;
            bool ok = true;
            for (int round = 0; ok && seek(round, w, true); ++round) {
                // Q's atom is free once the previous item's last Q.K^T has read it
                ok = mbar_wait_bounded_relaxed(q_empty, (n_items & 1) ^ 1, abort_flag);
                if (!ok) break;
                mbar_arrive_expect_tx(q_full, ATOM_BYTES);
                tma_load_3d(sQ, &tmQ, q_full, w.h * a.dh_qk, w.q0, w.b);
                ++n_items;
                for (int j = 0; j < w.n_kv; ++j) {
                    const int s = k_issued & 1;
                    const uint32_t ph = (k_issued >> 1) & 1;
                    ok = mbar_wait_bounded_relaxed(&k_empty[s], ph ^ 1, abort_flag);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&k_full[s], ATOM_BYTES);
                    tma_load_3d(sK + s * ATOM_BYTES, &tmK, &k_full[s], w.h * a.dh_qk, j * BKV, w.b);
                    ++k_issued;
                    ok = mbar_wait_bounded_relaxed(&v_empty[s], ph ^ 1, abort_flag);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&v_full[s], ATOM_BYTES);
                    tma_load_3d(sV + s * ATOM_BYTES, &tmV, &v_full[s], w.h * a.dh_v, j * BKV, w.b);
                    ++v_issued;
                }
            }
            if (!ok) report_error(a.err_word, abort_flag, DEV_TIMEOUT_ATTN_PRODUCER);
            if (*abort_flag) {
                // let copies in flight land before shared memory is released
                if (n_items > 0)
                    for (uint32_t it = 0; it < ET_SPIN_LIMIT; ++it)
                        if (mbar_try_wait(q_full, (n_items - 1) & 1)) break;
                for (int i = k_issued > AR_KV ? k_issued - AR_KV : 0; i < k_issued; ++i)
                    for (uint32_t it = 0; it < ET_SPIN_LIMIT; ++it)
                        if (mbar_try_wait(&k_full[i & 1], (i >> 1) & 1)) break;
                for (int i = v_issued > AR_KV ? v_issued - AR_KV : 0; i < v_issued; ++i)
                    for (uint32_t it = 0; it < ET_SPIN_LIMIT; ++it)
                        if (mbar_try_wait(&v_full[i & 1], (i >> 1) & 1)) break;
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (warp-uniform, one elected lane issues) ----------------
        // Blocks are numbered through all of the CTA's items; Q.K^T runs one block ahead of P.V, across
        // the end of an item too.
        const bool leader = elect_one();
        const uint32_t idesc_s = make_idesc_f16(BQ, BKV, 0, 0);
        const uint32_t idesc_o = make_idesc_f16(BQ, a.dh_v, 0, 1);  // V is MN-major
        const uint32_t q_lo = desc_lo(smem_u32(sQ)), k_lo = desc_lo(smem_u32(sK));
        // V tile: 16 keys = two groups of 8 rows of 128 bytes (stride 1024); one feature atom
        const uint32_t v_lo =
            ((smem_u32(sV) & 0x3FFFFu) >> 4) | (static_cast<uint32_t>(ATOM_BYTES >> 4) << 16);
        const int ksteps = a.dh_qk >> 4;
        Item ws, wo;
        int round_s = 0, js = 0, gs = 0, item_s = 0;
        bool more_s = seek(round_s, ws, true);
        bool ok = true;
        auto issue_s = [&]() -> bool {
            const int s = gs & 1;
            if ((js == 0 && !mbar_wait_bounded_warp(q_full, item_s & 1, abort_flag)) ||
                !mbar_wait_bounded_warp(&k_full[s], (gs >> 1) & 1, abort_flag) ||
                !mbar_wait_bounded_warp(s_free, (gs & 1) ^ 1, abort_flag))
                return false;
            tc_fence_after_sync();
            const bool last = js + 1 == ws.n_kv;
            if (leader) {
                const uint32_t kl = k_lo + s * (ATOM_BYTES >> 4);
                for (int kk = 0; kk < ksteps; ++kk)
                    mma_f16_ss_k128(tmem_base, q_lo + kk * 2, kl + kk * 2, idesc_s, kk != 0 ? 1u : 0u);
                mma_commit(s_full);
                mma_commit(&k_empty[s]);
                if (last) mma_commit(q_empty);
            }
            __syncwarp();
            ++gs;
            ++js;
            if (last) {
                js = 0;
                ++item_s;
                ++round_s;
                more_s = seek(round_s, ws, true);
            }
            return true;
        };
        if (more_s) ok = issue_s();
        int go = 0;
        for (int round_o = 0; ok && seek(round_o, wo, true); ++round_o) {
            for (int j = 0; ok && j < wo.n_kv; ++j, ++go) {
                const int s = go & 1;
                if (more_s) ok = issue_s();  // runs under this block's softmax
                ok = ok && mbar_wait_bounded_warp(&v_full[s], (go >> 1) & 1, abort_flag) &&
                     mbar_wait_bounded_warp(p_full, go & 1, abort_flag);
                if (!ok) break;
                tc_fence_after_sync();
                if (leader) {
                    const uint32_t vl = v_lo + s * (ATOM_BYTES >> 4);
#pragma unroll
                    for (int kk = 0; kk < BKV / 16; ++kk)
                        mma_f16_ts(tmem_base + AR_COL_O, tmem_base + AR_COL_P + kk * 8,
                                   vl + kk * (2048 >> 4), idesc_o, (j | kk) != 0 ? 1u : 0u);
                    mma_commit(o_full);
                    mma_commit(&v_empty[s]);
                }
                __syncwarp();
            }
        }
        if (!ok && leader) report_error(a.err_word, abort_flag, DEV_TIMEOUT_ATTN_MMA);
        __syncwarp();
    } else {
        // ---------------- softmax / output warps ----------------
        const int qd = warp & 3;          // tensor-memory lane quadrant
        const int r = qd * 32 + lane;     // row inside the CTA tile
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(qd * 32) << 16);
        const float NINF = -INFINITY;
        const uint64_t scale2 = pack_f32x2(a.scale_log2, a.scale_log2);
        bool ok = true;
        int g = 0;  // blocks so far
        Item w;

        for (int round = 0; ok && seek(round, w, false); ++round) {
            const int qrow = w.q0 + r;  // position inside the sequence
            float m_run = NINF, l_run = 0.f;
            for (int j = 0; j < w.n_kv; ++j, ++g) {
                ok = mbar_wait_bounded(s_full, g & 1, abort_flag);
                if (!ok) report_error(a.err_word, abort_flag, DEV_TIMEOUT_ATTN_SOFTMAX);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after_sync();

                const int kbase = j * BKV;
                const bool need_mask = (kbase + BKV > w.kv_len) ||
                                       (MASK == ET_MASK_CAUSAL && kbase + BKV - 1 > w.q0);
                // the row's last key of this block that takes part, counted from the block's first
                int lim = w.kv_len - 1 - kbase;
                if (MASK == ET_MASK_CAUSAL) lim = lim < qrow - kbase ? lim : qrow - kbase;
                auto mask_chunk = [&](uint32_t (&v)[32], int c) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = c * 32 + i <= lim ? v[i] : 0xff800000u;  // -inf
                };

                uint32_t ra[32], rb[32];
                // pass 1: the maximum of the row
                float m4[4] = {NINF, NINF, NINF, NINF};
                auto max_chunk = [&](uint32_t (&v)[32], int c) {
                    if (need_mask) mask_chunk(v, c);
#pragma unroll
                    for (int i = 0; i < 32; i += 2)
                        m4[(i >> 1) & 3] = fmaxf(m4[(i >> 1) & 3],
                                                 fmaxf(__uint_as_float(v[i]), __uint_as_float(v[i + 1])));
                };
                tmem_ld32(lane_base, ra);
                tmem_ld_wait_regs(ra);
                tmem_ld32(lane_base + 32, rb);
                max_chunk(ra, 0);
                tmem_ld_wait_regs(rb);
                tmem_ld32(lane_base + 64, ra);
                max_chunk(rb, 1);
                tmem_ld_wait_regs(ra);
                tmem_ld32(lane_base + 96, rb);
                max_chunk(ra, 2);
                tmem_ld_wait_regs(rb);
                max_chunk(rb, 3);
                // (the scale is positive)
                const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale_log2;

                // raise the running maximum only when it is -inf or the block exceeds it by more
                // than the slack
                const bool raise = (m_run == NINF) || (mx > m_run + RESCALE_SLACK);
                const float m_new = raise ? fmaxf(m_run, mx) : m_run;
                const float m_use = (m_new == NINF) ? 0.f : m_new;
                const float alpha = raise ? exp2_approx(m_run - m_use) : 1.0f;  // 0 when m_run = -inf

                if (j > 0) {
                    // P of the previous block must have been consumed, O produced
                    ok = mbar_wait_bounded(o_full, (g & 1) ^ 1, abort_flag);
                    if (!ok) report_error(a.err_word, abort_flag, DEV_TIMEOUT_ATTN_SOFTMAX);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (!__all_sync(0xffffffffu, alpha == 1.0f)) {
                        for (int c = 0; c < (a.dh_v >> 4); ++c) {
                            uint32_t o[16];
                            tmem_ld16(lane_base + AR_COL_O + c * 16, o);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                            tmem_st16(lane_base + AR_COL_O + c * 16, o);
                        }
                        tmem_st_wait();
                    }
                }

                // pass 2: probabilities -> tensor memory (A operand of P.V), their sum
                const uint64_t neg_m2 = pack_f32x2(-m_use, -m_use);
                uint64_t sum2[2] = {0ull, 0ull};
                auto exp_chunk = [&](const uint32_t (&v)[32], int c) {
                    uint32_t p[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const uint64_t x2 =
                            fma_f32x2(pack_f32x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])),
                                      scale2, neg_m2);
                        float e0, e1;
                        if ((i & 3) == 3) {
                            unpack_f32x2(exp2_poly_f32x2(x2), e0, e1);
                        } else {
                            unpack_f32x2(x2, e0, e1);
                            e0 = exp2_approx(e0);
                            e1 = exp2_approx(e1);
                        }
                        sum2[i & 1] = add_f32x2(sum2[i & 1], pack_f32x2(e0, e1));
                        p[i] = pack_half2(e0, e1);
                    }
                    tmem_st16(lane_base + AR_COL_P + c * 16, p);
                };
                // the last two chunks are still in registers (masked), the first two are read again
                // meanwhile: the exponentials drain once a block, not once a chunk
                exp_chunk(ra, 2);
                tmem_ld32(lane_base, ra);
                exp_chunk(rb, 3);
                tmem_ld32(lane_base + 32, rb);
                tmem_ld_wait_regs(ra);
                tmem_ld_wait_regs(rb);
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_free);  // S may be overwritten by the next Q.K^T
                if (need_mask) {
                    mask_chunk(ra, 0);
                    mask_chunk(rb, 1);
                }
                exp_chunk(ra, 0);
                exp_chunk(rb, 1);
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full);

                float s0, s1, s2, s3;
                unpack_f32x2(sum2[0], s0, s1);
                unpack_f32x2(sum2[1], s2, s3);
                l_run = l_run * alpha + ((s0 + s1) + (s2 + s3));
                m_run = m_new;
            }

            if (ok && w.n_kv > 0) {
                ok = mbar_wait_bounded(o_full, (g & 1) ^ 1, abort_flag);
                if (!ok) report_error(a.err_word, abort_flag, DEV_TIMEOUT_ATTN_SOFTMAX);
                ok = __all_sync(0xffffffffu, ok);
            }
            if (!ok) break;
            tc_fence_after_sync();
            const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
            const bool staged = a.tma_out && w.n_kv > 0;
            __half* zrow = a.Z + (static_cast<size_t>(w.b) * a.seq + (qrow < a.seq ? qrow : 0)) * a.ldz +
                           static_cast<size_t>(w.h) * a.dh_v;
            uint8_t* srow = sZ + r * 128;
            if (staged) {
                if (lane == 0) tma_store_wait_read();  // this warp's rows of the previous item
                __syncwarp();
            }
            uint32_t oa[32], ob[32];  // (columns past dh_v are not used)
            if (w.n_kv > 0) {
                tmem_ld32(lane_base + AR_COL_O, oa);
                tmem_ld32(lane_base + AR_COL_O + 32, ob);
                tmem_ld_wait_regs(oa);
                tmem_ld_wait_regs(ob);
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) oa[i] = ob[i] = 0u;
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                if (c * 8 >= a.dh_v) break;
                uint32_t h2[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = (c & 3) * 8 + 2 * i;
                    h2[i] = pack_half2(__uint_as_float(c < 4 ? oa[n] : ob[n]) * inv,
                                       __uint_as_float(c < 4 ? oa[n + 1] : ob[n + 1]) * inv);
                }
                const uint4 piece = make_uint4(h2[0], h2[1], h2[2], h2[3]);
                if (staged)
                    *reinterpret_cast<uint4*>(srow + ((c ^ (r & 7)) * 16)) = piece;
                else if (qrow < a.seq)
                    *reinterpret_cast<uint4*>(zrow + c * 8) = piece;
            }
            if (staged) {
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0 && w.q0 + qd * 32 < a.seq) {
                    tma_store_3d(&tmZ, sZ + qd * 32 * 128, w.h * a.dh_v, w.q0 + qd * 32, w.b);
                    tma_store_commit();
                }
            }
        }
        if (lane == 0) tma_store_wait_read();
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS_ATT);
}

template <int MASK>
int launch_rows_mask(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV,
                     const CUtensorMap& tmZ, const AttnArgs& a, const RowsSched& sched, cudaStream_t stream) {
    static std::atomic<bool> attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (cudaFuncSetAttribute(attention_rows_kernel<MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 AR_SMEM) != cudaSuccess)
            return ET_ERR_CUDA;
        attr_set[dev] = true;
    }
    const int slots = 2 * (sm_count() > 0 ? sm_count() : 148);
    const dim3 grid(static_cast<unsigned>(sched.items < slots ? sched.items : slots));
    return launch_kernel(attention_rows_kernel<MASK>, grid, dim3(AR_THREADS), AR_SMEM, stream, tmQ, tmK,
                         tmV, tmZ, a, sched) == cudaSuccess
               ? ET_OK
               : ET_ERR_CUDA;
}

}  // namespace

namespace attn {

bool attention_rows_applies(int dh_qk, int dh_v, dim3 blocks) {
    return dh_qk <= 64 && dh_v <= 64 && static_cast<long long>(blocks.x) * blocks.y * blocks.z <= (1 << 30);
}

int launch_attention_rows(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV,
                          const CUtensorMap& tmZ, const AttnArgs& a, dim3 blocks, cudaStream_t stream) {
    RowsSched sched;
    sched.nqb = static_cast<int>(blocks.x);
    sched.nh = static_cast<int>(blocks.y);
    sched.batch = static_cast<int>(blocks.z);
    sched.items = sched.nqb * sched.nh * sched.batch;
    // Causal items differ in length.  With few rounds the long ones go first (their keys, 32 KB a head and
    // block, stay in L2 meanwhile); with many, neighbours share keys and the rounds even out.
    const int sms = sm_count() > 0 ? sm_count() : 148;
    sched.heavy_first = a.mask_kind == ET_MASK_CAUSAL && sched.items <= 8 * sms;
    switch (a.mask_kind) {
        case ET_MASK_CAUSAL: return launch_rows_mask<ET_MASK_CAUSAL>(tmQ, tmK, tmV, tmZ, a, sched, stream);
        case ET_MASK_PADDING: return launch_rows_mask<ET_MASK_PADDING>(tmQ, tmK, tmV, tmZ, a, sched, stream);
        default: return launch_rows_mask<ET_MASK_NONE>(tmQ, tmK, tmV, tmZ, a, sched, stream);
    }
}

}  // namespace attn
}  // namespace et
