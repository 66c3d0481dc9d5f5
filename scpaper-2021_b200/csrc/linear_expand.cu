// Linear layers over irregular weight formats on the tensor cores:
//     Y[T, out] = act(X[T, in] . W^T + bias),   W stored as 1x16 vectors, packed 16x16 tiles or CSR.
//
// The tensor core cannot skip single vectors or values, but expanding them is cheap next to
// multiplying: a CTA owns BN output features and MB blocks of 128 tokens, and eight warps write the
// non-zero weights of the next K block into a zeroed, 128-byte-swizzled operand tile in shared
// memory - the layout a TMA load of a dense weight would produce - while the tensor core works on
// earlier ones.  The expanded weight never exists in global memory, and one expansion serves all MB
// token blocks (their accumulators, MB x BN columns, share tensor memory).
//
// Roles: warp 0 streams 128 x 64 activation tiles with TMA, one thread of warp 1 issues
// tcgen05.mma (M = 128, N = BN, K = 16), warps 2-9 expand and then run the epilogue (bias,
// activation, fp16, staging tile, 16-byte row stores).  All waits are bounded.
//
// What bounds it: a K block costs max(2 * BN, 240) tensor-pipe cycles per token block and pulls 16 KB
// of activations, 64 B/clk at BN = 128, within what an SM gets from L2; weights arrive compressed.
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "gemm_common.cuh"
#include "kernels.h"

namespace et {
namespace {

using namespace gemm;

enum : int { FMT_VEC = 0, FMT_PACKED = 1, FMT_CSRM = 2 };

constexpr int X_MAX_A = 8;                       // activation stages at most
constexpr int X_MAX_B = 4;                       // weight buffers at most
constexpr int X_MAX_MB = 8;                      // token blocks per CTA at most
constexpr int X_CSR_A = 4;                       // CSR: activation stages,
constexpr int X_CSR_BYTES = 128 * 1024;          // and bytes of expanded columns at most
constexpr int X_EXP_WARPS = EPI_WARPS;           // expander / epilogue warps
constexpr int X_EXP_THREADS = 32 * X_EXP_WARPS;
constexpr int X_ROW_LIST = 128 + 1;

struct ExpandArgs {
    // 1x16: tile_idx / row_idx / data; packed: masks / offsets / tiles; CSR: indptr / indices / data
    const int* idx0;
    const int* idx1;
    const __half* data;
    const __half* bias;
    const __half* X;
    __half* Y;
    int T, in, out, act;
    int mb;         // token blocks per CTA
    int ckb, nbuf;  // K blocks per weight buffer, weight buffers
    int na;         // activation stages
    int tmem_cols;
    int groups;     // CTAs along the tokens
    int vec_store;  // 1: 16-byte stores to Y are possible
    int* err_word;
};

// Writes the non-zero values of output rows [n0 + 16 set, + 16) x K block `kb` of a 1x16 weight
// into `tile` (16 rows of 128 bytes); one warp.  Indices are fetched two blocks ahead and vectors
// one block ahead of their use, so a block costs no exposed L2 round trip.
struct VecExpander {
    const int* tidx;  // this set's npart + 1 offsets
    const int* row_idx;
    const uint4* data;
    int npart;
    int lane;
    int b_next, b_next2;  // lane l < 5: offset of part 4 kb + l of the next blocks
    // the fetched block: up to 64 vectors, two per lane
    uint4 v[2][2];
    int pos[2];  // row * 4 + part of the vector, or -1

    __device__ __forceinline__ int offset_of(int kb) const {
        int p = kb * 4 + (lane < 5 ? lane : 4);
        p = p < npart ? p : npart;
        return __ldg(tidx + p);
    }
    __device__ __forceinline__ void fetch(int bounds) {
        const int o0 = __shfl_sync(0xffffffffu, bounds, 0), o1 = __shfl_sync(0xffffffffu, bounds, 1);
        const int o2 = __shfl_sync(0xffffffffu, bounds, 2), o3 = __shfl_sync(0xffffffffu, bounds, 3);
        const int o4 = __shfl_sync(0xffffffffu, bounds, 4);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = o0 + u * 32 + lane;
            pos[u] = -1;
            if (i < o4) {
                const int part = (i >= o1) + (i >= o2) + (i >= o3);
                pos[u] = (__ldg(row_idx + i) & 15) * 4 + part;
                v[u][0] = __ldg(data + static_cast<size_t>(i) * 2);
                v[u][1] = __ldg(data + static_cast<size_t>(i) * 2 + 1);
            }
        }
    }
    __device__ __forceinline__ void init(const ExpandArgs& a, int rset, int lane_) {
        lane = lane_;
        npart = a.in >> 4;
        tidx = a.idx0 + static_cast<size_t>(rset) * (npart + 1);
        row_idx = a.idx1;
        data = reinterpret_cast<const uint4*>(a.data);
    }
    __device__ __forceinline__ void start(int kb, int step) {
        const int b = offset_of(kb);
        b_next = offset_of(kb + step);
        b_next2 = offset_of(kb + 2 * step);
        fetch(b);
    }
    // writes block kb (already fetched) and moves on to kb + step
    __device__ __forceinline__ void write(uint8_t* tile, int kb, int step) {
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (pos[u] >= 0) {
                const int row = pos[u] >> 2, c = (pos[u] & 3) * 2;
                uint8_t* line = tile + row * 128;
                *reinterpret_cast<uint4*>(line + ((c ^ (row & 7)) * 16)) = v[u][0];
                *reinterpret_cast<uint4*>(line + (((c + 1) ^ (row & 7)) * 16)) = v[u][1];
            }
        const int b = b_next;
        b_next = b_next2;
        b_next2 = offset_of(kb + 3 * step);
        fetch(b);
    }
};

// The same for packed tile-CSR: block row r of its panel, up to four 16x16 tiles per K block.
struct PackedExpander {
    const uint32_t* mask;
    const int* off;
    const uint4* tiles;
    int nchunk, r, lane;
    uint32_t m_next, m_next2;
    int o_next, o_next2;
    uint4 v[4];
    uint32_t have;

    __device__ __forceinline__ void index_of(int kb, uint32_t& m, int& o) const {
        m = kb < nchunk ? __ldg(mask + kb) : 0u;
        o = kb < nchunk ? __ldg(off + kb) : 0;
    }
    __device__ __forceinline__ void fetch(uint32_t m, int o) {
        have = (m >> (4 * r)) & 0xFu;
        int slot = o + __popc(m & ((1u << (4 * r)) - 1u));
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if ((have >> c) & 1u) v[c] = __ldg(tiles + static_cast<size_t>(slot++) * 32 + lane);
    }
    __device__ __forceinline__ void init(const ExpandArgs& a, int br, int lane_) {
        lane = lane_;
        nchunk = (a.in + 63) >> 6;
        r = br & 7;
        mask = reinterpret_cast<const uint32_t*>(a.idx0) + static_cast<size_t>(br >> 3) * nchunk;
        off = a.idx1 + static_cast<size_t>(br >> 3) * nchunk;
        tiles = reinterpret_cast<const uint4*>(a.data);
    }
    __device__ __forceinline__ void start(int kb, int step) {
        uint32_t m;
        int o;
        index_of(kb, m, o);
        index_of(kb + step, m_next, o_next);
        index_of(kb + 2 * step, m_next2, o_next2);
        fetch(m, o);
    }
    __device__ __forceinline__ void write(uint8_t* tile, int kb, int step) {
        // the stored tile's 16-byte unit `lane`: row lane / 2, its halves swapped in rows 4-7, 12-15
        const int row = lane >> 1, half = (lane & 1) ^ ((row >> 2) & 1);
        uint8_t* line = tile + row * 128;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if ((have >> c) & 1u)
                *reinterpret_cast<uint4*>(line + (((c * 2 + half) ^ (row & 7)) * 16)) = v[c];
        const uint32_t m = m_next;
        const int o = o_next;
        m_next = m_next2;
        o_next = o_next2;
        index_of(kb + 3 * step, m_next2, o_next2);
        fetch(m, o);
    }
};

// Output feature n of one token from the stored entries alone.  The expanded operand multiplies every
// activation, by zero where nothing is stored, which is the same sum as long as the token is finite; the
// epilogue asks here for elements that are not, so that an infinity or NaN reaches exactly the outputs
// that store a weight for it (a vector or a tile is stored whole).
template <int FMT>
__device__ __noinline__ float stored_product(const int* idx0, const int* idx1, const __half* data, int in,
                                             int n, const __half* x) {
    float acc = 0.f;
    auto dot16 = [&](const __half* w, int k) {
        for (int j = 0; j < 16; ++j) acc += __half2float(__ldg(w + j)) * __half2float(__ldcg(x + k + j));
    };
    if (FMT == FMT_CSRM) {
        for (int e = __ldg(idx0 + n); e < __ldg(idx0 + n + 1); ++e) {
            const int k = __ldg(idx1 + e);
            if (k >= 0 && k < in) acc += __half2float(__ldg(data + e)) * __half2float(__ldcg(x + k));
        }
    } else if (FMT == FMT_VEC) {
        const int npart = in >> 4;
        const int* tidx = idx0 + static_cast<size_t>(n >> 4) * (npart + 1);
        for (int p = 0; p < npart; ++p)
            for (int i = __ldg(tidx + p); i < __ldg(tidx + p + 1); ++i)
                if ((__ldg(idx1 + i) & 15) == (n & 15)) dot16(data + static_cast<size_t>(i) * 16, p * 16);
    } else {
        const int nchunk = (in + 63) >> 6, r4 = ((n >> 4) & 7) * 4, row = n & 15;
        for (int kb = 0; kb < nchunk; ++kb) {
            const size_t at = static_cast<size_t>(n >> 7) * nchunk + kb;
            const uint32_t m = __ldg(reinterpret_cast<const uint32_t*>(idx0) + at);
            int slot = __ldg(idx1 + at) + __popc(m & ((1u << r4) - 1u));
            for (int c = 0; c < 4; ++c) {
                if (!((m >> (r4 + c)) & 1u)) continue;
                const __half* w = data + static_cast<size_t>(slot++) * 256 + row * 16;
                for (int j = 0; j < 16; ++j)  // (halves swapped in rows 4-7 and 12-15)
                    acc += __half2float(__ldg(w + (j ^ (((row >> 2) & 1) * 8)))) *
                           __half2float(__ldcg(x + kb * 64 + c * 16 + j));
            }
        }
    }
    return acc;
}

template <int FMT, int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
linear_expand_kernel(const __grid_constant__ CUtensorMap tmX, const ExpandArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int buf_bytes = g.ckb * BN * 128;
    uint8_t* sA = smem;
    uint8_t* sB = smem + g.na * A_STAGE_BYTES;
    uint8_t* misc = sB + g.nbuf * buf_bytes;
    uint64_t* a_full = reinterpret_cast<uint64_t*>(misc);
    uint64_t* a_empty = a_full + X_MAX_A;
    uint64_t* b_full = a_empty + X_MAX_A;
    uint64_t* b_empty = b_full + X_MAX_B;
    uint64_t* acc_full = b_empty + X_MAX_B;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* s_any_dup = reinterpret_cast<int*>(tmem_slot + 2);
    float* s_bias = reinterpret_cast<float*>(misc + 256);         // [BN]
    int* s_ptr = reinterpret_cast<int*>(s_bias + BN);             // CSR: [BN + 1] row starts
    int* s_dup = s_ptr + X_ROW_LIST;                              // CSR: [BN] row holds duplicates

    const int warp = uniform_warp_id();
    const int lane = threadIdx.x & 31;
    const int n0 = static_cast<int>(blockIdx.x / g.groups) * BN;
    const int m0 = static_cast<int>(blockIdx.x % g.groups) * g.mb * BM;
    int mb = (g.T - m0 + BM - 1) / BM;  // token blocks of this CTA
    mb = mb < g.mb ? mb : g.mb;
    const int nkb = (g.in + BK - 1) / BK;
    const int nchunk = (nkb + g.ckb - 1) / g.ckb;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmX);
        for (int s = 0; s < X_MAX_A; ++s) {
            mbar_init(&a_full[s], 1);
            mbar_init(&a_empty[s], 1);
        }
        for (int s = 0; s < X_MAX_B; ++s) {
            mbar_init(&b_full[s], X_EXP_WARPS);
            mbar_init(&b_empty[s], 1);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        *s_any_dup = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, g.tmem_cols);
        tmem_relinquish();
    }
    for (int i = threadIdx.x; i < BN; i += GEMM_THREADS) {
        s_bias[i] = (g.bias != nullptr && n0 + i < g.out) ? __half2float(__ldg(g.bias + n0 + i)) : 0.f;
        if (FMT == FMT_CSRM) s_dup[i] = 0;
    }
    if (FMT == FMT_CSRM)
        for (int i = threadIdx.x; i <= BN; i += GEMM_THREADS)
            s_ptr[i] = __ldg(g.idx0 + (n0 + i < g.out ? n0 + i : g.out));
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();

    if (warp == 0) {
        // ---------------- activation producer ----------------
        if (elect_one()) {
            pdl_wait();
            int it = 0, s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int kb = 0; ok && kb < nkb; ++kb)
                for (int tb = 0; tb < mb; ++tb, ++it) {
                    if (!mbar_wait_bounded(&a_empty[s], ph ^ 1, abort_flag)) {
                        report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_PRODUCER);
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&a_full[s], A_STAGE_BYTES);
                    tma_load_2d(sA + s * A_STAGE_BYTES, &tmX, &a_full[s], kb * BK, m0 + tb * BM);
                    if (++s == g.na) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            if (*abort_flag)  // let copies in flight land before shared memory is released
                for (int i = it > g.na ? it - g.na : 0; i < it; ++i)
                    for (uint32_t sp = 0; sp < ET_SPIN_LIMIT; ++sp)
                        if (mbar_try_wait(&a_full[i % g.na], (i / g.na) & 1)) break;
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // The whole warp walks the loop and one elected lane issues: control flow and descriptors
        // stay warp-uniform, which is what the issue instructions take their operands from.
        const bool leader = elect_one();
        constexpr uint32_t idesc = make_idesc_f16(BM, BN, 0, 0);
        const uint32_t a_base = desc_lo(smem_u32(sA)), b_base = desc_lo(smem_u32(sB));
        int s = 0, buf = 0;
        uint32_t ph = 0, bph = 0;
        bool ok = true;
        for (int c = 0; ok && c < nchunk; ++c) {
            if (!mbar_wait_bounded_warp(&b_full[buf], bph, abort_flag)) {
                ok = false;
                break;
            }
            const int kb_end = (c + 1) * g.ckb < nkb ? (c + 1) * g.ckb : nkb;
            uint32_t b_lo = b_base + ((buf * buf_bytes) >> 4);
            for (int kb = c * g.ckb; ok && kb < kb_end; ++kb, b_lo += (BN * 128) >> 4) {
                for (int tb = 0; tb < mb; ++tb) {
                    if (!mbar_wait_bounded_warp(&a_full[s], ph, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t a_lo = a_base + s * (A_STAGE_BYTES >> 4);
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)
                            mma_f16_ss_k128(tmem_base + tb * BN, a_lo + k * 2, b_lo + k * 2, idesc,
                                            (kb | k) != 0 ? 1u : 0u);
                        mma_commit(&a_empty[s]);
                    }
                    __syncwarp();
                    if (++s == g.na) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (leader) mma_commit(&b_empty[buf]);
            __syncwarp();
            if (++buf == g.nbuf) {
                buf = 0;
                bph ^= 1u;
            }
        }
        if (ok) {
            if (leader) mma_commit(acc_full);
        } else if (leader) {
            report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_MMA);
        }
        __syncwarp();
    } else {
        const int w = warp - 2;
        const int tid = threadIdx.x - 64;
        bool ok = true;
        // ---------------- expansion (weights only: no wait for earlier kernels) ----------------
        if (FMT == FMT_CSRM) {
            // Entries of the CTA's rows are one contiguous run, walked flat by all threads; an
            // entry finds its row by binary search.  A weight buffer holds as many columns as fit
            // (all of them up to in = 1024 or 2048), so the run is walked once per buffer and the
            // entries of a row may be in any order.
            const int e_begin = s_ptr[0], e_end = s_ptr[BN];
            for (int c = 0; c < nchunk; ++c) {
                const int buf = c % g.nbuf;
                if (ok) {
                    ok = mbar_wait_bounded(&b_empty[buf], ((c / g.nbuf) & 1) ^ 1, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                }
                uint8_t* tile = sB + buf * buf_bytes;
                for (int i = tid; i < buf_bytes / 16; i += X_EXP_THREADS)
                    reinterpret_cast<uint4*>(tile)[i] = make_uint4(0u, 0u, 0u, 0u);
                asm volatile("bar.sync 1, %0;" ::"n"(X_EXP_THREADS) : "memory");
                const int k0 = c * g.ckb * BK;
                const int width = g.ckb * BK;
                for (int e0 = e_begin + tid; e0 < e_end; e0 += 4 * X_EXP_THREADS) {
                    int col[4];
                    unsigned short val[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int e = e0 + u * X_EXP_THREADS;
                        col[u] = e < e_end ? __ldg(g.idx1 + e) : -1;
                        val[u] = e < e_end ? __ldg(reinterpret_cast<const unsigned short*>(g.data) + e) : 0;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int k = col[u] - k0;
                        if (col[u] < 0 || col[u] >= g.in || k < 0 || k >= width || (val[u] & 0x7fff) == 0)
                            continue;
                        const int e = e0 + u * X_EXP_THREADS;
                        int lo = 0, hi = BN - 1;  // the last row that starts at or before e
                        while (lo < hi) {
                            const int mid = (lo + hi + 1) >> 1;
                            if (s_ptr[mid] <= e) lo = mid; else hi = mid - 1;
                        }
                        uint8_t* word = tile + (k >> 6) * (BN * 128) + lo * 128 +
                                        ((((k & 63) >> 3) ^ (lo & 7)) * 16) + (k & 6) * 2;
                        const int sh = (k & 1) * 16;
                        // the buffer starts at zero and every stored (row, column) is added once,
                        // so the integer add is a store that does not disturb the word's other half
                        const uint32_t old = atomicAdd(reinterpret_cast<uint32_t*>(word),
                                                       static_cast<uint32_t>(val[u]) << sh);
                        if ((old >> sh) & 0xffffu) {  // stored twice: the epilogue recomputes the row
                            s_dup[lo] = 1;
                            *s_any_dup = 1;
                        }
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&b_full[buf]);
            }
        } else {
            // Item (16 output rows, K block) of a buffer per warp: BN / 16 row sets x ckb blocks = 8.
            constexpr int SETS = BN / 16;
            const int set = w % SETS, sub = w / SETS;  // sub < ckb
            const bool live = n0 + set * 16 < g.out;
            typename std::conditional<FMT == FMT_VEC, VecExpander, PackedExpander>::type x;
            if (live) {
                x.init(g, (n0 >> 4) + set, lane);
                x.start(sub, g.ckb);
            }
            int buf = 0;
            uint32_t bph = 0;
            for (int c = 0; c < nchunk; ++c) {
                if (ok) {
                    ok = mbar_wait_bounded(&b_empty[buf], bph ^ 1, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                }
                uint8_t* tile = sB + buf * buf_bytes + sub * (BN * 128) + set * (16 * 128);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    reinterpret_cast<uint4*>(tile)[i * 32 + lane] = make_uint4(0u, 0u, 0u, 0u);
                __syncwarp();
                if (live) x.write(tile, c * g.ckb + sub, g.ckb);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&b_full[buf]);
                if (++buf == g.nbuf) {
                    buf = 0;
                    bph ^= 1u;
                }
            }
        }

        // ---------------- epilogue ----------------
        const int q = warp & 3;
        const int half = w >> 2;
        pdl_wait();  // Y may still be read by an earlier kernel
        if (ok) {
            ok = mbar_wait_bounded_relaxed(acc_full, 0, abort_flag);
            if (!ok) report_error(g.err_word, abort_flag, DEV_TIMEOUT_GEMM_EPILOGUE);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            tc_fence_after_sync();
            // units of 32 rows x 64 (or 32) columns, dealt to the quadrant's two warps; the staging
            // tile reuses the idle activation ring
            constexpr int GROUP = BN < 64 ? BN : 64;
            constexpr int NG = BN / GROUP;
            uint8_t* tile = sA + w * 4096;
            const bool any_dup = FMT == FMT_CSRM && *reinterpret_cast<volatile int*>(s_any_dup) != 0;
            bool odd = false;  // a row of this thread is not finite: see below
            for (int u = half; u < mb * NG; u += 2) {
                const int tb = u / NG, cg = u - tb * NG;
                const int n_base = n0 + cg * GROUP;
                const int row0 = m0 + tb * BM + q * 32;
                if (row0 >= g.T || n_base >= g.out) continue;
                const uint32_t addr = tmem_base + tb * BN + cg * GROUP + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll
                for (int h = 0; h < GROUP / 32; ++h) {
                    uint32_t r[32];
                    tmem_ld32(addr + h * 32, r);
                    tmem_ld_wait_regs(r);
                    odd = odd || (r[0] & 0x7f800000u) == 0x7f800000u;
                    const float* b32 = s_bias + cg * GROUP + h * 32;
                    if (g.act == ET_ACT_GELU) stage_f16_chunk<ET_ACT_GELU>(r, b32, tile + lane * 128, h, lane);
                    else if (g.act == ET_ACT_RELU) stage_f16_chunk<ET_ACT_RELU>(r, b32, tile + lane * 128, h, lane);
                    else stage_f16_chunk<ET_ACT_NONE>(r, b32, tile + lane * 128, h, lane);
                }
                __syncwarp();
                if (g.vec_store) {
                    constexpr int PIECES = GROUP / 8, ROWS = 32 / PIECES;
                    const int piece = lane % PIECES, n = n_base + piece * 8;
#pragma unroll
                    for (int i = 0; i < 32 / ROWS; ++i) {
                        const int rr = i * ROWS + lane / PIECES;
                        if (row0 + rr < g.T && n < g.out)
                            *reinterpret_cast<uint4*>(g.Y + static_cast<size_t>(row0 + rr) * g.out + n) =
                                *reinterpret_cast<const uint4*>(tile + rr * 128 + ((piece ^ (rr & 7)) * 16));
                    }
                } else {
                    for (int rr = 0; rr < 32 && row0 + rr < g.T; ++rr)
                        for (int j = lane; j < GROUP && n_base + j < g.out; j += 32)
                            g.Y[static_cast<size_t>(row0 + rr) * g.out + n_base + j] =
                                *reinterpret_cast<const __half*>(tile + rr * 128 +
                                                                 (((j >> 3) ^ (rr & 7)) * 16) + (j & 7) * 2);
                }
                __syncwarp();
            }
            // Elements to be summed again from the stored entries: rows of the weight that hold a column
            // twice, and whatever is not finite.  (An activation that is not finite leaves no element of its
            // row finite, so one of 32 tells.  A pass of its own: inside the loop above it cost 3 % of
            // 1024 -> 3072 at 3072 tokens.)
            if (any_dup || __any_sync(0xffffffffu, odd))
                for (int u = half; u < mb * NG; u += 2) {
                    const int tb = u / NG, cg = u - tb * NG;
                    const int row0 = m0 + tb * BM + q * 32, m = row0 + lane;
                    if (row0 >= g.T || n0 + cg * GROUP >= g.out) continue;
                    for (int h = 0; h < GROUP / 32; ++h) {
                        const int nl = cg * GROUP + h * 32;  // first of 32 columns
                        uint32_t r[32];
                        __syncwarp();
                        tmem_ld32(tmem_base + tb * BN + nl + (static_cast<uint32_t>(q * 32) << 16), r);
                        tmem_ld_wait_regs(r);
                        uint32_t redo = 0;
                        if (any_dup)
                            redo = __ballot_sync(0xffffffffu, reinterpret_cast<volatile int*>(s_dup)[nl + lane]);
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            redo |= (r[j] & 0x7f800000u) == 0x7f800000u ? 1u << j : 0u;
                        for (; m < g.T && redo != 0; redo &= redo - 1) {
                            const int j = __ffs(redo) - 1, n = n0 + nl + j;
                            if (n >= g.out) break;
                            const float y = stored_product<FMT>(g.idx0, g.idx1, g.data, g.in, n,
                                                                g.X + static_cast<size_t>(m) * g.in) +
                                            s_bias[nl + j];
                            g.Y[static_cast<size_t>(m) * g.out + n] = __float2half_rn(apply_act(y, g.act));
                        }
                    }
                }
        }
    }

    pdl_wait();  // no CTA may retire before the kernels it depends on have completed
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, g.tmem_cols);
}

template <int FMT, int BN>
int launch_bn(const CUtensorMap& tmX, ExpandArgs& a, cudaStream_t stream) {
    const int buf = a.ckb * BN * 128;
    constexpr int misc = 256 + BN * 4 + (FMT == FMT_CSRM ? (X_ROW_LIST + BN) * 4 : 0);
    const int smem = a.na * A_STAGE_BYTES + a.nbuf * buf + misc + 1024;
    auto kern = linear_expand_kernel<FMT, BN>;
    // once, to the most that any width needs: two threads that each raised it to their own size could leave
    // the smaller one standing
    constexpr int most = (FMT == FMT_CSRM ? X_CSR_A * A_STAGE_BYTES + X_CSR_BYTES
                                          : X_MAX_A * A_STAGE_BYTES + X_MAX_B * 128 * 128) + misc + 1024;
    static_assert(most <= 227 * 1024, "shared memory budget exceeded");
    static std::atomic<bool> attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess)
            return ET_ERR_CUDA;
        attr_set[dev] = true;
    }
    const long panels = (a.out + BN - 1) / BN;
    return launch_kernel(kern, dim3(static_cast<unsigned>(panels * a.groups)), dim3(GEMM_THREADS), smem,
                         stream, tmX, a) == cudaSuccess
               ? ET_OK
               : ET_ERR_CUDA;
}

struct ExpandPlan {
    int bn;
    long panels, waves, cycles;
};

// Fills in a.mb, a.groups, a.ckb, a.nbuf and a.na.
template <int FMT>
ExpandPlan plan_expand(ExpandArgs& a) {
    const int sms = sm_count() > 0 ? sm_count() : 148;
    const long tblocks = (a.T + BM - 1) / BM;
    const int nkb = (a.in + BK - 1) / BK;
    // Width: 128 features unless that leaves most SMs idle - a K block costs the tensor pipe 256
    // cycles at N = 128 and still 240 at N = 64 or 32, but narrow panels expand and drain sooner.
    auto panels = [&](int bn) { return static_cast<long>((a.out + bn - 1) / bn); };
    int bn = 128;
    while (bn > 32 && panels(bn) * tblocks * 2 <= sms) bn >>= 1;
    // CSR buffers are walked once each: wide buffers need narrow panels
    if (FMT == FMT_CSRM && bn > 64) bn = 64;
    // Token blocks per CTA: the count whose waves x time is least; a CTA costs about 4000 cycles of
    // set-up and epilogue besides its K blocks.
    const int mb_max = 512 / bn < X_MAX_MB ? 512 / bn : X_MAX_MB;
    long best = -1, best_waves = 0;
    for (int mb = 1; mb <= mb_max && mb <= tblocks; ++mb) {
        const long groups = (tblocks + mb - 1) / mb;
        const long waves = (panels(bn) * groups + sms - 1) / sms;
        const long cost = waves * (4000 + static_cast<long>(mb) * (nkb * (bn == 128 ? 256 : 240) + 600));
        if (best < 0 || cost < best) {
            best = cost;
            best_waves = waves;
            a.mb = mb;
            a.groups = static_cast<int>(groups);
        }
    }
    if (FMT == FMT_CSRM) {
        const int fit = X_CSR_BYTES / (bn * 128);
        a.ckb = nkb < fit ? nkb : fit;
        a.nbuf = 1;
        a.na = X_CSR_A;
    } else {
        a.ckb = 128 / bn;  // eight warps, one (row set, K block) item each
        a.nbuf = X_MAX_B;
        a.na = X_MAX_A;
    }
    return ExpandPlan{bn, panels(bn), best_waves, best};
}

// Whether the kernel whose work follows the stored values (linear_misc.cu) is expected to be faster than
// expanding them, which costs a dense product whatever is stored.  Both times in microseconds, fitted to B200
// runs at 512 -> 512, 768 -> 768, 1024 -> 3072, 3072 -> 768 and 4096 -> 1024, 1 to 8192 tokens and 0 to 50 %
// stored: the faster one is chosen, or one within 20 % of it.  By values, by expansion: 3072 -> 768 at 2048 tokens
// 0.1 % stored 10.0 / 22.2, 0.5 % 22.5 / 25.2, 1 % 39.8 / 28.9; 1024 -> 3072 at 8192 tokens none stored 19 / 70,
// 0.1 % 39 / 72, 0.5 % 93 / 73; 4096 -> 1024 at 8192 tokens 0.1 % 50 / 113, 0.5 % 148 / 119.
int g_csr_rows = -1;  // test hook: -1 = automatic, 0 = never, 1 = always
bool csr_rows_pay(ExpandArgs a, int nnz) {
    if (g_csr_rows >= 0) return g_csr_rows != 0;
    const ExpandPlan p = plan_expand<FMT_CSRM>(a);
    const double sms = sm_count() > 0 ? sm_count() : 148;
    const double buffers = ((a.in + BK - 1) / BK + a.ckb - 1) / a.ckb;  // each waits for the one before it
    const double expand =
        0.3 + p.cycles / 1650.0 + p.waves * (1.9 * (buffers - 1) + 0.0012 * buffers * nnz / p.panels);
    const double ctas = a.T / 8.0 / sms;  // per SM
    const double rows = 2.1 + 0.0025 * a.out + 0.0022 * (nnz < a.out ? nnz : a.out) +
                        2.0 * a.T * a.in / 5e6 + 0.0007 * (ctas > 1.2 ? ctas : 1.2) * nnz;
    return rows < expand;
}

template <int FMT>
int launch_expand(ExpandArgs a, cudaStream_t stream) {
    CUtensorMap tmX;
    int st = encode_operand(&tmX, a.X, a.in, a.T, a.in, BM);
    if (st != ET_OK) return st;
    a.err_word = device_error_word();
    if (!a.err_word) return ET_ERR_NO_DEVICE;
    a.vec_store = (a.out % 8 == 0 && aligned16(a.Y)) ? 1 : 0;
    const int bn = plan_expand<FMT>(a).bn;
    int cols = 32;
    while (cols < a.mb * bn) cols <<= 1;
    a.tmem_cols = cols;
    if (bn == 32) return launch_bn<FMT, 32>(tmX, a, stream);
    if (bn == 64) return launch_bn<FMT, 64>(tmX, a, stream);
    return launch_bn<FMT, FMT == FMT_CSRM ? 64 : 128>(tmX, a, stream);
}

}  // namespace

int launch_linear_expand_packed(const uint32_t* pk_mask, const int* pk_off, const __half* pk_tiles,
                                const __half* bias, const __half* X, __half* Y, int T, int in, int out,
                                int act, cudaStream_t stream) {
    ExpandArgs a = {};
    a.idx0 = reinterpret_cast<const int*>(pk_mask);
    a.idx1 = pk_off;
    a.data = pk_tiles;
    a.bias = bias;
    a.X = X;
    a.Y = Y;
    a.T = T;
    a.in = in;
    a.out = out;
    a.act = act;
    return launch_expand<FMT_PACKED>(a, stream);
}

}  // namespace et

extern "C" {

int et_linear_1x16_fwd(const int32_t* tile_idx, const int32_t* row_idx, const et_half* data,
                       int nvec, const et_half* bias, const et_half* X, et_half* Y, int T, int in,
                       int out, int act, et_stream stream) {
    if (!tile_idx || !X || !Y || T <= 0 || in <= 0 || out <= 0 || nvec < 0)
        return ET_ERR_INVALID_ARG;
    if (nvec > 0 && (!row_idx || !data)) return ET_ERR_INVALID_ARG;
    if (act < ET_ACT_NONE || act > ET_ACT_GELU) return ET_ERR_INVALID_ARG;
    if (in % 16 || out % 16 || T > 65535 * 128) return ET_ERR_SHAPE;
    if (!et::aligned16(X) || !et::aligned16(Y) || (data && !et::aligned16(data)))
        return ET_ERR_ALIGNMENT;
    et::ExpandArgs a = {};
    a.idx0 = tile_idx;
    a.idx1 = row_idx;
    a.data = reinterpret_cast<const __half*>(data);
    a.bias = reinterpret_cast<const __half*>(bias);
    a.X = reinterpret_cast<const __half*>(X);
    a.Y = reinterpret_cast<__half*>(Y);
    a.T = T;
    a.in = in;
    a.out = out;
    a.act = act;
    return et::launch_expand<et::FMT_VEC>(a, static_cast<cudaStream_t>(stream));
}

int et_linear_csr_fwd(const int32_t* indptr, const int32_t* indices, const et_half* data,
                      int nnz, const et_half* bias, const et_half* X, et_half* Y, int T, int in,
                      int out, int act, et_stream stream) {
    if (!indptr || !X || !Y || T <= 0 || in <= 0 || out <= 0 || nnz < 0) return ET_ERR_INVALID_ARG;
    if (nnz > 0 && (!indices || !data)) return ET_ERR_INVALID_ARG;
    if (act < ET_ACT_NONE || act > ET_ACT_GELU) return ET_ERR_INVALID_ARG;
    if (in % 8 || in > 8192) return ET_ERR_SHAPE;
    if (!et::aligned16(X)) return ET_ERR_ALIGNMENT;
    et::ExpandArgs a = {};
    a.idx0 = indptr;
    a.idx1 = indices;
    a.data = reinterpret_cast<const __half*>(data);
    a.bias = reinterpret_cast<const __half*>(bias);
    a.X = reinterpret_cast<const __half*>(X);
    a.Y = reinterpret_cast<__half*>(Y);
    a.T = T;
    a.in = in;
    a.out = out;
    a.act = act;
    if (et::csr_rows_pay(a, nnz))
        return et::launch_linear_csr_rows(a.idx0, a.idx1, a.data, a.bias, a.X, a.Y, T, in, out, act,
                                          static_cast<cudaStream_t>(stream));
    return et::launch_expand<et::FMT_CSRM>(a, static_cast<cudaStream_t>(stream));
}

#ifdef ET_TEST_HOOKS
// Test hook: the CSR product by stored values: -1 = automatic, 0 = never, 1 = always.
void et_debug_set_csr_rows(int mode) { et::g_csr_rows = mode; }
// Test hook: 1 when that product is chosen for the size.
int et_debug_csr_rows_pay(int T, int in, int out, int nnz) {
    et::ExpandArgs a = {};
    a.T = T;
    a.in = in;
    a.out = out;
    return et::csr_rows_pay(a, nnz) ? 1 : 0;
}
#endif  // ET_TEST_HOOKS

}  // extern "C"
