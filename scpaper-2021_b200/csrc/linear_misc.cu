// Irregular weight formats off the tensor cores: the CSR product for weights that are almost empty, and the
// plan-time helpers of the 1x16 format (the other forward passes are in linear_expand.cu).
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace et {
namespace {

// CSR product on the CUDA cores: a CTA keeps 8 token rows in shared memory, its threads sweep the output
// features and gather activations by column.  Work follows the stored values, so it wins where hardly any are
// stored; linear_expand.cu has the rule.  What bounds it: one dependent chain of index, value and shared
// memory reads per output feature (8192 tokens, 1024 -> 3072, 0.1 % stored: 39 us; 1 % stored: 163 us).
constexpr int CSR_TOKENS = 8;
constexpr int CSR_THREADS = 256;
constexpr int CSR_MAX_IN = 8192;

__global__ void __launch_bounds__(CSR_THREADS)
linear_csr_rows_kernel(const int* __restrict__ indptr, const int* __restrict__ indices,
                       const __half* __restrict__ data, const __half* __restrict__ bias,
                       const __half* __restrict__ X, __half* __restrict__ Y, int T, int in, int out,
                       int act) {
    extern __shared__ __half xs[];  // [CSR_TOKENS][in]
    const int t0 = blockIdx.x * CSR_TOKENS;
    const int nt = (T - t0) < CSR_TOKENS ? (T - t0) : CSR_TOKENS;
    const int chunks = in >> 3;
    for (int i = threadIdx.x; i < CSR_TOKENS * chunks; i += CSR_THREADS) {
        const int tt = i / chunks, c = i - tt * chunks;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (tt < nt) v = __ldcg(reinterpret_cast<const uint4*>(X + static_cast<size_t>(t0 + tt) * in) + c);
        reinterpret_cast<uint4*>(xs + static_cast<size_t>(tt) * in)[c] = v;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < out; o += CSR_THREADS) {
        float acc[CSR_TOKENS];
#pragma unroll
        for (int tt = 0; tt < CSR_TOKENS; ++tt) acc[tt] = 0.f;
        const int beg = __ldg(indptr + o), end = __ldg(indptr + o + 1);
        for (int i = beg; i < end; ++i) {
            const float w = __half2float(__ldg(data + i));
            const int c = __ldg(indices + i);
            if (c < 0 || c >= in) continue;
#pragma unroll
            for (int tt = 0; tt < CSR_TOKENS; ++tt)
                acc[tt] += w * __half2float(xs[static_cast<size_t>(tt) * in + c]);
        }
        const float b = bias ? __half2float(__ldg(bias + o)) : 0.f;
#pragma unroll
        for (int tt = 0; tt < CSR_TOKENS; ++tt)
            if (tt < nt)
                Y[static_cast<size_t>(t0 + tt) * out + o] = __float2half_rn(apply_act(acc[tt] + b, act));
    }
}

// One CTA per 16-row set: dense[set * 16 + q][part * 16 .. + 16] = data[i] for every stored
// vector i of the set (q = row_idx[i] % 16); thread = (vector slot in a group of 16, element).
__global__ void densify_1x16_kernel(const int* __restrict__ tile_idx, const int* __restrict__ row_idx,
                                    const __half* __restrict__ data, int npart, int in,
                                    __half* __restrict__ dense) {
    const int rset = blockIdx.x;
    const int* tidx = tile_idx + static_cast<size_t>(rset) * (npart + 1);
    const int beg0 = __ldg(tidx), end0 = __ldg(tidx + npart);
    const int j = threadIdx.x & 15;
    for (int i = beg0 + (threadIdx.x >> 4); i < end0; i += blockDim.x >> 4) {
        // the part of vector i: the last p with tile_idx[p] <= i (binary search)
        int lo = 0, hi = npart - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(tidx + mid) <= i) lo = mid; else hi = mid - 1;
        }
        const int q = __ldg(row_idx + i) & 15;
        dense[(static_cast<size_t>(rset) * 16 + q) * in + lo * 16 + j] = data[static_cast<size_t>(i) * 16 + j];
    }
}

}  // namespace

int launch_linear_csr_rows(const int* indptr, const int* indices, const __half* data, const __half* bias,
                           const __half* X, __half* Y, int T, int in, int out, int act, cudaStream_t stream) {
    static std::atomic<bool> attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (cudaFuncSetAttribute(linear_csr_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 CSR_TOKENS * CSR_MAX_IN * 2) != cudaSuccess)
            return ET_ERR_CUDA;
        attr_set[dev] = true;
    }
    count_launch();
    linear_csr_rows_kernel<<<(T + CSR_TOKENS - 1) / CSR_TOKENS, CSR_THREADS, CSR_TOKENS * in * 2, stream>>>(
        indptr, indices, data, bias, X, Y, T, in, out, act);
    return cudaGetLastError() == cudaSuccess ? ET_OK : ET_ERR_CUDA;
}

}  // namespace et

extern "C" {

int et_1x16_prefer_dense(int in, int out, int nvec) {
    if (in <= 0 || out <= 0 || (in & 15) || (out & 15)) return 0;
    // et_linear_1x16_fwd expands the vectors into dense operand tiles and pays for the dense product on
    // top of that (1024 -> 3072 at 3072 tokens 17.4 us against 16.5, 3072 -> 768 at 1024 tokens 13.9 against
    // 10.8): the expanded weight in memory is only worth its space where something is stored
    const double total = static_cast<double>(out) * (in >> 4);
    return nvec > 0.01 * total ? 1 : 0;
}

int et_1x16_densify(const int32_t* tile_idx, const int32_t* row_idx, const et_half* data, int nvec,
                    int in, int out, et_half* dense, et_stream stream) {
    if (!tile_idx || !dense || in <= 0 || out <= 0 || nvec < 0) return ET_ERR_INVALID_ARG;
    if ((in & 15) || (out & 15)) return ET_ERR_SHAPE;
    if (nvec > 0 && (!row_idx || !data)) return ET_ERR_INVALID_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(dense, 0, static_cast<size_t>(in) * out * sizeof(__half), s) != cudaSuccess)
        return ET_ERR_CUDA;
    if (nvec > 0) {
        et::count_launch();
        et::densify_1x16_kernel<<<out >> 4, 256, 0, s>>>(tile_idx, row_idx,
                                                          reinterpret_cast<const __half*>(data),
                                                          in >> 4, in, reinterpret_cast<__half*>(dense));
        if (cudaGetLastError() != cudaSuccess) return ET_ERR_CUDA;
    }
    return ET_OK;
}

}  // extern "C"
