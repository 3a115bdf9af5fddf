// Elementwise / layout kernels of the MoE training step that sit between the grouped GEMMs:
//
//   transpose_bf16     batched [B, R, C] -> [B, C, R] through 64x64 shared-memory tiles (16-byte global accesses both ways);
//                      the weight-gradient GEMM reduces over tokens and wants them contiguous, the input-gradient GEMM wants
//                      the weights with their output dimension contiguous
//   swiglu_fwd / bwd   h = silu(gate) * up from h13 = [gate | up], and its gradient, in one pass each (fp32 math, bf16 I/O)
//   unpermute_bwd      both gradients of the weighted un-permute in one pass over its input
//   rowdot             d_w[n, k] = <a[pos[n, k]], b[n]>  (gradient of the gate weights through the weighted un-permute)
//
// The reference has no counterpart (it ships no model code); these replace chains of framework ops whose copies
// dominated the training step.
#include "gemm_api.h"
#include "launch.cuh"
#include "sigmoid.cuh"

#include <cuda_bf16.h>

namespace dx {

namespace {

constexpr int kTile = 64;

__global__ void __launch_bounds__(256) transpose_bf16_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out, int R, int C) {
    // 64x64 tile without padding; the 16-byte chunk `ch` of row r lives at chunk position ch ^ ((r >> 3) & 7). Rows that are a
    // multiple of 8 apart (what the lanes of the store phase read together) then sit in different banks, and the 8 lanes
    // that fill one row in the load phase still cover it exactly once.
    __shared__ __align__(16) __nv_bfloat16 tile[kTile][kTile];
    const size_t plane = (size_t)R * C;
    const __nv_bfloat16* src = in + blockIdx.z * plane;
    __nv_bfloat16* dst = out + blockIdx.z * plane;
    const int r0 = blockIdx.y * kTile, c0 = blockIdx.x * kTile;
    const int tid = threadIdx.x;
    for (int i = tid; i < kTile * 8; i += 256) {
        const int r = i >> 3, ch = i & 7;
        int4 v = make_int4(0, 0, 0, 0);
        if (r0 + r < R && c0 + ch * 8 < C) v = *reinterpret_cast<const int4*>(src + (size_t)(r0 + r) * C + c0 + ch * 8);
        *reinterpret_cast<int4*>(&tile[r][(ch ^ ((r >> 3) & 7)) * 8]) = v;
    }
    __syncthreads();
    // store: output row = input column c; lane (i & 7) = q assembles input rows 8q..8q+7 into one 16-byte chunk, so 8
    // consecutive lanes write one full 128-byte output row segment
    for (int i = tid; i < kTile * 8; i += 256) {
        const int c = i >> 3, q = i & 7;
        if (c0 + c >= C || r0 + q * 8 >= R) continue;
        const int col = (((c >> 3) ^ q) << 3) + (c & 7);  // (r >> 3) & 7 == q for the rows 8q..8q+7
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = tile[q * 8 + j][col];
        *reinterpret_cast<int4*>(dst + (size_t)(c0 + c) * R + r0 + q * 8) = *reinterpret_cast<const int4*>(v);
    }
}

// One thread per eight columns; `I` is a 32-bit index wherever the sizes allow (a 64-bit division per thread costs more than the
// arithmetic of the eight elements).
template <typename I>
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ h13, __nv_bfloat16* __restrict__ h, I work, int inter) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const I i = (I)blockIdx.x * 256 + threadIdx.x;
    if (i >= work) return;
    const I chunks = inter / 8;
    const I r = i / chunks;
    const int c = (int)(i - r * chunks) * 8;
    const __nv_bfloat16* row = h13 + (size_t)r * 2 * inter + c;
    const int4 g = *reinterpret_cast<const int4*>(row);
    const int4 u = *reinterpret_cast<const int4*>(row + inter);
    const __nv_bfloat16* gp = reinterpret_cast<const __nv_bfloat16*>(&g);
    const __nv_bfloat16* up = reinterpret_cast<const __nv_bfloat16*>(&u);
    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = __float2bfloat16(silu(__bfloat162float(gp[j])) * __bfloat162float(up[j]));
    *reinterpret_cast<int4*>(h + (size_t)r * inter + c) = *reinterpret_cast<const int4*>(o);
}

template <typename I>
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ h13, const __nv_bfloat16* __restrict__ dh,
                                                         __nv_bfloat16* __restrict__ dh13, I work, int inter) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const I i = (I)blockIdx.x * 256 + threadIdx.x;
    if (i >= work) return;
    const I chunks = inter / 8;
    const I r = i / chunks;
    const int c = (int)(i - r * chunks) * 8;
    const __nv_bfloat16* row = h13 + (size_t)r * 2 * inter + c;
    const int4 g = *reinterpret_cast<const int4*>(row);
    const int4 u = *reinterpret_cast<const int4*>(row + inter);
    const int4 d = *reinterpret_cast<const int4*>(dh + (size_t)r * inter + c);
    const __nv_bfloat16* gp = reinterpret_cast<const __nv_bfloat16*>(&g);
    const __nv_bfloat16* up = reinterpret_cast<const __nv_bfloat16*>(&u);
    const __nv_bfloat16* dp = reinterpret_cast<const __nv_bfloat16*>(&d);
    __align__(16) __nv_bfloat16 og[8], ou[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float x = __bfloat162float(gp[j]), uu = __bfloat162float(up[j]), dd = __bfloat162float(dp[j]);
        const float sig = sigmoid(x);
        og[j] = __float2bfloat16(dd * uu * sig * (1.f + x * (1.f - sig)));  // d silu(x)/dx = sig * (1 + x * (1 - sig))
        ou[j] = __float2bfloat16(dd * x * sig);
    }
    __nv_bfloat16* orow = dh13 + (size_t)r * 2 * inter + c;
    *reinterpret_cast<int4*>(orow) = *reinterpret_cast<const int4*>(og);
    *reinterpret_cast<int4*>(orow + inter) = *reinterpret_cast<const int4*>(ou);
}

// one warp per (n, k)
__global__ void __launch_bounds__(256) rowdot_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b, const int* __restrict__ pos,
                                                     float* __restrict__ out, int n_rows, int num_k, int hidden) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const int lane = threadIdx.x & 31;
    const long long total = (long long)n_rows * num_k;
    for (long long p = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); p < total; p += (long long)gridDim.x * 8) {
        const int src = pos[p];
        float acc = 0.f;
        if (src >= 0) {
            const int4* ar = reinterpret_cast<const int4*>(a + (size_t)src * hidden);
            const int4* br = reinterpret_cast<const int4*>(b + (size_t)(p / num_k) * hidden);
            const int n16 = hidden / 8;
            constexpr int U = 8;  // eight column chunks of both rows in flight per lane
            for (int i0 = 0; i0 < n16; i0 += 32 * U) {
                int4 x[U], y[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u * 32 + lane;
                    x[u] = i < n16 ? ar[i] : make_int4(0, 0, 0, 0);
                    y[u] = i < n16 ? br[i] : make_int4(0, 0, 0, 0);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&x[u]);
                    const __nv_bfloat162* yp = reinterpret_cast<const __nv_bfloat162*>(&y[u]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 xf = __bfloat1622float2(xp[j]), yf = __bfloat1622float2(yp[j]);
                        acc = fmaf(xf.x, yf.x, fmaf(xf.y, yf.y, acc));
                    }
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) out[p] = acc;
    }
}

// Both gradients of the weighted un-permute. One warp per (n, k): row a[pos] and row g[n] are read once and w * g[n] is written, where a
// row product and a gather of their own read g twice and could not hide the gather's writes (87 % of its traffic) behind reads. The
// num_k warps of a token are neighbours, so g[n] comes from L1 or L2 for all but the first. Further warps clear the padding rows.
__global__ void __launch_bounds__(256) unpermute_bwd_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ g,
                                                            const float* __restrict__ w, const int* __restrict__ pos,
                                                            const int* __restrict__ src_row, __nv_bfloat16* __restrict__ da, float* __restrict__ dw,
                                                            long long pairs, long long items, int num_k, int hidden) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const int lane = threadIdx.x & 31, n16 = hidden / 8;
    const long long p = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (p >= items) return;
    if (p >= pairs) {
        const long long m = p - pairs;
        if (src_row[m] >= 0) return;
        int4* row = reinterpret_cast<int4*>(da + (size_t)m * hidden);
        for (int i = lane; i < n16; i += 32) row[i] = make_int4(0, 0, 0, 0);
        return;
    }
    const int src = pos[p];
    float acc = 0.f;
    if (src >= 0) {
        const float sc = w[p];
        const int4* ar = reinterpret_cast<const int4*>(a + (size_t)src * hidden);
        const int4* gr = reinterpret_cast<const int4*>(g + (size_t)(p / num_k) * hidden);
        int4* dr = reinterpret_cast<int4*>(da + (size_t)src * hidden);
        constexpr int U = 4;  // column chunks of both rows in flight per lane
        for (int i0 = 0; i0 < n16; i0 += 32 * U) {
            int4 x[U], y[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * 32 + lane;
                x[u] = i < n16 ? ld_once(ar + i) : make_int4(0, 0, 0, 0);
                y[u] = i < n16 ? gr[i] : make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * 32 + lane;
                const uint32_t xw[4] = {(uint32_t)x[u].x, (uint32_t)x[u].y, (uint32_t)x[u].z, (uint32_t)x[u].w};
                uint32_t yw[4] = {(uint32_t)y[u].x, (uint32_t)y[u].y, (uint32_t)y[u].z, (uint32_t)y[u].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 xf = bf16x2_to_f2(xw[j]), yf = bf16x2_to_f2(yw[j]);
                    acc = fmaf(xf.x, yf.x, fmaf(xf.y, yf.y, acc));
                    yw[j] = f2_to_bf16x2(yf.x * sc, yf.y * sc);
                }
                if (i < n16) st_once(dr + i, make_int4((int)yw[0], (int)yw[1], (int)yw[2], (int)yw[3]));
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) dw[p] = acc;
}

}  // namespace

cudaError_t launch_unpermute_bwd(const void* a, const void* g, const float* w, const int* pos, const int* src_row, void* da, float* dw, int n_rows,
                                 int num_k, int m_rows, int hidden, cudaStream_t stream) {
    const long long pairs = (long long)n_rows * num_k, items = pairs + m_rows;
    if (items <= 0) return cudaSuccess;
    if ((hidden & 7) != 0) return cudaErrorInvalidValue;
    return launch_dependent(unpermute_bwd_kernel, dim3((unsigned)((items + 7) / 8)), 256, 0, stream, static_cast<const __nv_bfloat16*>(a),
                            static_cast<const __nv_bfloat16*>(g), w, pos, src_row, static_cast<__nv_bfloat16*>(da), dw, pairs, items, num_k, hidden);
}

cudaError_t launch_transpose_bf16(const void* in, void* out, int batch, int rows, int cols, cudaStream_t stream) {
    if (batch <= 0 || rows <= 0 || cols <= 0) return cudaSuccess;
    if ((rows & 7) != 0 || (cols & 7) != 0 || batch > 65535) return cudaErrorInvalidValue;
    dim3 grid((cols + kTile - 1) / kTile, (rows + kTile - 1) / kTile, batch);
    if (grid.y > 65535) return cudaErrorInvalidValue;
    transpose_bf16_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(in), static_cast<__nv_bfloat16*>(out), rows, cols);
    return cudaGetLastError();
}

cudaError_t launch_swiglu_fwd(const void* h13, void* h, long long rows, int inter, cudaStream_t stream) {
    if (rows <= 0) return cudaSuccess;
    if ((inter & 7) != 0) return cudaErrorInvalidValue;
    const long long work = rows * (inter / 8);
    const dim3 grid((unsigned)((work + 255) / 256));
    const auto* in = static_cast<const __nv_bfloat16*>(h13);
    auto* out = static_cast<__nv_bfloat16*>(h);
    if (work < (1ll << 31)) return launch_dependent(swiglu_fwd_kernel<unsigned>, grid, 256, 0, stream, in, out, (unsigned)work, inter);
    return launch_dependent(swiglu_fwd_kernel<long long>, grid, 256, 0, stream, in, out, work, inter);
}

// What the epilogues compute in fp32, beside the same with a division: [4, n] = silu, silu by division, sigmoid, sigmoid by division (for the tests).
__global__ void __launch_bounds__(256) logistic_kernel(const float* __restrict__ x, float* __restrict__ out, long long n) {
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const float v = x[i], d = 1.f + __expf(-v);
        out[i] = silu(v);
        out[n + i] = v / d;
        out[2 * n + i] = sigmoid(v);
        out[3 * n + i] = 1.f / d;
    }
}

cudaError_t launch_logistic(const float* x, float* out, long long n, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    logistic_kernel<<<148, 256, 0, stream>>>(x, out, n);
    return cudaGetLastError();
}

cudaError_t launch_swiglu_bwd(const void* h13, const void* dh, void* dh13, long long rows, int inter, cudaStream_t stream) {
    if (rows <= 0) return cudaSuccess;
    if ((inter & 7) != 0) return cudaErrorInvalidValue;
    const long long work = rows * (inter / 8);
    const dim3 grid((unsigned)((work + 255) / 256));
    const auto *in = static_cast<const __nv_bfloat16*>(h13), *din = static_cast<const __nv_bfloat16*>(dh);
    auto* out = static_cast<__nv_bfloat16*>(dh13);
    if (work < (1ll << 31)) return launch_dependent(swiglu_bwd_kernel<unsigned>, grid, 256, 0, stream, in, din, out, (unsigned)work, inter);
    return launch_dependent(swiglu_bwd_kernel<long long>, grid, 256, 0, stream, in, din, out, work, inter);
}

cudaError_t launch_rowdot(const void* a, const void* b, const int* pos, float* out, int n_rows, int num_k, int hidden, cudaStream_t stream) {
    const long long total = (long long)n_rows * num_k;
    if (total <= 0) return cudaSuccess;
    if ((hidden & 7) != 0) return cudaErrorInvalidValue;
    return launch_dependent(rowdot_kernel, dim3((unsigned)((total + 7) / 8)), 256, 0, stream, static_cast<const __nv_bfloat16*>(a),
                            static_cast<const __nv_bfloat16*>(b), pos, out, n_rows, num_k, hidden);
}

}  // namespace dx
