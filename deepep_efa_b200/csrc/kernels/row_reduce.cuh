// dst[n] = sum_k w[n,k] * src[row[n,k]] over BF16 rows with fp32 accumulation in rising k, shared by the home-side reduction of the
// fused layer and the weighted un-permutation.
//
// A warp takes a span of 64 sixteen-byte columns of one output row and has the loads of eight source rows x two columns in flight
// before it consumes the first. Short warps instead of one warp per row keep all SMs loading: 4096 x 8 rows of 14 KB took 138 us
// with a warp per row; 777 x 6 rows of 8 KB took 43 us when the rows were fetched one after the other.
#pragma once

#include "prims.cuh"

namespace dx {

constexpr int kReduceThreads = 256;
constexpr int kReduceSpan = 64;  // 16-byte columns per warp

__host__ __device__ __forceinline__ int reduce_spans(int n16) { return (n16 + kReduceSpan - 1) / kReduceSpan; }
inline int reduce_ctas(int rows, int n16) {
    const long long warps = (long long)rows * reduce_spans(n16);
    return (int)((warps + kReduceThreads / 32 - 1) / (kReduceThreads / 32));
}

// `my_row` / `my_w`: lane k holds source row and weight of selection k, row -1 = skip.
__device__ __forceinline__ void reduce_row_span(const int4* __restrict__ src, int4* __restrict__ dst, int n16, int span, int num_k, int my_row,
                                                float my_w, int lane) {
    constexpr int U = kReduceSpan / 32;
    const int i0 = span * kReduceSpan + lane;
    float acc[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[u][q] = 0.f;
    for (int k0 = 0; k0 < num_k; k0 += 8) {
        int4 v[8][U];
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const int row = __shfl_sync(0xffffffffu, my_row, (k0 + kk) & 31);
            const bool ok = k0 + kk < num_k && row >= 0;
#pragma unroll
            for (int u = 0; u < U; ++u) v[kk][u] = (ok && i0 + u * 32 < n16) ? ld_once(src + (size_t)row * n16 + i0 + u * 32) : make_int4(0, 0, 0, 0);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const float wk = __shfl_sync(0xffffffffu, my_w, (k0 + kk) & 31);
            const bool ok = k0 + kk < num_k && __shfl_sync(0xffffffffu, my_row, (k0 + kk) & 31) >= 0;
            if (!ok) continue;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t w4[4] = {(uint32_t)v[kk][u].x, (uint32_t)v[kk][u].y, (uint32_t)v[kk][u].z, (uint32_t)v[kk][u].w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 f = bf16x2_to_f2(w4[q]);
                    acc[u][2 * q] = fmaf(wk, f.x, acc[u][2 * q]);
                    acc[u][2 * q + 1] = fmaf(wk, f.y, acc[u][2 * q + 1]);
                }
            }
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (i0 + u * 32 >= n16) continue;
        int4 o;
        o.x = (int)f2_to_bf16x2(acc[u][0], acc[u][1]);
        o.y = (int)f2_to_bf16x2(acc[u][2], acc[u][3]);
        o.z = (int)f2_to_bf16x2(acc[u][4], acc[u][5]);
        o.w = (int)f2_to_bf16x2(acc[u][6], acc[u][7]);
        dst[i0 + u * 32] = o;
    }
}

}  // namespace dx
