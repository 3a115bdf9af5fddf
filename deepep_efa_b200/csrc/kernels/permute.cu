// Row gather kernels that move dispatch results into the expert-major, 128-row-aligned layout the grouped
// GEMM wants, and back (weighted) into receive order for combine.
//
//   build_plan:           the maps between the two orders, in one launch
//   gather_rows:          dst[m] = scale[m] * src[src_row[m]]            (src_row < 0 -> zero row)
//   permute_rows:         the unweighted gather of a plan, by whichever of its maps is the faster
//   gather_reduce_rows:   dst[n] = sum_k w[n,k] * src[pos[n,k]]          (pos < 0 skipped), fp32 accumulate
//
// The gathers are pure bandwidth kernels: a warp per span of columns of an output row, 16-byte accesses, no atomics. The
// unweighted ones are each other's backward pass; that of the weighted sum is unpermute_bwd in train_ops.cu, which reads each
// row once for both of its gradients.
//
// The reference has no counterpart: its users permute with framework indexing ops between dispatch and
// their expert GEMMs.
#include <cuda_bf16.h>

#include <algorithm>

#include "gemm_api.h"
#include "launch.cuh"
#include "prims.cuh"
#include "row_reduce.cuh"
#include "select_scan.cuh"

namespace dx {

constexpr int kPermThreads = 256;

// Generic byte rows (any dtype); optional fp32 scale is only legal for bf16 payloads.
// A warp copies a span of up to 256 sixteen-byte columns with all of its loads in flight (eight per lane). A source row is read once per selection: the stores
// leave the L2 to the sources (8192 tokens x 6, rows of 8 KB: 124 -> 98 us; 2000 x 8 of 14 KB 69 -> 42; 4096 x 8 of 4 KB 42 -> 26; where all fits the L2 no change).
constexpr int kGatherSpan = 256;

__global__ void __launch_bounds__(kPermThreads) gather_rows_kernel(const char* __restrict__ src, char* __restrict__ dst,
                                                                  const int* __restrict__ src_row, const float* __restrict__ scale,
                                                                  int num_dst_rows, int row_bytes) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const int lane = threadIdx.x & 31;
    const int n16 = row_bytes / 16, spans = (n16 + kGatherSpan - 1) / kGatherSpan;
    const int item = blockIdx.x * (kPermThreads / 32) + (threadIdx.x >> 5);
    const int m = item / spans;
    if (m >= num_dst_rows) return;
    const int s = src_row[m];
    const int i0 = (item % spans) * kGatherSpan + lane;
    int4* d = reinterpret_cast<int4*>(dst + (size_t)m * row_bytes);
    constexpr int U = kGatherSpan / 32;
    int4 v[U];
    const int4* p = reinterpret_cast<const int4*>(src + (size_t)max(s, 0) * row_bytes);
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = (s >= 0 && i0 + u * 32 < n16) ? __ldg(p + i0 + u * 32) : make_int4(0, 0, 0, 0);
    if (scale != nullptr && s >= 0) {
        const float sc = scale[m];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            uint32_t w[4] = {(uint32_t)v[u].x, (uint32_t)v[u].y, (uint32_t)v[u].z, (uint32_t)v[u].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = bf16x2_to_f2(w[j]);
                w[j] = f2_to_bf16x2(f.x * sc, f.y * sc);
            }
            v[u] = make_int4((int)w[0], (int)w[1], (int)w[2], (int)w[3]);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (i0 + u * 32 < n16) st_once(d + i0 + u * 32, v[u]);
}

// As many CTAs as are resident, each warp walking over spans: a warp per span spent a third of its life on the positions, and a
// CTA's place stayed empty until its last warp was done (8192 x 6 rows of 8 KB: 87 -> 77 us, 93 % of the measured copy bandwidth).
constexpr int kGatherReduceCtasPerSm = 2;

__global__ void __launch_bounds__(kReduceThreads, kGatherReduceCtasPerSm) gather_reduce_rows_kernel(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ dst,
                                                                           const int* __restrict__ pos, const float* __restrict__ w,
                                                                           int num_dst_rows, int num_k, int hidden) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const int lane = threadIdx.x & 31;
    const int n16 = hidden / 8, spans = reduce_spans(n16);
    const long long items = (long long)num_dst_rows * spans, step = (long long)gridDim.x * (kReduceThreads / 32);
    long long item = (long long)blockIdx.x * (kReduceThreads / 32) + (threadIdx.x >> 5);
    // positions and weights of the next span are on their way while this one is summed
    int my_pos = -1;
    float my_w = 0.f;
    auto fetch = [&](long long it) {
        if (it < items && lane < num_k) {
            const size_t i = (size_t)(it / spans) * num_k + lane;
            my_pos = pos[i];
            my_w = w != nullptr ? w[i] : 1.f;
        }
    };
    fetch(item);
    for (; item < items; item += step) {
        const int n = (int)(item / spans);
        // selections that are set, compacted onto the low lanes in their order: a row of a rank with peers has one or two of them
        const unsigned valid = __ballot_sync(0xffffffffu, my_pos >= 0);
        const int nv = __popc(valid);
        const int from = lane < nv ? (int)__fns(valid, 0, lane + 1) : 0;
        const int pos_c = __shfl_sync(0xffffffffu, my_pos, from);
        const float w_c = __shfl_sync(0xffffffffu, my_w, from);
        fetch(item + step);
        reduce_row_span(reinterpret_cast<const int4*>(src), reinterpret_cast<int4*>(dst) + (size_t)n * n16, n16, (int)(item % spans), nv, lane < nv ? pos_c : -1, w_c, lane);
    }
}

// Expert-major slot assignment: the selections of local expert e get the rows m_offsets[e], m_offsets[e] + 1, ... in token order;
// the rest of the expert's 128-aligned segment is padding (src_row -1). One launch: the group offsets arrive in the arguments, a
// CTA lists the selections of its experts (select_scan.cuh) and pads their segments, and CTA 0 marks the unselected ones. More experts
// than the arguments hold take a launch per kPlanMaxExperts of them.
struct PlanOffsets {
    int v[kPlanMaxExperts + 1];
};

__global__ void __launch_bounds__(kScanThreads, 1) build_plan_kernel(const int64_t* __restrict__ topk_idx, const __grid_constant__ PlanOffsets offs,
                                                                     int* __restrict__ m_offsets, int* __restrict__ m_ends, int* __restrict__ pos, int* __restrict__ src_row,
                                                                     int* __restrict__ src_k, int num_pairs, int num_topk, int num_local_experts,
                                                                     int first, int count, int per_cta) {
    pdl_wait_predecessor();
    pdl_release_successor();
    extern __shared__ int s_dyn[];
    int* s_run = s_dyn;
    uint32_t* s_vote = reinterpret_cast<uint32_t*>(s_dyn + kScanBatch);
    const int tid = threadIdx.x;
    if (blockIdx.x == 0)
        for (int e = tid; e <= count; e += kScanThreads) m_offsets[first + e] = offs.v[e];
    const int e0 = blockIdx.x * per_cta, ne = max(0, min(per_cta, count - e0));  // of the launch's experts [first, first + count)
    for (int b0 = 0; b0 < ne; b0 += kScanBatch) {
        const int nb = min(kScanBatch, ne - b0);
        scan_selections(topk_idx, num_pairs, num_local_experts, first + e0 + b0, nb, s_vote, s_run, first == 0 && blockIdx.x == 0 && b0 == 0,
                        [&](int j, int n, int i) {
                            const int row = offs.v[e0 + b0 + j] + n;
                            const bool fits = row < offs.v[e0 + b0 + j + 1];  // always, when the offsets come from the dispatch counts
                            if (fits) {
                                src_row[row] = i / num_topk;
                                src_k[row] = i % num_topk;
                            }
                            pos[i] = fits ? row : -1;
                        },
                        [&](int i) { pos[i] = -1; });
        for (int j = 0; j < nb; ++j) {
            const int end = offs.v[e0 + b0 + j + 1];
            if (tid == 0) m_ends[first + e0 + b0 + j] = min(offs.v[e0 + b0 + j] + s_run[j], end);
            for (int row = offs.v[e0 + b0 + j] + s_run[j] + tid; row < end; row += kScanThreads) {
                src_row[row] = -1;
                src_k[row] = 0;
            }
        }
        __syncthreads();
    }
}

cudaError_t launch_build_plan(const int64_t* topk_idx, const int* host_offsets, int* m_offsets, int* m_ends, int* pos, int* src_row, int* src_k,
                              int num_rows, int num_topk, int num_local_experts, cudaStream_t stream) {
    if (num_local_experts < 1) return cudaErrorInvalidValue;
    for (int first = 0; first < num_local_experts; first += kPlanMaxExperts) {
        const int count = std::min(num_local_experts - first, kPlanMaxExperts);
        PlanOffsets offs;
        for (int e = 0; e <= count; ++e) offs.v[e] = host_offsets[first + e];
        const int per_cta = (count + 147) / 148;
        const size_t smem = scan_smem_bytes(per_cta);
        cudaError_t e = cudaSuccess;
        if (smem > 48 * 1024) e = cudaFuncSetAttribute(build_plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = launch_dependent(build_plan_kernel, dim3((count + per_cta - 1) / per_cta), kScanThreads, smem, stream, topk_idx, offs, m_offsets, m_ends, pos, src_row,
                                 src_k, num_rows * num_topk, num_topk, num_local_experts, first, count, per_cta);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Rows that are no multiple of 16 bytes (scale rows of some hidden sizes), word by word.
__global__ void __launch_bounds__(kPermThreads) gather_words_kernel(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, const int* __restrict__ src_row,
                                                                   int num_dst_rows, int row_words) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const int m = blockIdx.x * (kPermThreads / 32) + (threadIdx.x >> 5);
    if (m >= num_dst_rows) return;
    const int s = src_row[m];
    for (int i = threadIdx.x & 31; i < row_words; i += 32) dst[(size_t)m * row_words + i] = s >= 0 ? src[(size_t)s * row_words + i] : 0u;
}

cudaError_t launch_gather_rows(const void* src, void* dst, const int* src_row, const float* scale, int num_dst_rows, int row_bytes,
                               cudaStream_t stream) {
    if (num_dst_rows <= 0 || row_bytes == 0) return cudaSuccess;
    if (row_bytes % 16 != 0) {
        if (row_bytes % 4 != 0 || scale != nullptr) return cudaErrorInvalidValue;
        return launch_dependent(gather_words_kernel, dim3((num_dst_rows + kPermThreads / 32 - 1) / (kPermThreads / 32)), kPermThreads, 0, stream,
                                static_cast<const uint32_t*>(src), static_cast<uint32_t*>(dst), src_row, num_dst_rows, row_bytes / 4);
    }
    const int spans = (row_bytes / 16 + kGatherSpan - 1) / kGatherSpan;
    const long long warps = (long long)num_dst_rows * spans;
    return launch_dependent(gather_rows_kernel, dim3((unsigned)((warps + kPermThreads / 32 - 1) / (kPermThreads / 32))), kPermThreads, 0, stream,
                            static_cast<const char*>(src), static_cast<char*>(dst), src_row, scale, num_dst_rows, row_bytes);
}

// dst[m] = src[src_row[m]] like the gather, each source row read once: a warp takes a span of a row and stores it to all its places, or, in front of those,
// looks at four rows of the result and fills the ones that no place names: zeros where src_row says padding. A place counts where src_row agrees with it, so that
// a plan whose maps have been changed since they were built has the gather's result, row for row. That agreement costs 0 to 2 % (8192 tokens x 6, rows of 8 KB 79.8 /
// 81.2 us, 6300 x 2 30.7 / 30.2, x 1 16.4 / 14.7, 4096 x 8 of 14 KB 90.4 / 91.8); with the filling warps last, eight rows each, 92 / 45 / 23 / 112.
constexpr int kSpreadLoads = 4;
constexpr int kSpreadSpan = 32 * kSpreadLoads;  // 16-byte columns
constexpr int kSpreadFill = 4;                  // rows of the result

__global__ void __launch_bounds__(kPermThreads) spread_rows_kernel(const char* __restrict__ src, char* __restrict__ dst, const int* __restrict__ pos,
                                                                  const int* __restrict__ src_row, int num_src_rows, int num_k, int num_dst_rows, int n16) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const int lane = threadIdx.x & 31, spans = (n16 + kSpreadSpan - 1) / kSpreadSpan;
    const long long fill = (num_dst_rows + kSpreadFill - 1) / kSpreadFill, item = (long long)blockIdx.x * (kPermThreads / 32) + (threadIdx.x >> 5) - fill, spread = (long long)num_src_rows * spans;
    if (item >= spread) return;
    if (item < 0) {
        constexpr int kLanes = 32 / kSpreadFill;
        constexpr unsigned kMask = 0xffffffffu >> (32 - kLanes);
        const long long m0 = (item + fill) * kSpreadFill, m = m0 + lane / kLanes;
        const int s = m < num_dst_rows ? src_row[m] : -1;
        bool placed = false;
        if (s >= 0 && s < num_src_rows)
            for (int k = lane % kLanes; k < num_k; k += kLanes) placed |= pos[(size_t)s * num_k + k] == (int)m;
        const unsigned named = __ballot_sync(0xffffffffu, placed);
        for (int j = 0; j < kSpreadFill; ++j) {
            if (m0 + j >= num_dst_rows || ((named >> (kLanes * j)) & kMask) != 0) continue;
            const int from = __shfl_sync(0xffffffffu, s, kLanes * j);
            const int4* p = reinterpret_cast<const int4*>(src) + (size_t)max(from, 0) * n16;
            int4* d = reinterpret_cast<int4*>(dst) + (size_t)(m0 + j) * n16;
            for (int i = lane; i < n16; i += 32) st_once(d + i, from >= 0 ? __ldg(p + i) : make_int4(0, 0, 0, 0));
        }
        return;
    }
    const int n = (int)(item / spans), i0 = (int)(item % spans) * kSpreadSpan + lane;
    const int4* p = reinterpret_cast<const int4*>(src) + (size_t)n * n16 + i0;
    int place = lane < num_k ? pos[(size_t)n * num_k + lane] : -1;  // (in front of the row, so that what src_row says to it comes no later than the row)
    int4 v[kSpreadLoads];
#pragma unroll
    for (int u = 0; u < kSpreadLoads; ++u)
        if (i0 + u * 32 < n16) v[u] = ld_once(p + u * 32);
    if (place >= num_dst_rows || (place >= 0 && src_row[place] != n)) place = -1;
    for (int k = 0; k < num_k; ++k) {
        const int row = __shfl_sync(0xffffffffu, place, k);
        if (row < 0) continue;
        int4* d = reinterpret_cast<int4*>(dst) + (size_t)row * n16 + i0;
#pragma unroll
        for (int u = 0; u < kSpreadLoads; ++u)
            if (i0 + u * 32 < n16) st_once(d + u * 32, v[u]);
    }
}

// e4m3 rows and their scales (num_kb per row) together: the scales of a row come and go with its first span, as floats or as the words of scale atoms (row r of
// a tile at (r & 31) * 16 + (r >> 5) * 4 of the K block's 512 bytes). Two launches, or three with the atoms, cost a short prompt more than the copies.
__global__ void __launch_bounds__(kPermThreads) gather_quantised_kernel(const char* __restrict__ src, const float* __restrict__ src_scales, char* __restrict__ dst,
                                                                       float* __restrict__ scales, uint8_t* __restrict__ atoms, const int* __restrict__ src_row,
                                                                       int* __restrict__ sched, int num_dst_rows, int hidden) {
    pdl_wait_predecessor();
    pdl_release_successor();
    if (sched != nullptr && blockIdx.x == 0 && threadIdx.x < 2) sched[threadIdx.x] = 0;
    const int lane = threadIdx.x & 31;
    const int n16 = hidden / 16, num_kb = hidden / 128, spans = (n16 + kGatherSpan - 1) / kGatherSpan;
    const int item = blockIdx.x * (kPermThreads / 32) + (threadIdx.x >> 5);
    const int m = item / spans, span = item % spans;
    if (m >= num_dst_rows) return;
    const int s = src_row[m];
    const int i0 = span * kGatherSpan + lane;
    constexpr int U = kGatherSpan / 32;
    int4 v[U];
    const int4* p = reinterpret_cast<const int4*>(src + (size_t)max(s, 0) * hidden);
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = (s >= 0 && i0 + u * 32 < n16) ? __ldg(p + i0 + u * 32) : make_int4(0, 0, 0, 0);
    if (span == 0) {
        for (int kb = lane; kb < num_kb; kb += 32) {
            const float f = s >= 0 ? src_scales[(size_t)s * num_kb + kb] : 0.f;
            if (atoms != nullptr)
                *reinterpret_cast<uint32_t*>(atoms + ((size_t)(m >> 7) * num_kb + kb) * 512 + (m & 31) * 16 + ((m >> 5) & 3) * 4) = ((__float_as_uint(f) >> 23) & 0xffu) * 0x01010101u;
            else scales[(size_t)m * num_kb + kb] = f;
        }
    }
    int4* d = reinterpret_cast<int4*>(dst + (size_t)m * hidden);
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (i0 + u * 32 < n16) st_once(d + i0 + u * 32, v[u]);
}

// Sources that the rows written would push out of the L2 between one reading and the next go the other way round, each row read once (52736 rows of 8 KB are
// written at 3.2 TB/s with gathered reads from 67 MB, at 6.5 without reads). Time spread / gathered, rows of 2 to 14 KB, 2 to 8 places each:
//   source MB   8          16         24         32         40         48         56         64         80
//               0.89-1.13  0.96-1.13  0.99-1.09  0.94-1.05  0.90-1.04  0.88-1.00  0.85-1.01  0.82-0.97  0.78-0.95
constexpr long long kSpreadMinBytes = 48ll << 20;

cudaError_t launch_permute_rows(const void* src, void* dst, const int* pos, const int* src_row, int num_src_rows, int num_k, int num_dst_rows, int row_bytes, cudaStream_t stream) {
    if (num_dst_rows <= 0 || row_bytes == 0) return cudaSuccess;
    if (row_bytes % 16 != 0 || pos == nullptr || num_k < 1 || num_k > 32 || (long long)num_src_rows * row_bytes < kSpreadMinBytes)
        return launch_gather_rows(src, dst, src_row, nullptr, num_dst_rows, row_bytes, stream);
    const int n16 = row_bytes / 16;
    const long long warps = (long long)num_src_rows * ((n16 + kSpreadSpan - 1) / kSpreadSpan) + (num_dst_rows + kSpreadFill - 1) / kSpreadFill;
    return launch_dependent(spread_rows_kernel, dim3((unsigned)((warps + kPermThreads / 32 - 1) / (kPermThreads / 32))), kPermThreads, 0, stream, static_cast<const char*>(src),
                            static_cast<char*>(dst), pos, src_row, num_src_rows, num_k, num_dst_rows, n16);
}

cudaError_t launch_gather_quantised(const void* src, const float* src_scales, void* dst, float* scales, uint8_t* atoms, const int* src_row, int num_dst_rows, int hidden,
                                    int* sched, cudaStream_t stream) {
    if (num_dst_rows <= 0) return cudaSuccess;
    if (hidden % 128 != 0 || hidden == 0 || (scales == nullptr) == (atoms == nullptr)) return cudaErrorInvalidValue;
    const int spans = (hidden / 16 + kGatherSpan - 1) / kGatherSpan;
    const long long warps = (long long)num_dst_rows * spans;
    return launch_dependent(gather_quantised_kernel, dim3((unsigned)((warps + kPermThreads / 32 - 1) / (kPermThreads / 32))), kPermThreads, 0, stream,
                            static_cast<const char*>(src), src_scales, static_cast<char*>(dst), scales, atoms, src_row, sched, num_dst_rows, hidden);
}

cudaError_t launch_gather_reduce_rows(const void* src, void* dst, const int* pos, const float* w, int num_dst_rows, int num_k, int hidden,
                                      cudaStream_t stream) {
    if (num_dst_rows <= 0) return cudaSuccess;
    if (hidden % 8 != 0 || num_k > 32 || num_k < 1) return cudaErrorInvalidValue;
    if (hidden == 0) return cudaSuccess;
    return launch_dependent(gather_reduce_rows_kernel, dim3(std::min(reduce_ctas(num_dst_rows, hidden / 8), 148 * kGatherReduceCtasPerSm)), kReduceThreads, 0, stream,
                            static_cast<const __nv_bfloat16*>(src), static_cast<__nv_bfloat16*>(dst), pos, w, num_dst_rows, num_k, hidden);
}

}  // namespace dx
