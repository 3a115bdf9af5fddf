// Stable listing of the selections of a few experts out of topk_idx, by one CTA.
//
// Every CTA reads all expert ids (8 bytes per selection, from L2 after the first CTA) and keeps the ones of its own experts, so the
// list of an expert comes out in selection order without atomics, a sort or a second launch. Cost per CTA: the ids stream through
// at L2 speed (32768 selections: about 3 us), one vote per 32 selections and expert. Votes of one expert on eight groups at a time keep that to a
// compare, a vote and a store each, and the CTAs do not all start at the same ids: build_plan of 4096 x 8 selections, 256 experts 12.1 -> 10.0 us, of
// 8192 x 8, 64 experts 17.9 -> 13.9, of 20000 x 8 81 -> 61.
#pragma once

#include "prims.cuh"

namespace dx {

constexpr int kScanThreads = 1024;
constexpr int kScanWarps = kScanThreads / 32;
constexpr int kScanChunk = kScanThreads * 32;  // selections per pass: one 32-selection group per thread

constexpr int kScanBatch = 16;  // experts of one pass over the ids (more experts per CTA take more passes)

// Dynamic shared memory of a scanning CTA: a running count per expert, then a vote word per (expert, group).
__host__ __device__ constexpr size_t scan_smem_bytes(int experts_per_cta) {
    return kScanBatch * sizeof(int) + (size_t)(experts_per_cta < kScanBatch ? experts_per_cta : kScanBatch) * kScanThreads * sizeof(uint32_t);
}

// Calls emit(j, n, i) for the n-th selection i (index into ids) of expert e0 + j, and none(i) for selections without a valid expert
// when `want_none` is set; s_run[j] ends up as the number of selections of expert e0 + j. All threads of the CTA take part.
template <typename Emit, typename None>
__device__ __forceinline__ void scan_selections(const int64_t* __restrict__ ids, int total, int num_experts, int e0, int ne, uint32_t* s_vote,
                                                int* s_run, bool want_none, Emit emit, None none) {
    __shared__ int s_warp_sum[kScanWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int j = tid; j < ne; j += kScanThreads) s_run[j] = 0;
    for (int c0 = 0; c0 < total; c0 += kScanChunk) {
        __syncthreads();
        // warp w votes on the groups w, w + 32, ... of the chunk, eight id loads in flight per lane: a short list is one trip to memory for all warps, where 32
        // neighbouring groups per warp were four for a few of them (build_plan, 64 experts, 777 x 6 selections: 9.0 -> 4.8 us; 256 experts, 777 x 8 11.0 -> 6.0).
        // (CTAs start at different quarters of the chunk: all of them read the same ids)
        for (int r = 0; r < 32; r += 8) {
            const int g0 = (r + (blockIdx.x & 3) * 8) & 31;
            if (c0 + g0 * kScanThreads >= total) continue;
            int64_t id[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = c0 + ((g0 + u) * 32 + warp) * 32 + lane;
                id[u] = i < total ? ids[i] : (int64_t)num_experts;
            }
            int rel[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = c0 + ((g0 + u) * 32 + warp) * 32 + lane;
                const bool valid = id[u] >= 0 && id[u] < num_experts;
                if (want_none && !valid && i < total) none(i);
                rel[u] = valid ? (int)id[u] - e0 : -1;
            }
            for (int j = 0; j < ne; ++j) {
                uint32_t* votes = s_vote + j * kScanThreads + g0 * 32 + warp;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const unsigned b = __ballot_sync(0xffffffffu, rel[u] == j);
                    if (lane == 0) votes[u * 32] = b;
                }
            }
        }
        __syncthreads();
        // thread t owns group t: its place in the list is the number of votes in the groups before it
        for (int j = 0; j < ne; ++j) {
            unsigned votes = c0 + tid * 32 < total ? s_vote[j * kScanThreads + tid] : 0u;
            const int n = __popc(votes);
            const int incl = warp_incl_scan(n);
            if (lane == 31) s_warp_sum[warp] = incl;
            __syncthreads();
            int before = 0, all = 0;
            {
                const int v = s_warp_sum[lane];
                const int vi = warp_incl_scan(v);
                before = __shfl_sync(0xffffffffu, vi - v, warp);
                all = __shfl_sync(0xffffffffu, vi, 31);
            }
            const int base = s_run[j];
            int slot = base + before + incl - n;
            for (; votes != 0; votes &= votes - 1) emit(j, slot++, c0 + tid * 32 + __ffs(votes) - 1);
            __syncthreads();
            if (tid == 0) s_run[j] = base + all;
        }
    }
    __syncthreads();
}

}  // namespace dx
