// get_dispatch_layout: from topk_idx[T,K] compute how many tokens go to every rank and expert and the
// [T,R] membership matrix, in ONE launch that needs no pre-zeroed outputs.
//
// Up to 1024 tokens one CTA histograms them in shared memory, up to 8192 the CTAs of one cluster do. Beyond, each CTA stores the partial
// histogram of 256 tokens, takes a ticket, and the last CTA to finish sums the partials. Experts are block-partitioned over ranks:
// expert e lives on rank e / (E/R). A selection of -1 (or out of range) is ignored.
//
// Reference counterpart: csrc/kernels/layout.cu:9-149 (one CTA per 4 experts / 8 ranks, every CTA
// re-reading all of topk_idx). Outputs are identical: num_tokens_per_rank[R] i32,
// num_tokens_per_expert[E] i32, is_token_in_rank[T,R] bool.
#include <algorithm>

#include "api.h"
#include "launch.cuh"
#include "prims.cuh"

namespace dx {

constexpr int kLayoutThreads = 256;
constexpr int kLayoutMaxThreads = 1024;
constexpr int kLayoutCluster = 8;

// bins per CTA: experts, ranks, and one per NVLink domain when those are counted too
size_t layout_scratch_ints(int num_experts, int num_ranks, int num_tokens, int num_nodes) {
    const size_t ctas = (num_tokens + kLayoutThreads - 1) / kLayoutThreads;
    return 1 + (ctas > 0 ? ctas : 1) * (size_t)(num_experts + num_ranks + num_nodes);
}

struct LayoutBins {
    int L, P, nodes, all;
    __device__ __forceinline__ explicit LayoutBins(const LayoutArgs& a)
        : L(a.num_experts / a.num_ranks), P(a.ranks_per_node > 0 ? a.ranks_per_node : a.num_ranks),
          nodes(a.num_tokens_per_node != nullptr ? a.num_ranks / P : 0), all(a.num_experts + a.num_ranks + nodes) {}
};

// Counts token t into s_hist ([E] experts, [R] ranks, [R / ranks_per_node] NVLink domains) and writes its membership row; every lane of the warp takes part.
__device__ __forceinline__ void count_token(const LayoutArgs& a, const LayoutBins& bins, int* s_hist, int t) {
    const int E = a.num_experts, R = a.num_ranks, K = a.num_topk, L = bins.L, P = bins.P, nodes = bins.nodes;
    uint64_t mask = 0;
    if (t < a.num_tokens) {
        const int64_t* row = a.topk_idx + (size_t)t * K;
        // eight ids are requested before the first one is looked at: one trip to memory per eight selections
        for (int k0 = 0; k0 < K; k0 += 8) {
            int64_t ids[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) ids[k] = k0 + k < K ? row[k0 + k] : -1;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (ids[k] >= 0 && ids[k] < E) {
                    atomicAdd(&s_hist[(int)ids[k]], 1);
                    mask |= 1ull << ((int)ids[k] / L);
                }
            }
        }
        if (R == 8) {
            uint64_t packed = 0;
#pragma unroll
            for (int r = 0; r < 8; ++r) packed |= (uint64_t)((mask >> r) & 1u) << (8 * r);
            *reinterpret_cast<uint64_t*>(a.is_token_in_rank + (size_t)t * 8) = packed;
        } else {
            for (int r = 0; r < R; ++r) a.is_token_in_rank[(size_t)t * R + r] = (mask >> r) & 1u;
        }
    }
    for (int n = 0; n < nodes; ++n) {
        const uint64_t node_bits = (P >= 64 ? ~0ull : ((1ull << P) - 1ull)) << (n * P);
        const unsigned b = __ballot_sync(0xffffffffu, (mask & node_bits) != 0);
        if ((threadIdx.x & 31) == 0 && b) atomicAdd(&s_hist[E + R + n], __popc(b));
    }
    // per-rank counts: one ballot per rank, one shared atomic per warp
    for (int r = 0; r < R; ++r) {
        const unsigned b = __ballot_sync(0xffffffffu, (mask >> r) & 1u);
        if ((threadIdx.x & 31) == 0 && b) atomicAdd(&s_hist[E + r], __popc(b));
    }
}

__device__ __forceinline__ void publish_bin(const LayoutArgs& a, int i, int sum) {
    const int E = a.num_experts, R = a.num_ranks;
    if (i < E) a.num_tokens_per_expert[i] = sum;
    else if (i < E + R) a.num_tokens_per_rank[i - E] = sum;
    else a.num_tokens_per_node[i - E - R] = sum;
}

__global__ void __launch_bounds__(kLayoutMaxThreads) layout_kernel(const LayoutArgs a) {
    extern __shared__ int s_hist[];
    const LayoutBins bins(a);
    for (int i = threadIdx.x; i < bins.all; i += blockDim.x) s_hist[i] = 0;
    pdl_wait_predecessor();
    pdl_release_successor();
    __syncthreads();
    count_token(a, bins, s_hist, blockIdx.x * blockDim.x + threadIdx.x);
    __syncthreads();
    if (gridDim.x == 1) {  // one CTA has seen every token
        for (int i = threadIdx.x; i < bins.all; i += blockDim.x) publish_bin(a, i, s_hist[i]);
        return;
    }
    int* partial = a.scratch + 1 + (size_t)blockIdx.x * bins.all;
    for (int i = threadIdx.x; i < bins.all; i += blockDim.x) partial[i] = s_hist[i];

    if (cta_is_last(a.scratch, gridDim.x)) {
        for (int i = threadIdx.x; i < bins.all; i += blockDim.x) {
            int sum = 0;
#pragma unroll 8
            for (int b = 0; b < (int)gridDim.x; ++b) sum += __ldcg(a.scratch + 1 + (size_t)b * bins.all + i);
            publish_bin(a, i, sum);
        }
    }
}

// Up to 8192 tokens: the CTAs of one cluster sum their histograms from each other's shared memory, where partial histograms in global memory, a ticket and
// the last CTA's loads were two trips more (us, before / after: 257 x 6 of 64 experts 5.2 / 3.2, 777 x 6 5.9 / 4.0, 1500 x 8 of 256 7.3 / 4.4, 4096 x 8 6.0 / 5.4).
__global__ void __launch_bounds__(kLayoutMaxThreads) __cluster_dims__(kLayoutCluster, 1, 1) layout_cluster_kernel(const LayoutArgs a) {
    extern __shared__ int s_hist[];
    const LayoutBins bins(a);
    for (int i = threadIdx.x; i < bins.all; i += blockDim.x) s_hist[i] = 0;
    pdl_wait_predecessor();
    pdl_release_successor();
    __syncthreads();
    count_token(a, bins, s_hist, blockIdx.x * blockDim.x + threadIdx.x);
    cluster_sync();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < bins.all; i += kLayoutCluster * blockDim.x) {
        const uint32_t own = (uint32_t)__cvta_generic_to_shared(s_hist + i);
        int sum = 0;
#pragma unroll
        for (int b = 0; b < kLayoutCluster; ++b) sum += ld_cluster_s32(own, b);
        publish_bin(a, i, sum);
    }
    cluster_sync();  // nobody leaves while its histogram may still be read
}

cudaError_t launch_layout(const LayoutArgs& a, cudaStream_t stream) {
    if (a.num_ranks > 64) return cudaErrorInvalidValue;
    const size_t smem = (size_t)(a.num_experts + 2 * a.num_ranks) * sizeof(int);  // upper bound of the bins
    auto warps = [](int tokens) { return std::max((tokens + 31) / 32 * 32, 32); };
    if (a.num_tokens <= kLayoutMaxThreads) return launch_dependent(layout_kernel, dim3(1), std::max(warps(a.num_tokens), kLayoutThreads), smem, stream, a);
    if (a.num_tokens <= kLayoutCluster * kLayoutMaxThreads)
        return launch_dependent(layout_cluster_kernel, dim3(kLayoutCluster), warps((a.num_tokens + kLayoutCluster - 1) / kLayoutCluster), smem, stream, a);
    return launch_dependent(layout_kernel, dim3((a.num_tokens + kLayoutThreads - 1) / kLayoutThreads), kLayoutThreads, smem, stream, a);
}

}  // namespace dx
