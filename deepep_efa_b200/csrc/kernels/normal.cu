// Normal (high-throughput) mode over one NVSwitch domain: notify, dispatch, combine, barrier.
//
// Design (differs from the reference on purpose):
//  * No ring queues, no channels, no flow control. With 180 GB per GPU the receiver's FINAL output
//    tensors live in its peer-mapped symmetric arena, and a count exchange tells every sender the
//    exact destination row of every token before any payload moves. Senders then store rows straight
//    into the peers' final tensors (push, 16-byte stores, optional fused BF16->FP8 block quantisation)
//    and the receiver never touches the payload.
//  * Combine is the mirror image as a PULL: the token's home rank loads the <= R expert-output rows
//    from the peers' symmetric memory, reduces them in fp32 (+bias), and writes BF16 once.
//  * Completion is one cross-rank sequence barrier at the end of each kernel; all sequence numbers
//    are monotonic, so nothing is cleaned between calls.
//  * Every wait is bounded and reports through the status word.
//
// Row order at the receiver is (source rank, source token order), which is exactly the order the
// reference produces with its (rank, channel, token) rings because channels are contiguous token
// ranges (csrc/kernels/intranode.cu:410-426, 464).
//
// Reference counterparts: notify_dispatch / cached_notify_dispatch (intranode.cu:11-195),
// dispatch (:197-610), cached_notify_combine / combine (:612-1099), intranode::barrier (runtime.cu:13-26).
#include <algorithm>

#include "api.h"
#include "prims.cuh"
#include "launch.cuh"

namespace dx {

// Indices into RankCtx::local_scratch (ints, zero between kernels).
constexpr int kTicketDispatch = 0;
constexpr int kTicketCombine = 1;
constexpr int kTicketNotify = 2;

// =============================================================================================
// notify
// =============================================================================================
constexpr int kNotifyThreads = 1024;

template <int V>
__global__ void __launch_bounds__(kNotifyThreads, 1) notify_kernel(const __grid_constant__ ArgPack<NotifyArgs, V> pack) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const NotifyArgs& a = pack.a[blockIdx.y];
    const RankCtx& c = a.ctx;
    const int R = c.num_ranks, me = c.rank;
    const int E = a.num_experts, L = E / R, C = a.num_channels, T = a.num_tokens;
    const int tid = threadIdx.x;
    const uint64_t seq = next_seq(c, kFamNotify);
    __shared__ int s_ok;
    __shared__ int s_warp_sums[kNotifyThreads / 32];
    __shared__ int s_off[kNotifyThreads + 1];

    if (blockIdx.x == 0) {
        // ---- CTA 0: exchange counts with every rank, build the prefix matrix, tell the host ----
        if (tid == 0) s_ok = 1;
        for (int d = 0; d < R; ++d) {
            ControlBlock* pc = c.ctrl(d);
            if (tid < R) st_relaxed_sys(&pc->notify_rank_counts[me][tid], a.num_tokens_per_rank[tid]);
            for (int i = tid; i < L; i += kNotifyThreads)
                st_relaxed_sys(&pc->notify_expert_counts[me][i], a.num_tokens_per_expert[d * L + i]);
        }
        __syncthreads();
        // this rank's own counts need no flag: the barrier above orders them for this CTA, their only reader
        if (tid < R && tid != me) {
            st_release_sys(&c.ctrl(tid)->notify_seq[me], seq);
            if (!wait_ge_sys(&c.my_ctrl()->notify_seq[tid], seq, c.timeout_cycles)) {
                report(c.status, kTimeoutNotify, me, tid, 0);
                s_ok = 0;
            }
        }
        __syncthreads();
        if (!s_ok) {
            if (tid == 0 && a.host_recv_counter != nullptr) {
                *a.host_recv_counter = -2;  // tells the host to stop waiting
                __threadfence_system();
            }
            return;
        }
        ControlBlock* my = c.my_ctrl();
        if (tid < R) {
            int running = 0;
            for (int i = 0; i < R; ++i) {
                running += ld_relaxed_sys(&my->notify_rank_counts[i][tid]);
                a.rank_prefix_matrix[i * R + tid] = running;
            }
            if (tid == me && a.host_recv_counter != nullptr) *a.host_recv_counter = running;
        }
        for (int e = tid; e < L && a.host_expert_counter != nullptr; e += kNotifyThreads) {
            int sum = 0;
            for (int i = 0; i < R; ++i) sum += ld_relaxed_sys(&my->notify_expert_counts[i][e]);
            const int al = a.expert_alignment;
            a.host_expert_counter[e] = (sum + al - 1) / al * al;
        }
        // (the host polls every one of these words for itself, so they need no order among themselves)
        // channel prefix rows pushed by the scan CTAs of my peers; my own row is written by my scan CTA
        if (tid < R && tid != me) {
            uint64_t dummy;
            if (!mailbox_wait(c, kMbChanPrefix, tid, seq, &dummy, 0)) {
                report(c.status, kTimeoutNotify, me, tid, 1);
                s_ok = 0;
            }
        }
        __syncthreads();
        if (!s_ok) return;
        for (int i = tid; i < R * C; i += kNotifyThreads)
            if (i / C != me) a.recv_channel_prefix_matrix[i] = ld_relaxed_sys(&my->chan_prefix_in[i / C][i % C]);
        if (cta_is_last(c.local_scratch + kTicketNotify, gridDim.x) && tid == 0) commit_seq(c, kFamNotify, seq);
        return;
    }

    // ---- CTA 1+d: positions of my tokens inside the (me -> d) stream ----
    const int d = blockIdx.x - 1;
    const int per = (T + kNotifyThreads - 1) / kNotifyThreads;
    const int begin = min(tid * per, T), end = min(begin + per, T);
    int cnt = 0;
    for (int t = begin; t < end; ++t) cnt += a.is_token_in_rank[(size_t)t * R + d] ? 1 : 0;
    // block exclusive scan of cnt
    const int incl = warp_incl_scan(cnt);
    if ((tid & 31) == 31) s_warp_sums[tid >> 5] = incl;
    __syncthreads();
    if (tid < 32) {
        const int w = s_warp_sums[tid];
        const int wi = warp_incl_scan(w);
        s_warp_sums[tid] = wi - w;
    }
    __syncthreads();
    int pos = s_warp_sums[tid >> 5] + incl - cnt;
    // keep exclusive offsets for the channel prefix computation
    s_off[tid] = pos;
    if (tid == kNotifyThreads - 1) s_off[kNotifyThreads] = pos + cnt;
    for (int t = begin; t < end; ++t) {
        const bool in = a.is_token_in_rank[(size_t)t * R + d];
        a.send_head[(size_t)t * R + d] = in ? pos : -1;
        pos += in ? 1 : 0;
    }
    __syncthreads();
    // channel ch covers tokens [ch*tpc, min((ch+1)*tpc, T)); prefix = tokens to d in channels <= ch
    const int tpc = (T + C - 1) / C;
    if (tid < C) {
        const int b = min((tid + 1) * tpc, T);  // count flagged tokens with index < b
        int owner = per > 0 ? b / per : 0;
        if (owner > kNotifyThreads) owner = kNotifyThreads;
        int prefix = s_off[owner];
        if (owner < kNotifyThreads)
            for (int t = owner * per; t < b; ++t) prefix += a.is_token_in_rank[(size_t)t * R + d] ? 1 : 0;
        a.channel_prefix_matrix[d * C + tid] = prefix;
        if (d == me) a.recv_channel_prefix_matrix[me * C + tid] = prefix;
        else st_relaxed_sys(&c.ctrl(d)->chan_prefix_in[me][tid], prefix);
    }
    __syncthreads();
    if (tid == 0 && d != me) {
        mailbox_post(c, kMbChanPrefix, d, nullptr, 0, seq);
    }
    if (cta_is_last(c.local_scratch + kTicketNotify, gridDim.x) && tid == 0) commit_seq(c, kFamNotify, seq);
}

// A lone rank exchanges nothing: the counts go from the layout's tensors to the host, and one CTA numbers the tokens. The general kernel takes the counts through
// the words that peers would write, and reads every flag three times (us, before / after: 1 token 6.2 / 4.7, 777 5.7 / 4.6, 4096 6.0 / 4.9, 8192 9.0 / 8.1).
__global__ void __launch_bounds__(kNotifyThreads, 1) notify_lone_kernel(const __grid_constant__ NotifyArgs a) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const int T = a.num_tokens, C = a.num_channels, tid = threadIdx.x;
    __shared__ int s_warp_sums[kNotifyThreads / 32];
    __shared__ int s_off[kNotifyThreads + 1];
    // flags of this thread's tokens; up to 8192 tokens they stay in a register
    const int per = (T + kNotifyThreads - 1) / kNotifyThreads;
    const int begin = min(tid * per, T), end = min(begin + per, T);
    auto flag = [&](int t) { return a.is_token_in_rank[t] ? 1u : 0u; };
    unsigned bits = 0;
    int cnt = 0;
    if (per <= 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (begin + j < end) bits |= flag(begin + j) << j;
        cnt = __popc(bits);
    } else {
        for (int t = begin; t < end; ++t) cnt += (int)flag(t);
    }
    if (tid == 0) {
        const int total = a.num_tokens_per_rank[0];
        a.rank_prefix_matrix[0] = total;
        if (a.host_recv_counter != nullptr) *a.host_recv_counter = total;
    }
    const int al = a.expert_alignment;
    for (int e = tid; e < a.num_experts && a.host_expert_counter != nullptr; e += kNotifyThreads)
        a.host_expert_counter[e] = (a.num_tokens_per_expert[e] + al - 1) / al * al;
    const int incl = warp_incl_scan(cnt);
    if ((tid & 31) == 31) s_warp_sums[tid >> 5] = incl;
    __syncthreads();
    const int before = warp_incl_scan(s_warp_sums[tid & 31]);  // every warp for itself
    int pos = incl - cnt + ((tid >> 5) > 0 ? __shfl_sync(0xffffffffu, before, (tid >> 5) - 1) : 0);
    s_off[tid] = pos;
    if (tid == kNotifyThreads - 1) s_off[kNotifyThreads] = pos + cnt;
    for (int t = begin; t < end; ++t) {
        const bool in = per <= 8 ? (bits >> (t - begin)) & 1u : flag(t) != 0;
        a.send_head[t] = in ? pos : -1;
        pos += in ? 1 : 0;
    }
    __syncthreads();
    const int tpc = (T + C - 1) / C;  // channel ch covers the tokens [ch * tpc, (ch + 1) * tpc)
    if (tid < C) {
        const int b = min((tid + 1) * tpc, T);
        const int owner = per > 0 ? min(b / per, kNotifyThreads) : 0;
        int prefix = s_off[owner];
        if (owner < kNotifyThreads)
            for (int t = owner * per; t < b; ++t) prefix += (int)flag(t);
        a.channel_prefix_matrix[tid] = prefix;
        a.recv_channel_prefix_matrix[tid] = prefix;
    }
}

cudaError_t launch_notify(const NotifyArgs* a, int nv, cudaStream_t stream) {
    if (nv == 1 && a->ctx.num_ranks == 1) return launch_dependent(notify_lone_kernel, dim3(1), kNotifyThreads, 0, stream, *a);
    return DX_LAUNCH_RANKED_PDL(notify_kernel, NotifyArgs, a, nv, 1 + a[0].ctx.num_ranks, kNotifyThreads, 0, stream);
}

// =============================================================================================
// dispatch (push)
// =============================================================================================
constexpr int kDispatchThreads = 1024;
constexpr int kDispatchWarps = kDispatchThreads / 32;

struct PeerDst {
    char* x;
    float* scales;
    int64_t* topk_idx;
    float* topk_w;
    int* src_idx;
    int base_row;  // rows of ranks before me at that peer
};

// A warp's share of the rows: item i = (token i / pieces, piece i % pieces). Items are dealt out CTA by CTA, so that every SM
// gets work when there are fewer items than warps, and a small batch cuts its rows into pieces (each at least kMinPiece 16-byte
// columns of the row) until there is about one item per warp: a lone warp moves an 8 KB row in four dependent steps, about 4 us.
constexpr int kMinPiece16 = 64;
constexpr int kMaxPieces = 8;

__device__ __forceinline__ int row_pieces(int num_tokens, int n16, int total_warps) {
    int p = 1;
    while (p < kMaxPieces && 2 * p * num_tokens <= total_warps && n16 / (2 * p) >= kMinPiece16) p *= 2;
    return p;
}

// CTAs of a launch: the caller's bound, and no more than have a token to move.
template <typename Args>
int grid_ctas(const Args* a, int nv) {
    int most = 1;
    for (int i = 0; i < nv; ++i) most = a[i].num_tokens > most ? a[i].num_tokens : most;
    return a[0].num_sms < most ? a[0].num_sms : most;
}

template <int kRanks>
__device__ __forceinline__ void dispatch_rows(const DispatchArgs& a, const PeerDst* s_dst, float* s_scales, int warp, int lane) {
    const RankCtx& c = a.ctx;
    const int R = c.num_ranks, T = a.num_tokens, K = a.num_topk;
    const int L = a.num_experts / R;
    const int H = a.hidden;
    const bool quant = a.quantize != 0;
    const size_t out_row_bytes = (size_t)H * (quant ? 1 : a.x_elem_bytes);
    const int num_scales = H / 128;
    // columns of a row in the unit its pieces are cut in: 16 bytes, or (quantising) the 512 channels a warp converts per step
    const int n16 = (int)(out_row_bytes / 16);
    const int pieces = row_pieces(T, quant ? H / 8 : n16, gridDim.x * kDispatchWarps);

    for (int item = blockIdx.x + gridDim.x * warp; item < T * pieces; item += gridDim.x * kDispatchWarps) {
        const int t = item / pieces, piece = item % pieces;
        // destination rows
        int head = (lane < R) ? a.send_head[(size_t)t * R + lane] : -1;
        const unsigned dmask = __ballot_sync(0xffffffffu, head >= 0);
        if (dmask == 0) continue;
        int rows[kRanks];
#pragma unroll
        for (int d = 0; d < kRanks; ++d) {
            const int h = __shfl_sync(0xffffffffu, head, d);
            rows[d] = (d < R && h >= 0) ? s_dst[d].base_row + h : -1;
            if (c.debug_extent != 0 && rows[d] >= 0 && !peer_range_ok(c, d, s_dst[d].x + (size_t)rows[d] * out_row_bytes, out_row_bytes, 1)) rows[d] = -1;
        }

        if (!quant) {
            // ---- pass-through rows (bf16 or already-quantised e4m3) ----
            const int per = (((n16 + pieces - 1) / pieces) + 31) & ~31;
            const int end = min(n16, (piece + 1) * per);
            const int4* src = reinterpret_cast<const int4*>(reinterpret_cast<const char*>(a.x) + (size_t)t * out_row_bytes);
            // loads in flight per lane: a store to a peer occupies the lane for longer than one to this GPU, so the one-rank form
            // (bound by the latency of its own loads) asks for twice as many
            constexpr int U = kRanks == 1 ? 8 : 4;
            for (int i0 = piece * per; i0 < end; i0 += 32 * U) {
                int4 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u * 32 + lane;
                    if (i < end) v[u] = ld_stream(src + i);
                }
#pragma unroll
                for (int d = 0; d < kRanks; ++d) {
                    if (rows[d] < 0) continue;
                    int4* dst = reinterpret_cast<int4*>(s_dst[d].x + (size_t)rows[d] * out_row_bytes);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int i = i0 + u * 32 + lane;
                        if (i < end) st_stream(dst + i, v[u]);
                    }
                }
            }
            if (a.x_scales != nullptr && piece == 0) {
                for (int i = lane; i < num_scales; i += 32) {
                    const float s = a.x_scales[(size_t)t * num_scales + i];
#pragma unroll
                    for (int d = 0; d < kRanks; ++d)
                        if (rows[d] >= 0) s_dst[d].scales[(size_t)rows[d] * num_scales + i] = s;
                }
            }
        } else {
            // ---- fused BF16 -> e4m3 with one fp32 scale per 128 channels ----
            // A lane owns 16 consecutive channels, 8 lanes own one scale group, a warp covers 512
            // channels per step.
            const int per = (((H + pieces - 1) / pieces) + 511) & ~511;
            const int begin = piece * per, end = min(H, begin + per);
            const char* src = reinterpret_cast<const char*>(a.x) + (size_t)t * H * 2;
            // four 16-byte loads per lane in flight: the next 1024 channels are requested before the current ones are converted
            int4 cur[4], nxt[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int ch = begin + h * 512 + lane * 16;
                cur[2 * h] = cur[2 * h + 1] = make_int4(0, 0, 0, 0);
                if (ch < end) {
                    cur[2 * h] = ld_cached(reinterpret_cast<const int4*>(src + (size_t)ch * 2));
                    cur[2 * h + 1] = ld_cached(reinterpret_cast<const int4*>(src + (size_t)ch * 2 + 16));
                }
            }
            for (int c0 = begin; c0 < end; c0 += 1024) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int chn = c0 + 1024 + h * 512 + lane * 16;
                    nxt[2 * h] = nxt[2 * h + 1] = make_int4(0, 0, 0, 0);
                    if (chn < end) {
                        nxt[2 * h] = ld_cached(reinterpret_cast<const int4*>(src + (size_t)chn * 2));
                        nxt[2 * h + 1] = ld_cached(reinterpret_cast<const int4*>(src + (size_t)chn * 2 + 16));
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int ch = c0 + h * 512 + lane * 16;
                    const bool act = ch < end;
                    const int4 r0 = cur[2 * h], r1 = cur[2 * h + 1];
                    float f[16];
                    {
                        const uint32_t w[8] = {(uint32_t)r0.x, (uint32_t)r0.y, (uint32_t)r0.z, (uint32_t)r0.w,
                                               (uint32_t)r1.x, (uint32_t)r1.y, (uint32_t)r1.z, (uint32_t)r1.w};
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float2 p = bf16x2_to_f2(w[j]);
                            f[2 * j] = p.x;
                            f[2 * j + 1] = p.y;
                        }
                    }
                    float amax = 0.f;
#pragma unroll
                    for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(f[j]));
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
                    float scale, inv;
                    fp8_scale_from_amax(amax, a.round_scale != 0, scale, inv);
                    int4 q;
                    q.x = (int)pack_e4m3x4(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv);
                    q.y = (int)pack_e4m3x4(f[4] * inv, f[5] * inv, f[6] * inv, f[7] * inv);
                    q.z = (int)pack_e4m3x4(f[8] * inv, f[9] * inv, f[10] * inv, f[11] * inv);
                    q.w = (int)pack_e4m3x4(f[12] * inv, f[13] * inv, f[14] * inv, f[15] * inv);
                    if (act && (lane & 7) == 0) s_scales[ch >> 7] = scale;
                    if (act) {
#pragma unroll
                        for (int d = 0; d < kRanks; ++d)
                            if (rows[d] >= 0) st_stream(reinterpret_cast<int4*>(s_dst[d].x + (size_t)rows[d] * H + ch), q);
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) cur[j] = nxt[j];
            }
            __syncwarp();
            for (int i = (begin >> 7) + lane; i < (end >> 7); i += 32) {
                const float s = s_scales[i];
#pragma unroll
                for (int d = 0; d < kRanks; ++d)
                    if (rows[d] >= 0) s_dst[d].scales[(size_t)rows[d] * num_scales + i] = s;
            }
            __syncwarp();
        }
        if (piece != 0) continue;

        // ---- metadata: local expert ids, weights, source token index ----
        if (a.topk_idx != nullptr && lane < K) {
            const int64_t e = a.topk_idx[(size_t)t * K + lane];
            const float w = a.topk_weights != nullptr ? a.topk_weights[(size_t)t * K + lane] : 0.f;
#pragma unroll
            for (int d = 0; d < kRanks; ++d) {
                if (rows[d] < 0) continue;
                const bool mine = e >= (int64_t)d * L && e < (int64_t)(d + 1) * L;
                s_dst[d].topk_idx[(size_t)rows[d] * K + lane] = mine ? e - (int64_t)d * L : -1;
                if (a.topk_weights != nullptr) s_dst[d].topk_w[(size_t)rows[d] * K + lane] = mine ? w : 0.f;
            }
        }
        if (lane == 0 && a.recv_src_idx_off != kNoOffset) {
#pragma unroll
            for (int d = 0; d < kRanks; ++d)
                if (rows[d] >= 0) s_dst[d].src_idx[rows[d]] = t;
        }
    }
}

template <int V>
__global__ void __launch_bounds__(kDispatchThreads, 1) dispatch_kernel(const __grid_constant__ ArgPack<DispatchArgs, V> pack) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const DispatchArgs& a = pack.a[blockIdx.y];
    const RankCtx& c = a.ctx;
    const int R = c.num_ranks, me = c.rank, K = a.num_topk;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t seq = next_seq(c, kFamDispatch);
    __shared__ PeerDst s_dst[kMaxRanks];
    __shared__ int s_ok;
    __shared__ float s_scales[kDispatchWarps][64];

    if (tid == 0) s_ok = 1;
    __syncthreads();
    // Publish where my rows go, then learn where every peer wants its rows (my own place I know without asking).
    if (blockIdx.x == 0 && tid < R && tid != me) {
        uint64_t w[5] = {a.recv_x_off, a.recv_scales_off, a.recv_topk_idx_off, a.recv_topk_w_off, a.recv_src_idx_off};
        mailbox_post(c, kMbDispatchDesc, tid, w, 5, seq);
    }
    if (tid < R) {
        uint64_t w[5] = {a.recv_x_off, a.recv_scales_off, a.recv_topk_idx_off, a.recv_topk_w_off, a.recv_src_idx_off};
        if (tid != me && !mailbox_wait(c, kMbDispatchDesc, tid, seq, w, 5)) {
            report(c.status, kTimeoutDescriptor, me, tid, 0);
            s_ok = 0;
        } else {
            PeerDst p;
            p.x = c.at<char>(tid, w[0]);
            p.scales = c.at<float>(tid, w[1]);
            p.topk_idx = c.at<int64_t>(tid, w[2]);
            p.topk_w = c.at<float>(tid, w[3]);
            p.src_idx = c.at<int>(tid, w[4]);
            p.base_row = me > 0 ? a.rank_prefix_matrix[(me - 1) * R + tid] : 0;
            s_dst[tid] = p;
        }
    }
    __syncthreads();
    if (!s_ok) return;

    if (R <= 1) dispatch_rows<1>(a, s_dst, s_scales[warp], warp, lane);
    else if (R <= 2) dispatch_rows<2>(a, s_dst, s_scales[warp], warp, lane);
    else if (R <= 4) dispatch_rows<4>(a, s_dst, s_scales[warp], warp, lane);
    else dispatch_rows<8>(a, s_dst, s_scales[warp], warp, lane);

    // worst-case sized outputs: mark the unused tail of my own recv_topk_idx
    if (a.num_worst_tokens > 0 && a.topk_idx != nullptr) {
        const int num_recv = a.rank_prefix_matrix[(R - 1) * R + me];
        int64_t* mine = c.at<int64_t>(me, a.recv_topk_idx_off);
        const size_t lo = (size_t)num_recv * K, hi = (size_t)a.num_worst_tokens * K;
        for (size_t i = lo + (size_t)blockIdx.x * kDispatchThreads + tid; i < hi; i += (size_t)gridDim.x * kDispatchThreads)
            mine[i] = -1;
    }

    // ---- completion: when my last CTA is done, tell every peer; CTA 0 waits for every peer. A lone rank has nobody to tell
    // or to wait for (the end of the kernel is its completion), and no sequence number that anybody compares.
    if (R == 1) return;
    if (cta_is_last(c.local_scratch + kTicketDispatch, gridDim.x)) {
        if (tid < R && tid != me) st_release_sys(&c.ctrl(tid)->barrier_in[kBarDispatch][me], seq);
        if (tid == 0) commit_seq(c, kFamDispatch, seq);
    }
    if (blockIdx.x == 0 && tid < R && tid != me) {
        if (!wait_ge_sys(&c.my_ctrl()->barrier_in[kBarDispatch][tid], seq, c.timeout_cycles))
            report(c.status, kTimeoutBarrier, me, tid, 100);
    }
}

// A lone rank that may use the whole GPU: the rows only move within its memory, at the speed of a copy. A warp takes one piece of one row
// (2 KB to read when it casts, 4 KB otherwise), asks for all of it together with the row's place, stores it and ends; four CTAs of eight such
// warps share an SM, three when it combines with two biases. Casting, resident warps go on to their next piece, which is on its way while this one is
// cast (4096 x 7168 19.2 -> 17.0 us, 8192 x 7168 34.3 -> 31.1 beside one piece per warp and five CTAs; copies have no registers for that: 19.6 -> 24). With a warp per row that walked over its columns, 32 to an SM, a row of 14 KB was seven dependent steps (one B200,
// 4096 x 7168: cast to FP8 31.4 -> 19.2 us, back in BF16 27.4 -> 17.5 us with what overlaps the predecessor; 3001 x 4096 in BF16 with one
// bias 11.5 -> 8.0 and 18.3 -> 12.0 us).
constexpr int kLoneThreads = 256;
constexpr int kLoneWarps = kLoneThreads / 32;

template <bool kQuant>
__global__ void __launch_bounds__(kLoneThreads, 4) dispatch_lone_kernel(const __grid_constant__ DispatchArgs a, const int pieces) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const RankCtx& c = a.ctx;
    const int T = a.num_tokens, K = a.num_topk, H = a.hidden;
    const int lane = threadIdx.x & 31;
    const size_t out_row_bytes = (size_t)H * (kQuant ? 1 : a.x_elem_bytes);
    char* out = c.at<char>(0, a.recv_x_off);
    float* scales = c.at<float>(0, a.recv_scales_off);
    constexpr int U = kQuant ? 4 : 8;
    const int n16 = (int)(out_row_bytes / 16);
    const unsigned items = (unsigned)T * (unsigned)pieces, step = gridDim.x * kLoneWarps;
    int4 next[U];
    int next_row = -1;
    auto fetch = [&](unsigned item) {
        const int t = (int)(item / (unsigned)pieces), piece = (int)(item % (unsigned)pieces);
        const int ch = piece * 1024 + lane * 16, col = piece * 32 * U + lane;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            next[u] = make_int4(0, 0, 0, 0);
            if (item >= items) continue;
            if constexpr (kQuant) {
                const int at = ch + (u >> 1) * 512;
                if (at < H) next[u] = ld_stream(reinterpret_cast<const int4*>(reinterpret_cast<const char*>(a.x) + ((size_t)t * H + at) * 2) + (u & 1));
            } else {
                if (col + u * 32 < n16) next[u] = ld_stream(reinterpret_cast<const int4*>(reinterpret_cast<const char*>(a.x) + (size_t)t * out_row_bytes) + col + u * 32);
            }
        }
        next_row = item < items ? a.send_head[t] : -1;
    };
    unsigned item = blockIdx.x * kLoneWarps + (threadIdx.x >> 5);
    fetch(item);
    for (; item < items; item += step) {
        const int t = (int)(item / (unsigned)pieces), piece = (int)(item % (unsigned)pieces);
        const int ch = piece * 1024 + lane * 16;  // casting: 16 channels here and 16 in the other half of the piece
        const int col = piece * 32 * U + lane;    // copying
        int4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = next[u];
        int row = next_row;
        if constexpr (kQuant) fetch(item + step);  // (copying, a warp has one piece)
        if (row >= 0 && !peer_range_ok(c, 0, out + (size_t)row * out_row_bytes, out_row_bytes, 1)) row = -1;
        if (row >= 0) {
            char* dst = out + (size_t)row * out_row_bytes;
            if constexpr (kQuant) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int at = ch + h * 512;
                    const int4 r0 = v[2 * h], r1 = v[2 * h + 1];
                    const uint32_t w[8] = {(uint32_t)r0.x, (uint32_t)r0.y, (uint32_t)r0.z, (uint32_t)r0.w,
                                           (uint32_t)r1.x, (uint32_t)r1.y, (uint32_t)r1.z, (uint32_t)r1.w};
                    float f[16];
                    float amax = 0.f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float2 p = bf16x2_to_f2(w[j]);
                        f[2 * j] = p.x;
                        f[2 * j + 1] = p.y;
                        amax = fmaxf(amax, fmaxf(fabsf(p.x), fabsf(p.y)));
                    }
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
                    float scale, inv;
                    fp8_scale_from_amax(amax, a.round_scale != 0, scale, inv);
                    int4 q;
                    q.x = (int)pack_e4m3x4(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv);
                    q.y = (int)pack_e4m3x4(f[4] * inv, f[5] * inv, f[6] * inv, f[7] * inv);
                    q.z = (int)pack_e4m3x4(f[8] * inv, f[9] * inv, f[10] * inv, f[11] * inv);
                    q.w = (int)pack_e4m3x4(f[12] * inv, f[13] * inv, f[14] * inv, f[15] * inv);
                    if (at < H) {
                        st_stream(reinterpret_cast<int4*>(dst + at), q);
                        if ((lane & 7) == 0) scales[(size_t)row * (H / 128) + (at >> 7)] = scale;
                    }
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (col + u * 32 < n16) st_stream(reinterpret_cast<int4*>(dst) + col + u * 32, v[u]);
                if (a.x_scales != nullptr && piece == 0)
                    for (int i = lane; i < H / 128; i += 32) scales[(size_t)row * (H / 128) + i] = a.x_scales[(size_t)t * (H / 128) + i];
            }
            if (piece == 0) {
                if (a.topk_idx != nullptr && lane < K) {
                    const int64_t e = a.topk_idx[(size_t)t * K + lane];
                    const bool mine = e >= 0 && e < a.num_experts;
                    c.at<int64_t>(0, a.recv_topk_idx_off)[(size_t)row * K + lane] = mine ? e : -1;
                    if (a.topk_weights != nullptr) c.at<float>(0, a.recv_topk_w_off)[(size_t)row * K + lane] = mine ? a.topk_weights[(size_t)t * K + lane] : 0.f;
                }
                if (lane == 0 && a.recv_src_idx_off != kNoOffset) c.at<int>(0, a.recv_src_idx_off)[row] = t;
            }
        }
    }
    if (a.num_worst_tokens > 0 && a.topk_idx != nullptr) {  // see dispatch_kernel
        const int num_recv = a.rank_prefix_matrix[0];
        int64_t* mine = c.at<int64_t>(0, a.recv_topk_idx_off);
        const size_t lo = (size_t)num_recv * K, hi = (size_t)a.num_worst_tokens * K;
        for (size_t i = lo + (size_t)blockIdx.x * kLoneThreads + threadIdx.x; i < hi; i += (size_t)gridDim.x * kLoneThreads) mine[i] = -1;
    }
}

// Whether the call is a lone rank's that nobody asked to leave SMs to something else.
template <typename Args>
bool lone_and_unbounded(const Args* a, int nv) { return nv == 1 && a->ctx.num_ranks == 1 && a->num_sms >= 148; }

cudaError_t launch_dispatch(const DispatchArgs* a, int nv, cudaStream_t stream) {
    if (lone_and_unbounded(a, nv)) {
        const bool quant = a->quantize != 0;
        const int pieces = quant ? (a->hidden + 1023) / 1024 : (a->hidden * a->x_elem_bytes / 16 + 255) / 256;
        const long long ids = (long long)a->num_worst_tokens * (a->topk_idx != nullptr ? a->num_topk : 0);
        const long long moving = ((long long)a->num_tokens * std::max(pieces, 1) + kLoneWarps - 1) / kLoneWarps;
        const long long marking = std::min<long long>((ids + 8 * kLoneThreads - 1) / (8 * kLoneThreads), 4 * 148);
        const unsigned ctas = (unsigned)std::max<long long>(1, std::max(quant ? std::min<long long>(moving, 148 * 4) : moving, marking));
        return quant ? launch_dependent(dispatch_lone_kernel<true>, dim3(ctas), kLoneThreads, 0, stream, *a, std::max(pieces, 1))
                     : launch_dependent(dispatch_lone_kernel<false>, dim3(ctas), kLoneThreads, 0, stream, *a, std::max(pieces, 1));
    }
    // few tokens with outputs for many rows: enough CTAs that no thread marks more than eight unused ids
    const long long ids = (long long)a[0].num_worst_tokens * (a[0].topk_idx != nullptr ? a[0].num_topk : 0);
    const long long marking = (ids + 8 * kDispatchThreads - 1) / (8 * kDispatchThreads);
    const int ctas = (int)std::max<long long>(grid_ctas(a, nv), std::min<long long>(marking, a[0].num_sms));
    return DX_LAUNCH_RANKED_PDL(dispatch_kernel, DispatchArgs, a, nv, ctas, kDispatchThreads, 0, stream);
}

// =============================================================================================
// combine (pull)
// =============================================================================================
constexpr int kCombineThreads = 512;
constexpr int kCombineWarps = kCombineThreads / 32;

struct PeerSrc {
    const int4* x;
    const float* w;
    int base_row;
};

template <int kRanks>
__device__ __forceinline__ void combine_rows(const CombineArgs& a, const PeerSrc* s_src, int warp, int lane, int R) {
    const int T = a.num_tokens, H = a.hidden, K = a.num_topk;
    const int n16 = H / 8;
    const int pieces = row_pieces(T, n16, gridDim.x * kCombineWarps);
    const int per = (((n16 + pieces - 1) / pieces) + 31) & ~31;
    // columns per lane and pass: about sixteen 16-byte loads in flight whatever the number of ranks (eight with one rank, where
    // two biases may come on top)
    constexpr int U = kRanks == 1 ? 8 : (kRanks == 2 ? 4 : 2);
    for (int item = blockIdx.x + gridDim.x * warp; item < T * pieces; item += gridDim.x * kCombineWarps) {
        const int t = item / pieces, piece = item % pieces;
        int head = (lane < R) ? a.send_head[(size_t)t * R + lane] : -1;
        const int4* rowp[kRanks];
        const float* wp[kRanks];
#pragma unroll
        for (int r = 0; r < kRanks; ++r) {
            const int h = __shfl_sync(0xffffffffu, head, r);
            const bool ok = r < R && h >= 0;
            rowp[r] = ok ? s_src[r].x + (size_t)(s_src[r].base_row + h) * n16 : nullptr;
            if (a.ctx.debug_extent != 0 && ok && !peer_range_ok(a.ctx, r, rowp[r], (size_t)n16 * 16, 2)) rowp[r] = nullptr;
            wp[r] = (ok && rowp[r] != nullptr && s_src[r].w != nullptr) ? s_src[r].w + (size_t)(s_src[r].base_row + h) * K : nullptr;
        }
        const int4* bias[2] = {a.bias0 ? reinterpret_cast<const int4*>(a.bias0) + (size_t)t * n16 : nullptr,
                               a.bias1 ? reinterpret_cast<const int4*>(a.bias1) + (size_t)t * n16 : nullptr};
        int4* out = reinterpret_cast<int4*>(a.out) + (size_t)t * n16;
        const int end = min(n16, (piece + 1) * per);
        for (int i0 = piece * per; i0 < end; i0 += 32 * U) {
            int4 v[kRanks][U];
#pragma unroll
            for (int r = 0; r < kRanks; ++r) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u * 32 + lane;
                    v[r][u] = (rowp[r] != nullptr && i < end) ? ld_peer(rowp[r] + i) : make_int4(0, 0, 0, 0);
                }
            }
            // the first bias is requested together with the rows
            int4 bv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * 32 + lane;
                bv[u] = (bias[0] != nullptr && i < end) ? ld_stream(bias[0] + i) : make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * 32 + lane;
                if (i >= end) continue;
                float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                auto add = [&](const int4& x) {
                    const uint32_t w[4] = {(uint32_t)x.x, (uint32_t)x.y, (uint32_t)x.z, (uint32_t)x.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 p = bf16x2_to_f2(w[j]);
                        acc[2 * j] += p.x;
                        acc[2 * j + 1] += p.y;
                    }
                };
#pragma unroll
                for (int r = 0; r < kRanks; ++r) add(v[r][u]);
                if (bias[0] != nullptr) add(bv[u]);
                if (bias[1] != nullptr) add(ld_cached(bias[1] + i));
                int4 o;
                o.x = (int)f2_to_bf16x2(acc[0], acc[1]);
                o.y = (int)f2_to_bf16x2(acc[2], acc[3]);
                o.z = (int)f2_to_bf16x2(acc[4], acc[5]);
                o.w = (int)f2_to_bf16x2(acc[6], acc[7]);
                st_stream(out + i, o);
            }
        }
        if (a.out_topk_w != nullptr && piece == 0 && lane < K) {
            float sum = 0.f;
#pragma unroll
            for (int r = 0; r < kRanks; ++r)
                if (wp[r] != nullptr) sum += __int_as_float(ld_relaxed_sys(reinterpret_cast<const int*>(wp[r] + lane)));
            a.out_topk_w[(size_t)t * K + lane] = sum;
        }
    }
}

template <int V>
__global__ void __launch_bounds__(kCombineThreads, 1) combine_kernel(const __grid_constant__ ArgPack<CombineArgs, V> pack) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const CombineArgs& a = pack.a[blockIdx.y];
    const RankCtx& c = a.ctx;
    const int R = c.num_ranks, me = c.rank;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t seq = next_seq(c, kFamCombine);
    __shared__ PeerSrc s_src[kMaxRanks];
    __shared__ int s_ok;
    if (tid == 0) s_ok = 1;
    __syncthreads();
    // "my expert outputs are final and live at this offset" -> every other home rank
    if (blockIdx.x == 0 && tid < R && tid != me) {
        uint64_t w[2] = {a.x_off, a.topk_w_off};
        mailbox_post(c, kMbCombineSrc, tid, w, 2, seq);
    }
    if (tid < R) {
        uint64_t w[2] = {a.x_off, a.topk_w_off};
        if (tid != me && !mailbox_wait(c, kMbCombineSrc, tid, seq, w, 2)) {
            report(c.status, kTimeoutCombineReady, me, tid, 0);
            s_ok = 0;
        } else {
            PeerSrc p;
            p.x = c.at<const int4>(tid, w[0]);
            p.w = (w[1] == ~0ull) ? nullptr : c.at<const float>(tid, w[1]);
            p.base_row = me > 0 ? a.rank_prefix_matrix[(me - 1) * R + tid] : 0;
            s_src[tid] = p;
        }
    }
    __syncthreads();
    if (!s_ok) return;

    if (R <= 1) combine_rows<1>(a, s_src, warp, lane, R);
    else if (R <= 2) combine_rows<2>(a, s_src, warp, lane, R);
    else if (R <= 4) combine_rows<4>(a, s_src, warp, lane, R);
    else combine_rows<8>(a, s_src, warp, lane, R);

    // Peers may reuse their expert-output buffers only after every home rank has finished reading. (A lone rank: see dispatch.)
    if (R == 1) return;
    if (cta_is_last(c.local_scratch + kTicketCombine, gridDim.x)) {
        if (tid < R && tid != me) st_release_sys(&c.ctrl(tid)->barrier_in[kBarCombine][me], seq);
        if (tid == 0) commit_seq(c, kFamCombine, seq);
    }
    if (blockIdx.x == 0 && tid < R && tid != me) {
        if (!wait_ge_sys(&c.my_ctrl()->barrier_in[kBarCombine][tid], seq, c.timeout_cycles))
            report(c.status, kTimeoutBarrier, me, tid, 200);
    }
}

// The lone rank's form, as in dispatch: a warp takes 256 sixteen-byte columns of a row, or 128 where biases come on top, and has all of
// its loads in flight.
template <int kBiases>
constexpr int kCombineLoneLoads = kBiases == 0 ? 8 : 4;

template <int kBiases>
__global__ void __launch_bounds__(kLoneThreads, kBiases == 2 ? 3 : 4) combine_lone_kernel(const __grid_constant__ CombineArgs a, const int pieces) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const RankCtx& c = a.ctx;
    const int T = a.num_tokens, K = a.num_topk, n16 = a.hidden / 8;
    const int lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * kLoneWarps + (threadIdx.x >> 5);
    if (item >= (long long)T * pieces) return;
    const int t = (int)(item / pieces), piece = (int)(item % pieces);
    constexpr int U = kCombineLoneLoads<kBiases>;
    const int col = piece * 32 * U + lane;
    const int4* bias[2] = {reinterpret_cast<const int4*>(a.bias0 != nullptr ? a.bias0 : a.bias1) + (size_t)t * n16,
                           reinterpret_cast<const int4*>(a.bias1) + (size_t)t * n16};
    int4 v[1 + kBiases][U];
#pragma unroll
    for (int b = 0; b < kBiases; ++b)
#pragma unroll
        for (int u = 0; u < U; ++u) v[1 + b][u] = col + u * 32 < n16 ? ld_stream(bias[b] + col + u * 32) : make_int4(0, 0, 0, 0);
    const int head = a.send_head[t];
    const int4* row = head >= 0 ? c.at<const int4>(0, a.x_off) + (size_t)head * n16 : nullptr;
    if (row != nullptr && !peer_range_ok(c, 0, row, (size_t)n16 * 16, 2)) row = nullptr;
#pragma unroll
    for (int u = 0; u < U; ++u) v[0][u] = row != nullptr && col + u * 32 < n16 ? ld_stream(row + col + u * 32) : make_int4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (col + u * 32 >= n16) continue;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int b = 0; b <= kBiases; ++b) {
            const uint32_t w[4] = {(uint32_t)v[b][u].x, (uint32_t)v[b][u].y, (uint32_t)v[b][u].z, (uint32_t)v[b][u].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 p = bf16x2_to_f2(w[j]);
                acc[2 * j] += p.x;
                acc[2 * j + 1] += p.y;
            }
        }
        int4 o;
        o.x = (int)f2_to_bf16x2(acc[0], acc[1]);
        o.y = (int)f2_to_bf16x2(acc[2], acc[3]);
        o.z = (int)f2_to_bf16x2(acc[4], acc[5]);
        o.w = (int)f2_to_bf16x2(acc[6], acc[7]);
        st_stream(reinterpret_cast<int4*>(a.out) + (size_t)t * n16 + col + u * 32, o);
    }
    if (a.out_topk_w != nullptr && piece == 0 && lane < K)
        a.out_topk_w[(size_t)t * K + lane] = row != nullptr && a.topk_w_off != ~0ull ? 0.f + c.at<const float>(0, a.topk_w_off)[(size_t)head * K + lane] : 0.f;
}

template <int kBiases>
cudaError_t launch_combine_lone(const CombineArgs& a, cudaStream_t stream) {
    const int span = 32 * kCombineLoneLoads<kBiases>, pieces = std::max((a.hidden / 8 + span - 1) / span, 1);
    const long long ctas = ((long long)a.num_tokens * pieces + kLoneWarps - 1) / kLoneWarps;
    if (ctas == 0) return cudaSuccess;
    return launch_dependent(combine_lone_kernel<kBiases>, dim3((unsigned)ctas), kLoneThreads, 0, stream, a, pieces);
}

cudaError_t launch_combine(const CombineArgs* a, int nv, cudaStream_t stream) {
    if (lone_and_unbounded(a, nv)) {
        const int biases = (a->bias0 != nullptr ? 1 : 0) + (a->bias1 != nullptr ? 1 : 0);
        return biases == 0 ? launch_combine_lone<0>(*a, stream) : biases == 1 ? launch_combine_lone<1>(*a, stream) : launch_combine_lone<2>(*a, stream);
    }
    return DX_LAUNCH_RANKED_PDL(combine_kernel, CombineArgs, a, nv, grid_ctas(a, nv), kCombineThreads, 0, stream);
}

// =============================================================================================
// barrier / timeout probe
// =============================================================================================
template <int V>
__global__ void __launch_bounds__(32, 1) barrier_kernel(const __grid_constant__ ArgPack<BarrierArgs, V> pack) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const BarrierArgs& a = pack.a[blockIdx.y];
    const uint64_t seq = next_seq(a.ctx, kFamBarrier);
    cta_rank_barrier(a.ctx, seq);
    if (threadIdx.x == 0) commit_seq(a.ctx, kFamBarrier, seq);
}

cudaError_t launch_barrier(const BarrierArgs* a, int nv, cudaStream_t stream) {
    return DX_LAUNCH_RANKED_PDL(barrier_kernel, BarrierArgs, a, nv, 1, 32, 0, stream);
}

__global__ void timeout_probe_kernel(const RankCtx c, uint64_t* flag) {
    if (!wait_ge_sys(flag, 1, c.timeout_cycles)) report(c.status, kTimeoutTest, c.rank, -1, 0);
}

cudaError_t launch_timeout_probe(const RankCtx& ctx, uint64_t* never_set_flag, cudaStream_t stream) {
    timeout_probe_kernel<<<1, 1, 0, stream>>>(ctx, never_set_flag);
    return cudaGetLastError();
}

}  // namespace dx
