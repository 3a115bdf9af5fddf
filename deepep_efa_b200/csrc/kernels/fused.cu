// Expert-major dispatch for the fused MoE layer: rows land at the receiver already grouped by expert, 128-row
// aligned, in the order the grouped GEMM consumes them, and the GEMM starts on an expert as soon as its rows are in.
//
//   em_notify   every rank lists its selections per GLOBAL expert (a CTA votes over all of them for its share of the experts;
//               rows of an expert keep token order), all-gathers the E counts (+ the offsets of its receive buffers) with one
//               release flag per peer, and derives from the R x E matrix everything the layer needs without a host round trip:
//               where each of its (token, expert) rows goes, the group offsets of its own experts, and how many rows
//               each of its experts will receive (added to a monotonic expectation that the GEMM compares with the
//               arrival counter).
//   em_dispatch a warp takes a unit of up to 8 rows of one expert, quantises each BF16 row to e4m3 (one scale per 128
//               channels, as fp32 or as the UE8M0 words of the tensor core's scale atoms; or copies rows that were quantised
//               once per token beforehand, which is what the overlapped layer does), stores it at its final row
//               of the expert's rank, and bumps that expert's arrival counter with one release reduction. Units are
//               issued expert-major (local expert index first, then destination rank), so on every rank expert 0
//               completes first and the GEMM's group order equals the arrival order.
//   stage_reduce the home rank's sum_k w[t,k] * stage[t,k] after the second GEMM scattered its output rows into the
//               stage (grouped_gemm.cu, scatter epilogue).
// The kernels never wait on each other except for the count exchange (bounded, reports through the status word).
//
// The reference dispatches rank-major through ring queues (csrc/kernels/intranode.cu:197-610) and leaves the
// expert-major permutation to its users; it has no counterpart of the arrival gating.
#include "api.h"
#include "launch.cuh"
#include "prims.cuh"
#include "row_reduce.cuh"
#include "select_scan.cuh"

namespace dx {

constexpr int kEmNotifyThreads = kScanThreads;
constexpr int kEmNotifyWarps = kEmNotifyThreads / 32;
constexpr int kTicketFused = 5;

__device__ __forceinline__ int align128(int v) { return (v + 127) & ~127; }

// Experts of one CTA: as few as the SMs allow (a CTA scans all selections whatever their number, see select_scan.cuh). 256 experts,
// 4096 x 8 selections on one B200: 104 us with one warp per expert and the ids staged in shared memory, 14 us this way. A lone rank's kernel as a whole, with the
// cast's end in front of it, 21.8 -> 18 us (16 tokens 13.8 -> 12.2) by the votes' order (there), by the units' prefix beside the rows' and without trips to its own control words.
__host__ __device__ constexpr int em_experts_per_cta(int num_experts, int ctas) { return (num_experts + ctas - 1) / ctas; }

template <int V>
__global__ void __launch_bounds__(kEmNotifyThreads, 1) em_notify_kernel(const __grid_constant__ ArgPack<EmNotifyArgs, V> pack) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const EmNotifyArgs& a = pack.a[blockIdx.y];
    const RankCtx& c = a.ctx;
    const int R = c.num_ranks, me = c.rank, T = a.num_tokens, K = a.num_topk, E = a.num_experts, L = E / R;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t seq = next_seq(c, kFamFused);
    extern __shared__ int s_dyn[];

    // ---- every CTA: the selections of its experts in token order ----
    const int per_cta = em_experts_per_cta(E, gridDim.x);
    const int e0 = blockIdx.x * per_cta, ne = max(0, min(per_cta, E - e0));
    {
        int* s_run = s_dyn;
        uint32_t* s_vote = reinterpret_cast<uint32_t*>(s_dyn + kScanBatch);
        for (int b0 = 0; b0 < ne; b0 += kScanBatch) {
            const int nb = min(kScanBatch, ne - b0);
            scan_selections(a.topk_idx, T * K, E, e0 + b0, nb, s_vote, s_run, a.places != nullptr && e0 + b0 == 0,
                            [&](int j, int n, int i) {
                                if (n < T) a.sel_list[(size_t)(e0 + b0 + j) * T + n] = i;  // an expert is selected at most once per token
                                if (a.places != nullptr) a.places[i] = make_int2(e0 + b0 + j, n);
                            },
                            [&](int i) { a.places[i] = make_int2(-1, 0); });
            for (int j = tid; j < nb; j += kEmNotifyThreads) a.my_counts[e0 + b0 + j] = min(s_run[j], T);
        }
    }

    // ---- the last CTA to finish exchanges the counts and derives the plan ----
    if (!cta_is_last(c.local_scratch + kTicketFused, gridDim.x)) return;
    int* s_cnt = s_dyn;                 // [E] my counts
    int* s_total = s_dyn + E;           // [E] rows every expert receives from all ranks
    int* s_off = s_dyn + 2 * E;         // [E] rows of ranks before me inside every expert
    int* s_base = s_dyn + 3 * E;        // [E] first row of every expert at its own rank
    __shared__ int s_ok;
    __shared__ int s_rank_rows[kMaxRanks];
    if (tid == 0) s_ok = 1;
    for (int i = tid; i < E; i += kEmNotifyThreads) s_cnt[i] = __ldcg(&a.my_counts[i]);
    __syncthreads();
    const int P = (int)(seq & 1);
    for (int d = 0; d < R; ++d) {
        ControlBlock* pc = c.ctrl(d);
        for (int i = tid; i < E; i += kEmNotifyThreads) st_relaxed_sys(&pc->em_counts[P][me][i], s_cnt[i]);
        if (tid < 4) {
            const uint64_t w = tid == 0 ? a.recv_x_off : tid == 1 ? a.recv_scales_off : tid == 2 ? a.recv_info_off : a.stage_off;
            st_relaxed_sys(&pc->em_desc[P][me][tid], w);
        }
    }
    __syncthreads();
    if (tid < R && tid != me) {  // my own words are ordered by the barrier above
        st_release_sys(&c.ctrl(tid)->em_seq[me], seq);
        if (!wait_ge_sys(&c.my_ctrl()->em_seq[tid], seq, c.timeout_cycles)) {
            report(c.status, kTimeoutFusedNotify, me, tid, 0);
            s_ok = 0;
        }
    }
    __syncthreads();
    if (s_ok) {
        ControlBlock* my = c.my_ctrl();
        for (int i = tid; i < E; i += kEmNotifyThreads) {
            int total = 0, before = 0;
            for (int src = 0; src < R; ++src) {
                const int v = src == me ? s_cnt[i] : ld_relaxed_sys(&my->em_counts[P][src][i]);
                total += v;
                if (src < me) before += v;
            }
            s_total[i] = total;
            s_off[i] = before;
        }
        __syncthreads();
        // first row of every expert at its rank: exclusive prefix of the 128-aligned totals, one warp per rank
        for (int d = warp; d < R; d += kEmNotifyWarps) {
            int carry = 0;
            for (int l0 = 0; l0 < L; l0 += 32) {
                const int le = l0 + lane;
                const int v = le < L ? align128(s_total[d * L + le]) : 0;
                const int incl = warp_incl_scan(v);
                if (le < L) s_base[d * L + le] = carry + incl - v;
                carry += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) s_rank_rows[d] = carry;
        }
        // work units of the dispatch kernel, expert-major: order index o = local expert * R + destination rank (by a warp that has no rank's prefix to form)
        if (warp == kEmNotifyWarps - 1) {
            int carry = 0;
            for (int o0 = 0; o0 < E; o0 += 32) {
                const int o = o0 + lane;
                const int ex = o < E ? (o % R) * L + o / R : 0;
                const int v = o < E ? (s_cnt[ex] + a.unit_rows - 1) / a.unit_rows : 0;
                const int incl = warp_incl_scan(v);
                if (o < E) a.unit_start[o] = carry + incl - v;
                carry += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) a.unit_start[E] = carry;
        }
        __syncthreads();
        // Every rank computes the same row totals, so all of them see an overflow of some rank's receive buffer alike: the
        // call then moves no rows at all (no work units, empty groups, expectations unchanged) and reports the error.
        bool overflow = false;
        for (int d = 0; d < R; ++d) overflow = overflow || s_rank_rows[d] > a.rows_cap;
        if (overflow) {
            if (tid == 0) report(c.status, kBadArgument, me, -1, s_rank_rows[me]);
            for (int i = tid; i <= E; i += kEmNotifyThreads) a.unit_start[i] = 0;
            if (tid == 0) *a.unit_counter = 0;
            for (int le = tid; le <= L; le += kEmNotifyThreads) {
                a.m_offsets[le] = 0;
                if (le < L) a.m_ends[le] = 0;
            }
            __syncthreads();
            if (tid == 0) commit_seq(c, kFamFused, seq);
            return;
        }
        for (int i = tid; i < E; i += kEmNotifyThreads) a.send_base[i] = s_base[i] + s_off[i];
        for (int le = tid; le < L; le += kEmNotifyThreads) {
            const int g = me * L + le;
            a.m_offsets[le] = s_base[g];
            a.m_ends[le] = s_base[g] + s_total[g];
            // rows this expert will have received once this call's dispatch is complete (monotonic over the calls). What a lone rank was to receive by now is
            // in place: the kernels of earlier calls are complete, also those that count no arrivals (em_dispatch_lone_kernel).
            const uint64_t expected = c.seq[kFusedExpectedWord0 + le];
            if (R == 1) my->em_arrived[le] = expected;
            c.seq[kFusedExpectedWord0 + le] = expected + (uint64_t)s_total[g];
        }
        if (tid == 0) a.m_offsets[L] = s_rank_rows[me];
        if (tid == 0) *a.unit_counter = 0;
        if (tid < 4 * R) {
            const int which = tid / R, r = tid % R;
            const uint64_t mine = which == 0 ? a.recv_x_off : which == 1 ? a.recv_scales_off : which == 2 ? a.recv_info_off : a.stage_off;
            a.peer_bases[tid] = reinterpret_cast<uint64_t>(c.at<char>(r, r == me ? mine : ld_relaxed_sys(&my->em_desc[P][r][which])));
        }
    }
    if (tid == 0) commit_seq(c, kFamFused, seq);
}

cudaError_t launch_em_notify(const EmNotifyArgs* a, int nv, cudaStream_t stream) {
    const int E = a[0].num_experts;
    if (E < 1 || E > kMaxFusedExperts || E % a[0].ctx.num_ranks != 0 || a[0].unit_rows < 1) return cudaErrorInvalidValue;
    const int fit = nv == 1 ? 148 : 148 / nv - 1;  // emulated ranks must be co-resident
    const int per_cta = em_experts_per_cta(E, E < fit ? E : fit);
    const int ctas = (E + per_cta - 1) / per_cta;
    const size_t scan = scan_smem_bytes(per_cta), plan = (size_t)4 * E * sizeof(int);
    const size_t smem = scan > plan ? scan : plan;
    return DX_LAUNCH_RANKED_PDL(em_notify_kernel, EmNotifyArgs, a, nv, ctas, kEmNotifyThreads, smem, stream);
}

// =============================================================================================
// dispatch
// =============================================================================================
constexpr int kEmDispatchThreads = 128;  // small CTAs with few registers: they share SMs with the persistent GEMM CTAs
constexpr int kEmDispatchWarps = kEmDispatchThreads / 32;

__device__ __forceinline__ unsigned long long global_timer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

template <int V>
__global__ void __launch_bounds__(kEmDispatchThreads, 6) em_dispatch_kernel(const __grid_constant__ ArgPack<EmDispatchArgs, V> pack) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const EmDispatchArgs& a = pack.a[blockIdx.y];
    const RankCtx& c = a.ctx;
    const int R = c.num_ranks, me = c.rank, T = a.num_tokens, K = a.num_topk, E = a.num_experts, L = E / R, H = a.hidden;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    extern __shared__ int s_unit_start[];  // [E+1]
    for (int i = tid; i <= E; i += kEmDispatchThreads) s_unit_start[i] = a.unit_start[i];
    __syncthreads();
    if (a.trace != nullptr && tid == 0) atomicMin(&a.trace[0], global_timer());
    const int total_units = s_unit_start[E];
    const int num_kb = H / 128;
    char* const* rows_base = reinterpret_cast<char* const*>(a.peer_bases);
    char* const* scales_base = reinterpret_cast<char* const*>(a.peer_bases + R);
    int* const* info_base = reinterpret_cast<int* const*>(a.peer_bases + 2 * R);

    // Units are handed out through one counter (reset by the count exchange), so they are taken in order by whichever warps
    // are running: experts complete in order even when only part of the grid is resident next to a GEMM.
    while (true) {
        int u = 0;
        if (lane == 0) u = atomicAdd(a.unit_counter, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= total_units) break;
        int lo = 0, hi = E;  // largest o with unit_start[o] <= u
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_unit_start[mid] <= u) lo = mid;
            else hi = mid;
        }
        const int o = lo, d = o % R, le = o / R, e = d * L + le;
        const int s0 = (u - s_unit_start[o]) * a.unit_rows;
        const int cnt = a.my_counts[e];
        const int n = min(a.unit_rows, cnt - s0);
        const int base_row = a.send_base[e] + s0;
        char* dst_rows = rows_base[d];
        char* dst_scales = scales_base[d];
        int sent = 0;
        for (int s = 0; s < n; ++s) {
            const int sel = a.sel_list[(size_t)e * T + s0 + s];
            const int t = sel / K;
            const int row = base_row + s;
            if (c.debug_extent != 0 && !peer_range_ok(c, d, dst_rows + (size_t)row * H, (size_t)H, 6)) continue;
            char* drow = dst_rows + (size_t)row * H;
            if (a.x_scales != nullptr) {
                // rows quantised beforehand (once per token instead of once per selection): a pure copy, 4 KiB per pass
                const int n16 = H / 16;
                const int4* src16 = reinterpret_cast<const int4*>(reinterpret_cast<const char*>(a.x) + (size_t)t * H);
                for (int i0 = 0; i0 < n16; i0 += 256) {
                    int4 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int i = i0 + u * 32 + lane;
                        if (i < n16) v[u] = ld_cached(src16 + i);
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int i = i0 + u * 32 + lane;
                        if (i < n16) st_stream(reinterpret_cast<int4*>(drow) + i, v[u]);
                    }
                }
                for (int kb = lane; kb < num_kb; kb += 32) {
                    const float scale = a.x_scales[(size_t)t * num_kb + kb];
                    if (a.native_atoms) {
                        const uint32_t ex = (__float_as_uint(scale) >> 23) & 0xffu;
                        *reinterpret_cast<uint32_t*>(dst_scales + ((size_t)(row >> 7) * num_kb + kb) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4) =
                            ex * 0x01010101u;
                    } else {
                        reinterpret_cast<float*>(dst_scales)[(size_t)row * num_kb + kb] = scale;
                    }
                }
                if (lane == 0) {
                    info_base[d][row] = (me << 24) | sel;
                    if (a.dst_row != nullptr) a.dst_row[sel] = row;
                }
                ++sent;
                continue;
            }
            const char* src = reinterpret_cast<const char*>(a.x) + (size_t)t * H * 2;
            // a lane owns 16 consecutive channels, 8 lanes share a scale, a warp covers 512 channels per half step; the loads
            // of the next 1024 channels are issued before the current ones are converted
            int4 cur[4], nxt[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int ch = h * 512 + lane * 16;
                cur[2 * h] = cur[2 * h + 1] = make_int4(0, 0, 0, 0);
                if (ch < H) {
                    cur[2 * h] = ld_cached(reinterpret_cast<const int4*>(src + (size_t)ch * 2));
                    cur[2 * h + 1] = ld_cached(reinterpret_cast<const int4*>(src + (size_t)ch * 2 + 16));
                }
            }
            for (int c0 = 0; c0 < H; c0 += 1024) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int chn = c0 + 1024 + h * 512 + lane * 16;
                    nxt[2 * h] = nxt[2 * h + 1] = make_int4(0, 0, 0, 0);
                    if (chn < H) {
                        nxt[2 * h] = ld_cached(reinterpret_cast<const int4*>(src + (size_t)chn * 2));
                        nxt[2 * h + 1] = ld_cached(reinterpret_cast<const int4*>(src + (size_t)chn * 2 + 16));
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int ch = c0 + h * 512 + lane * 16;
                    const bool act = ch < H;
                    const int4 q0 = cur[2 * h], q1 = cur[2 * h + 1];
                    const uint32_t w[8] = {(uint32_t)q0.x, (uint32_t)q0.y, (uint32_t)q0.z, (uint32_t)q0.w,
                                           (uint32_t)q1.x, (uint32_t)q1.y, (uint32_t)q1.z, (uint32_t)q1.w};
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
                    fp8_scale_from_amax(amax, a.round_scale != 0 || a.native_atoms != 0, scale, inv);
                    int4 q;
                    q.x = (int)pack_e4m3x4(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv);
                    q.y = (int)pack_e4m3x4(f[4] * inv, f[5] * inv, f[6] * inv, f[7] * inv);
                    q.z = (int)pack_e4m3x4(f[8] * inv, f[9] * inv, f[10] * inv, f[11] * inv);
                    q.w = (int)pack_e4m3x4(f[12] * inv, f[13] * inv, f[14] * inv, f[15] * inv);
                    if (act) {
                        st_stream(reinterpret_cast<int4*>(drow + ch), q);
                        if ((lane & 7) == 0) {
                            const int kb = ch >> 7;
                            if (a.native_atoms) {
                                // UE8M0 word of the scale atom of (128-row tile, K block): row m0 + 32*m1 sits at m0*16 + m1*4
                                const uint32_t ex = (__float_as_uint(scale) >> 23) & 0xffu;
                                *reinterpret_cast<uint32_t*>(dst_scales + ((size_t)(row >> 7) * num_kb + kb) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4) =
                                    ex * 0x01010101u;
                            } else {
                                reinterpret_cast<float*>(dst_scales)[(size_t)row * num_kb + kb] = scale;
                            }
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) cur[j] = nxt[j];
            }
            if (lane == 0) {
                info_base[d][row] = (me << 24) | sel;
                if (a.dst_row != nullptr) a.dst_row[sel] = row;
            }
            ++sent;
        }
        __syncwarp();
        // one release per unit: everything this warp stored for expert (d, le) is visible before the counter moves
        if (lane == 0 && sent > 0) {
            // (GPU scope is enough only where nobody else adds to the counter: additions of two scopes to one word are not atomic to each other)
            if (R == 1) red_add_release_gpu(&c.ctrl(d)->em_arrived[le], (uint64_t)sent);
            else red_add_release_sys(&c.ctrl(d)->em_arrived[le], (uint64_t)sent);
        }
    }
    if (a.trace != nullptr) {
        __syncthreads();
        if (tid == 0) atomicMax(&a.trace[1], global_timer());
    }
}

// A lone rank copies its quantised rows within its own memory, so experts need not complete in order: a warp loads a span of a token's row once and stores it to
// all of the token's rows. Expert by expert the rows were read again for each selection, from HBM, since what is written pushes them out of the L2 (rows of
// 52736 x 8 KB written at 3.2 TB/s with reads from 67 MB, at 6.5 without). Behind the exchange, 4096 x 8 rows of 1 KB 38.4 -> 25.3 us, 4096 x 6 27.4 -> 19.0; in a layer
// at the power limit, 4096 x 8 rows of 7 KB 96 -> 55. No CTA knows when an expert's rows are complete, so arrivals are not counted here: nothing on this GPU may
// gate on them (a gate would run into its limit), and the next exchange makes up for it. Counted by the last CTA to finish, with a ticket, the kernel
// itself took 11.4 -> 13.8 us with rows of 1 KB, 46.4 -> 47.8 with 7 KB.
// With more than four places per token four CTAs share an SM instead of six, by shared memory that none of them uses: more write more rows at a time than the memory takes
// well. With fewer places the loads want more of them. Exchange and dispatch, us, CTAs per SM 6 / 5 / 4 (rows x places of a size): 7000 x 2 of 2 KB 18.3 / 19.8 / 20.3, 4096 x 2
// of 7 KB 24.3 / 24.9 / 26.1, 7000 x 4 of 2 KB 26.1 / 26.4 / 27.6; 2000 x 6 of 4 KB 26.2 / 25.4 / 22.9, 4096 x 8 of 1 KB 28.5 / 27.0 / 25.0, of 2 KB 39.8 / 36.7 / 33.0, of 7 KB
// 60.9 / 61.7 / 61.6, 7000 x 8 of 2 KB 40.6 / 40.2 / 40.4.
constexpr int kEmLoneThreads = 256;
constexpr int kEmLoneLoads = 4;
constexpr int kEmLoneSpan = 32 * kEmLoneLoads * 16;  // bytes of a row per warp: 16 of its scales
constexpr int kEmLoneSmem = 46 * 1024;  // of the 228 KB of an SM, 1 KB more per CTA is the system's
inline long long em_lone_ctas(const EmDispatchArgs& a) {
    const long long warps = (long long)a.num_tokens * ((a.hidden + kEmLoneSpan - 1) / kEmLoneSpan);
    return std::max(1ll, (warps + kEmLoneThreads / 32 - 1) / (kEmLoneThreads / 32));
}

__global__ void __launch_bounds__(kEmLoneThreads) em_dispatch_lone_kernel(const __grid_constant__ EmDispatchArgs a) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const int T = a.num_tokens, K = a.num_topk, E = a.num_experts, H = a.hidden;
    const int tid = threadIdx.x, lane = tid & 31;
    const int n16 = H / 16, num_kb = H / 128, spans = (H + kEmLoneSpan - 1) / kEmLoneSpan;
    const long long item = (long long)blockIdx.x * (kEmLoneThreads / 32) + (tid >> 5);
    const int t = (int)(item / spans), span = (int)(item % spans);
    if (t < T && a.unit_start[E] > 0) {  // (no units after an overflow)
        const int i0 = span * (kEmLoneSpan / 16) + lane, kb = span * (kEmLoneSpan / 128) + (lane & 15);
        const int4* src = reinterpret_cast<const int4*>(reinterpret_cast<const char*>(a.x) + (size_t)t * H) + i0;
        int4 v[kEmLoneLoads];
#pragma unroll
        for (int u = 0; u < kEmLoneLoads; ++u)
            if (i0 + u * 32 < n16) v[u] = ld_once(src + u * 32);
        const float scale = kb < num_kb ? a.x_scales[(size_t)t * num_kb + kb] : 0.f;
        int row = -1;
        if (lane < K) {
            const int2 place = a.places[(size_t)t * K + lane];
            if ((unsigned)place.x < (unsigned)E && (unsigned)place.y < (unsigned)a.my_counts[place.x]) row = a.send_base[place.x] + place.y;
        }
        char* rows = reinterpret_cast<char*>(a.peer_bases[0]);
        char* scales = reinterpret_cast<char*>(a.peer_bases[1]);
        for (int k = 0; k < K; ++k) {
            const int dst_row = __shfl_sync(0xffffffffu, row, k);
            if (dst_row < 0) continue;
            int4* dst = reinterpret_cast<int4*>(rows + (size_t)dst_row * H) + i0;
#pragma unroll
            for (int u = 0; u < kEmLoneLoads; ++u)
                if (i0 + u * 32 < n16) st_once(dst + u * 32, v[u]);
        }
        for (int k0 = 0; k0 < K; k0 += 2) {  // two rows' scales at a time
            const int dst_row = __shfl_sync(0xffffffffu, row, (k0 + (lane >> 4)) & 31);
            if (k0 + (lane >> 4) >= K || dst_row < 0 || kb >= num_kb) continue;
            if (a.native_atoms)
                *reinterpret_cast<uint32_t*>(scales + ((size_t)(dst_row >> 7) * num_kb + kb) * 512 + (dst_row & 31) * 16 + ((dst_row >> 5) & 3) * 4) =
                    ((__float_as_uint(scale) >> 23) & 0xffu) * 0x01010101u;
            else reinterpret_cast<float*>(scales)[(size_t)dst_row * num_kb + kb] = scale;
        }
        if (span == 0 && row >= 0) {
            reinterpret_cast<int*>(a.peer_bases[2])[row] = t * K + lane;  // (source rank 0 << 24) | selection
            if (a.dst_row != nullptr) a.dst_row[t * K + lane] = row;
        }
    }
}

cudaError_t launch_em_dispatch(const EmDispatchArgs* a, int nv, cudaStream_t stream) {
    if (a[0].hidden % 128 != 0 || a[0].num_sms < 1) return cudaErrorInvalidValue;
    if (nv == 1 && a->ctx.num_ranks == 1 && a->num_sms >= 148 && a->places != nullptr && a->x_scales != nullptr && a->ctx.debug_extent == 0 && a->trace == nullptr)
        return launch_dependent(em_dispatch_lone_kernel, dim3((unsigned)em_lone_ctas(*a)), kEmLoneThreads, a->num_topk > 4 ? kEmLoneSmem : 0, stream, *a);
    const size_t smem = (size_t)(a[0].num_experts + 1) * sizeof(int);
    return DX_LAUNCH_RANKED_PDL(em_dispatch_kernel, EmDispatchArgs, a, nv, a[0].num_sms, kEmDispatchThreads, smem, stream);
}

// =============================================================================================
// home-side reduction of the scattered expert outputs
// =============================================================================================
// out[t] = sum_k w[t,k] * stage[t*K + k] over the valid selections of token t (fp32 accumulate, fixed k order).
__global__ void __launch_bounds__(kReduceThreads) stage_reduce_kernel(const __nv_bfloat16* __restrict__ stage, __nv_bfloat16* __restrict__ out,
                                                                      const int64_t* __restrict__ topk_idx, const float* __restrict__ w,
                                                                      int num_tokens, int num_topk, int num_experts, int hidden) {
    pdl_wait_predecessor();
    pdl_release_successor();
    const int lane = threadIdx.x & 31;
    const int n16 = hidden / 8, spans = reduce_spans(n16);
    const int item = blockIdx.x * (kReduceThreads / 32) + (threadIdx.x >> 5);
    const int t = item / spans;
    if (t >= num_tokens) return;
    int row = -1;
    float my_w = 0.f;
    if (lane < num_topk) {
        const int64_t e = topk_idx[(size_t)t * num_topk + lane];
        my_w = w[(size_t)t * num_topk + lane];
        if (e >= 0 && e < num_experts) row = t * num_topk + lane;
    }
    reduce_row_span(reinterpret_cast<const int4*>(stage), reinterpret_cast<int4*>(out) + (size_t)t * n16, n16, item % spans, num_topk, row, my_w, lane);
}

cudaError_t launch_stage_reduce(const void* stage, void* out, const int64_t* topk_idx, const float* w, int num_tokens, int num_topk,
                                int num_experts, int hidden, cudaStream_t stream) {
    if (num_tokens <= 0) return cudaSuccess;
    if (hidden % 8 != 0 || num_topk < 1 || num_topk > 32) return cudaErrorInvalidValue;
    if (hidden == 0) return cudaSuccess;
    return launch_dependent(stage_reduce_kernel, dim3(reduce_ctas(num_tokens, hidden / 8)), kReduceThreads, 0, stream, static_cast<const __nv_bfloat16*>(stage),
                            static_cast<__nv_bfloat16*>(out), topk_idx, w, num_tokens, num_topk, num_experts, hidden);
}

}  // namespace dx
