// Grouped expert GEMM in BF16 on CTA pairs (cta_group::2) with the weights as the M operand and the tokens as the N operand:
//
//   C[m, n] = sum_k A[m, k] * B[g][n, k]     (forward: B is [G, N, K])
//   C[m, n] = sum_k A[m, k] * B[g][k, n]     (input gradient: B is the forward weight [G, K, N], read in place as an MN-major operand)
//
// Why the operands change places. At these sizes the products bound the time, and inside a training step the power limit bounds the products: a
// tile of 256 token rows multiplies whatever lies behind a group's end, and with 832 padded rows per expert (13/4 tiles) a fifth of the products
// was for nothing. The columns of an MMA come in steps of 32, so a group's rows are cut into equal tiles of at most `token_cap` of them with
// at most 31 too many. Both forward products and both input gradients of a layer in a loop, us, rows / columns: 64 experts of 4096 -> 1408 with 130 rows
// each 1019 / 885, 160 rows 1087 / 957, 290 rows 1687 / 1496, 384 rows 1808 / 1659, 768 rows 2978 / 2888, skewed 3166 / 3014; 60 of 2304 -> 640, 260 rows 434 / 379.
// Where nothing was multiplied in vain before, nothing is gained: 8 experts of 4096 -> 1408, 3000 rows 1286 / 1289.
//
//   warp 0      TMA producer   each CTA: its own 128 features and its own half of the tile's tokens (no multicast), signalling the leader
//   warp 1      MMA issuer     leader CTA: M = 256 features, N = the tile's tokens; two accumulator windows
//   warps 2..9  epilogue       lane = feature, column = token; two warps per TMEM lane quarter take alternate units of 32 tokens, turn them
//                              over in shared memory and store rows of 64 bytes (four warps with a TMA store per unit, two in
//                              flight, were slower wherever K is short: 32 experts of 1024 -> 1024, 250 rows 178 us instead of 156)
//
// The issuer's loop is one elected thread from end to end: with an election per K block an MMA cost 73 cycles to issue instead of 37, because its
// operands then pass through ordinary registers (four MMAs and a commit: 451 and 300 cycles).
//
// Every wait is bounded, as in grouped_gemm.cu.
#include <algorithm>
#include <cstring>

#include "launch.cuh"
#include "tc_prims.cuh"

namespace dx {

namespace {

constexpr int kPairEpiWarps = 8;
constexpr int kPairThreads = 64 + 32 * kPairEpiWarps;
constexpr int kPairMaxStages = 8;
constexpr int kPairWindowCols = 256;
constexpr int kUnit = 32;                            // step of the N operand of a pair
constexpr int kBlockBytes = kUnit * 32 * 2;          // 32 tokens x 32 features, BF16
constexpr int kPairMaxSmem = 232448 - 512;

struct PairMaps {
    CUtensorMap w;     // 128 features x one K block
    CUtensorMap t[4];  // boxes of 128, 64, 32 and 16 token rows
};

struct PairTile {
    int group, ft, row, cols, valid;  // cols: columns of the MMA; valid: rows that may be stored
    int tail, tail_end;               // rows of the group's padding that this tile clears
};

__host__ __device__ constexpr int pair_stage_bytes(int cap) { return kATileBytes + cap / 2 * kKBlockBytes; }

template <bool kMn>
__global__ void __launch_bounds__(kPairThreads, 1)
token_pairs_gemm_kernel(const __grid_constant__ PairMaps maps, const GroupedGemmArgs p, const int stages) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* stage_base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t cta_rank = cluster_ctarank();  // 0 = leader
    const int cap = p.token_cap, stage_bytes = pair_stage_bytes(cap), G = p.num_groups;
    uint8_t* out_base = stage_base + (size_t)stages * stage_bytes;           // a block per epilogue warp
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_base + kPairEpiWarps * kBlockBytes);
    uint64_t* full = bars;
    uint64_t* empty = bars + kPairMaxStages;
    uint64_t* tmem_full = bars + 2 * kPairMaxStages;
    uint64_t* tmem_empty = tmem_full + 2;
    int* tile_start = reinterpret_cast<int*>(bars + 32);  // [G+1]
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_kb = p.k / 64;
    const int feature_tiles = (p.n + 255) / 256;
    const int sched_id = (int)(blockIdx.x >> 1), sched_stride = (int)(gridDim.x >> 1);

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int w = 0; w < 2; ++w) {
            mbar_init(&tmem_full[w], 1);
            mbar_init(&tmem_empty[w], 2 * kPairEpiWarps);  // the leader collects both CTAs' epilogue warps
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tma_prefetch_desc(&maps.w);
        for (int i = 0; i < 4; ++i) tma_prefetch_desc(&maps.t[i]);
    }
    if (warp == 1) tmem_alloc_pair(&s_tmem_base, 2 * kPairWindowCols);
    cluster_sync_all();  // the peer's barriers exist before anything signals them
    pdl_wait_predecessor();
    pdl_release_successor();
    // A group's rows in units of 32, cut into tiles of at most token_cap of them that differ by a unit at most. A group that has no rows but
    // padding to clear is one tile without products.
    auto padding = [&](int g, int begin, int rows) { return p.zero_tail ? max(p.m_offsets[g + 1] - begin - rows, 0) : 0; };
    auto row_tiles = [&](int g, int begin, int rows) {
        if (rows <= 0) return padding(g, begin, 0) > 0 ? 1 : 0;
        const int units = (rows + kUnit - 1) / kUnit, most = cap / kUnit;
        return (units + most - 1) / most;
    };
    if (warp == 2) {
        build_tile_table(p, tile_start, lane, [&](int g, int begin, int rows) { return row_tiles(g, begin, rows) * feature_tiles; });
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    const int total_tiles = tile_start[G];
    volatile int* abort_flag = &s_abort;
    const long long limit = p.timeout_cycles;

    auto decode = [&](int tile, int& g, PairTile& t) {
        while (tile >= tile_start[g + 1]) ++g;
        const int local = tile - tile_start[g];
        const int m0 = p.m_offsets[g], rows = group_rows(p, g, m0), tiles_m = row_tiles(g, m0, rows);
        const int mt = local % tiles_m;  // consecutive tiles share the weights
        const int units = (rows + kUnit - 1) / kUnit;
        const int u0 = (int)((long long)units * mt / tiles_m), u1 = (int)((long long)units * (mt + 1) / tiles_m);
        t.group = g;
        t.ft = local / tiles_m;
        t.row = m0 + u0 * kUnit;
        t.cols = (u1 - u0) * kUnit;
        t.valid = max(min(rows - u0 * kUnit, t.cols), 0);
        t.valid = min(t.valid, p.m_total - t.row);
        t.tail = t.tail_end = 0;
        if (p.zero_tail && mt == tiles_m - 1) {
            t.tail_end = min(p.m_offsets[g + 1], p.m_total);
            t.valid = min(t.cols, t.tail_end - t.row);  // rows between the group's end and the next unit hold zeros
            t.tail = m0 + units * kUnit;
        }
    };

    if (warp == 0) {
        // ================= TMA producer =================
        int stage = 0, phase = 0, g = 0, issued = 0;
        bool ok = true;
        PairTile t;
        const uint32_t stage_u32 = smem_u32(stage_base), full_leader = mapa_shared(smem_u32(full), 0);
        for (int tile = sched_id; tile < total_tiles && ok; tile += sched_stride) {
            decode(tile, g, t);
            if (t.cols == 0) continue;
            const int half = t.cols / 2, row = t.row + (int)cta_rank * half;
            const int feature = t.ft * 256 + (int)cta_rank * 128;
            const uint32_t tx = 2u * (kATileBytes + half * kKBlockBytes);
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1, abort_flag, limit))) {
                    ok = false;
                    break;
                }
                if (elect_one()) {
                    const uint32_t bar = full_leader + stage * 8, sw = stage_u32 + stage * stage_bytes;
                    if (cta_rank == 0) mbar_expect_tx(&full[stage], tx);  // of both CTAs
                    if constexpr (kMn) tma_load_3d_pair_at(&maps.w, bar, sw, 0, g * p.k + kb * 64, feature / 64);
                    else tma_load_2d_pair_at(&maps.w, bar, sw, kb * 64, g * p.n + feature);
                    uint32_t st = sw + kATileBytes;
                    int r = row;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (half & (128 >> i)) {
                            tma_load_2d_pair_at(&maps.t[i], bar, st, kb * 64, r);
                            st += (128 >> i) * kKBlockBytes;
                            r += 128 >> i;
                        }
                    }
                }
                __syncwarp();
                if (issued < stages) ++issued;
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        // copies in flight land in this CTA's shared memory (see grouped_gemm.cu)
        if (!ok) {
            if (cta_rank == 1) {
                const long long t0 = clock64();
                while (clock64() - t0 < 400000) {
                }
            } else {
                int s = stage, ph = phase;
                for (int i = 0; i < stages && i < issued; ++i) {
                    if (--s < 0) {
                        s = stages - 1;
                        ph ^= 1;
                    }
                    const long long t0 = clock64();
                    while (!mbar_try_wait(&full[s], ph) && clock64() - t0 < limit) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        if (cta_rank == 0 && elect_one()) {
            int stage = 0, phase = 0, g = 0, win = 0, win_phase = 0;
            bool ok = true;
            PairTile t;
            const uint32_t stage_u32 = smem_u32(stage_base);
            const uint32_t empty_own = smem_u32(empty), empty_peer = mapa_shared(empty_own, 1);
            const uint32_t tf_own = smem_u32(tmem_full), tf_peer = mapa_shared(tf_own, 1);
            constexpr uint64_t kWStep = kMn ? 128 : 2;  // 16 K-steps of the features' operand, in 16-byte units
            for (int tile = sched_id; tile < total_tiles && ok; tile += sched_stride) {
                decode(tile, g, t);
                if (t.cols == 0) continue;
                const uint32_t idesc = make_idesc<false>(t.cols, 256, kMn ? 1 : 0, 0);
                if (!mbar_wait(&tmem_empty[win], win_phase ^ 1, abort_flag, limit)) break;
                const uint32_t tmem_d = tmem_base + (uint32_t)(win * kPairWindowCols);
                for (int kb = 0; kb < num_kb; ++kb) {
                    if (!mbar_wait(&full[stage], phase, abort_flag, limit)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sw = stage_u32 + (uint32_t)(stage * stage_bytes);
                    const uint64_t wdesc = kMn ? make_smem_desc_mn(sw) : make_smem_desc(sw), tdesc = make_smem_desc(sw + kATileBytes);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        umma_pair<false>(tmem_d, wdesc + (uint64_t)j * kWStep, tdesc + (uint64_t)(j * 2), idesc, (kb == 0 && j == 0) ? 0u : 1u);
                    umma_commit_pair(empty_own + stage * 8);
                    umma_commit_pair(empty_peer + stage * 8);
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                umma_commit_pair(tf_own + win * 8);
                umma_commit_pair(tf_peer + win * 8);
                win ^= 1;
                if (win == 0) win_phase ^= 1;
            }
        }
        __syncwarp();
    } else {
        // ================= epilogue =================
        const int q = warp & 3, half = (warp - 2) >> 2;
        uint32_t* block = reinterpret_cast<uint32_t*>(out_base + (warp - 2) * kBlockBytes);
        int g = 0, win = 0, win_phase = 0;
        bool ok = true;
        PairTile t;
        for (int tile = sched_id; tile < total_tiles && ok; tile += sched_stride) {
            decode(tile, g, t);
            const int col = t.ft * 256 + (int)cta_rank * 128 + q * 32;  // first of this warp's 32 features
            const bool mine = col < p.n;                                 // an odd count of 128 features ends in half a tile
            // lane l stores 16 bytes of the rows l / 4, l / 4 + 8, ... of a unit
            __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.c) + (size_t)(t.row + (lane >> 2)) * p.n + col + (lane & 3) * 8;
            if (t.cols > 0) {
                if (!mbar_wait(&tmem_full[win], win_phase, abort_flag, limit)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(win * kPairWindowCols);
                if (mine) {
                    for (int t0 = half * kUnit; t0 < t.valid; t0 += 2 * kUnit) {
                        uint32_t v[32];
                        tmem_ld32(taddr + t0, v);
                        tmem_ld_wait();
                        // lanes 2i and 2i + 1 exchange halves: the even one gets token 2j of both features, the odd one token 2j + 1
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const uint32_t w = f2_to_bf16x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                            const uint32_t o = __shfl_xor_sync(0xffffffffu, w, 1);
                            block[(2 * j + (lane & 1)) * 16 + (lane >> 1)] = __byte_perm(w, o, (lane & 1) ? 0x3276 : 0x5410);
                        }
                        __syncwarp();
                        int4 piece[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) piece[i] = *reinterpret_cast<const int4*>(block + (i * 8 + (lane >> 2)) * 16 + (lane & 3) * 4);
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (t0 + i * 8 + (lane >> 2) < t.valid) *reinterpret_cast<int4*>(out + (size_t)(t0 + i * 8) * p.n) = piece[i];
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (cta_rank == 0) mbar_arrive(&tmem_empty[win]);
                    else mbar_arrive_cluster(mapa_shared(smem_u32(&tmem_empty[win]), 0));
                }
                win ^= 1;
                if (win == 0) win_phase ^= 1;
            }
            if (mine) {
                for (int r = t.tail + half * 8 + (lane >> 2); r < t.tail_end; r += 16)
                    *reinterpret_cast<int4*>(out + (ptrdiff_t)(r - (lane >> 2) - t.row) * p.n) = make_int4(0, 0, 0, 0);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves while the other may still signal it or read its operands
    if (threadIdx.x == 0 && s_abort && p.error_flag != nullptr) atomicExch(p.error_flag, 1);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 2 * kPairWindowCols);
    }
}

template <bool kMn>
cudaError_t launch_pairs_impl(const GroupedGemmArgs& a, cudaStream_t stream) {
    PairMaps maps;
    const uint64_t G = (uint64_t)a.num_groups;
    if (!(kMn ? make_map_mn(&maps.w, a.b, G * a.k, (uint64_t)a.n, kBlockM) : make_map(&maps.w, a.b, false, G * a.n, (uint64_t)a.k, kBlockM))) return cudaErrorInvalidValue;
    for (int i = 0; i < 4; ++i)
        if (!make_map(&maps.t[i], a.a, false, (uint64_t)a.m_total, (uint64_t)a.k, 128 >> i)) return cudaErrorInvalidValue;
    const size_t fixed = 1024 /*align*/ + kPairEpiWarps * kBlockBytes + 256 /*barriers*/ + ((size_t)(a.num_groups + 1) * 4 + 15) / 16 * 16;
    const int stages = std::min(kPairMaxStages, (int)((kPairMaxSmem - fixed) / pair_stage_bytes(a.token_cap)));
    const size_t smem = std::max(kTensorKernelSmem, fixed + (size_t)stages * pair_stage_bytes(a.token_cap));
    auto kernel = token_pairs_gemm_kernel<kMn>;
    static bool smem_opted_in[64] = {};  // per device, once: the attribute is sticky
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !smem_opted_in[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairMaxSmem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) smem_opted_in[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.num_sms & ~1), 1, 1);
    cfg.blockDim = dim3(kPairThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, maps, a, stages);
}

}  // namespace

cudaError_t launch_token_pairs_gemm(const GroupedGemmArgs& a, cudaStream_t stream) {
    if (a.num_groups < 1 || a.num_groups > kMaxGroups || a.num_sms < 2 || a.mode != 0 || a.fp8 || a.swiglu || a.a_mn) return cudaErrorInvalidValue;
    if (a.token_cap < 64 || a.token_cap > 256 || a.token_cap % 64 != 0 || a.k % 64 != 0 || a.k <= 0 || a.n % 128 != 0) return cudaErrorInvalidValue;
    if (a.zero_tail && a.m_ends == nullptr) return cudaErrorInvalidValue;
    if (a.m_total <= 0) return cudaSuccess;  // (tensors without rows have no address)
    return a.b_mn ? launch_pairs_impl<true>(a, stream) : launch_pairs_impl<false>(a, stream);
}

}  // namespace dx
