// Grouped expert GEMM for groups of few to some hundred rows, natively block-scaled e4m3: the weights are the M operand and the tokens
// the N operand of tcgen05.mma.
//
// A layer whose experts have about a tile of rows each is bound by its weights, which every row tile pulls anew from L2: with tiles
// of 128 rows, an expert of 137 tokens costs two passes over them and 256 rows of products. Here a tile is 256 weight rows by ALL
// tokens of the group up to `token_cap` (at most 224, in steps of 16), so the weights of such an expert are read once and the products are those of its
// tokens; a longer group is cut into several (see row_tiles).
//
// The issuer's and the loader's loops are run by whole warps, with one elected lane issuing. The same loops as a branch that only lane 0 takes
// were slower, most of all here, where a K block of few tokens is eight short MMAs (one B200, both GEMMs, decode of 20 tokens, 64 experts of 4096 ->
// 1408: 212 -> 189 us; of 128 tokens, 256 experts of 7168 -> 2048: 1835 -> 1735 us, with 64 tokens in a tile 1692).
//
//   warp 0      TMA producer   global -> smem ring
//   warp 1      MMA issuer     two M = 128 products per K step (SwiGLU: gate and up rows of the same 128 features)
//   warps 2..9  epilogue       lane = weight row, column = token; two warps per TMEM lane quarter take alternate chunks of 16 tokens
//
// A stage holds 32 KB of weights, `token_cap` rows of 128 bytes and the scale atoms; the ring has as many stages as fit (five for 64
// tokens, four up to 160, three beyond), because bytes in flight are what streams weights. There is one accumulator window (two products of up
// to 224 columns and the scale factors fill TMEM): the epilogue packs it to BF16 in registers, hands it back, and does the rest (row
// maxima, quantisation, stores) while the next tile accumulates. That rest still bounds tiles of many tokens and few K blocks: without it (timing only)
// 64 experts of 188 rows, 4096 -> 1408, took 258 us instead of 358 for both GEMMs, and 256 experts of 128 rows, 7168 -> 2048, 1875 instead of 2100.
// Two chunks of tokens per exchange, scales from the exponent's bits and stores of 16 bytes brought the first to 304 (tokens as rows: 341).
//
// Every wait is bounded, as in grouped_gemm.cu.
#include <algorithm>

#include "launch.cuh"
#include "tc_prims.cuh"

namespace dx {

namespace {

constexpr int kWeightRows = 256;
constexpr int kWeightBytes = kWeightRows * kKBlockBytes;
constexpr int kSfStageBytes = 2048;     // two atoms of the weights, then up to two of the tokens
constexpr int kMaxTokenCap = 224;
constexpr int kHalfCols = kMaxTokenCap; // TMEM columns between the two products
constexpr int kSfCol0 = 2 * kHalfCols;  // two alternating sets of 8 + 8 columns
constexpr int kChunk = 16;              // tokens an epilogue warp takes at a time
constexpr int kChunks = kMaxTokenCap / (2 * kChunk);
constexpr int kMaxStages = 6;
constexpr int kColsEpiWarps = 8;
constexpr int kColsThreads = 64 + 32 * kColsEpiWarps;
constexpr int kMaxSmem = 232448;
constexpr int kColsAheadBlocks = 10;    // K blocks of the first tile's weights fetched into L2 before the predecessor ends (see grouped_gemm.cu)

// Boxes of 128, 64, 32 and 16 token rows: any multiple of 16 up to 224 rows in at most three copies.
struct TokenMaps {
    CUtensorMap m[4];
};

struct ColTile {
    int group, nt, row, valid, cols;  // cols: valid rows rounded up to the step of the N operand
    int w_row, w_row2;
};

__host__ __device__ constexpr size_t cols_table_bytes(int groups) { return ((size_t)(groups + 1) * 4 + 15) / 16 * 16; }
// SwiGLU: maxima of two tiles; else a block of 8 tokens x 32 features per epilogue warp
__host__ __device__ constexpr size_t cols_exchange_bytes(int cap, bool swiglu) { return swiglu ? (size_t)2 * cap * 16 : (size_t)kColsEpiWarps * 512; }
__host__ __device__ constexpr int cols_stage_bytes(int cap) { return kWeightBytes + cap * kKBlockBytes + kSfStageBytes; }

template <bool kSwiGLU>
__global__ void __launch_bounds__(kColsThreads, 1)
token_cols_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ TokenMaps maps_t, const GroupedGemmArgs p, const int stages) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* stage_base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int cap = p.token_cap;
    const int stage_bytes = cols_stage_bytes(cap);
    const int G = p.num_groups;
    uint64_t* bars = reinterpret_cast<uint64_t*>(stage_base + (size_t)stages * stage_bytes);
    uint64_t* full = bars;
    uint64_t* empty = bars + kMaxStages;
    uint64_t* tmem_full = bars + 2 * kMaxStages;
    uint64_t* tmem_empty = tmem_full + 1;
    uint64_t* tile_full = tmem_full + 2;
    uint64_t* tile_free = tile_full + kTileSlots;
    static_assert(2 * kMaxStages + 2 + 2 * kTileSlots <= 32, "barrier block");
    int* tile_start = reinterpret_cast<int*>(bars + 32);  // [G+1]
    uint8_t* xch_base = reinterpret_cast<uint8_t*>(tile_start) + cols_table_bytes(G);
    volatile uint32_t* xch = reinterpret_cast<volatile uint32_t*>(xch_base);  // SwiGLU: [2][cap][4]
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    __shared__ volatile int s_tile[kTileSlots];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_kb = p.k / 128, tiles_n = p.n / kWeightRows;

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(tmem_full, 1);
        mbar_init(tmem_empty, kColsEpiWarps);
        for (int i = 0; i < kTileSlots; ++i) {
            mbar_init(&tile_full[i], 1);
            mbar_init(&tile_free[i], 1 + kColsEpiWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tma_prefetch_desc(&map_w);
        for (int i = 0; i < 4; ++i) tma_prefetch_desc(&maps_t.m[i]);
    }
    if constexpr (kSwiGLU) {
        for (int i = threadIdx.x; i < 2 * cap * 4; i += kColsThreads) xch[i] = 0u;
    }
    if (warp == 1) tmem_alloc(&s_tmem_base, 512);
    // early_table and hold_successor: see grouped_gemm.cu
    if (!p.early_table) {
        pdl_wait_predecessor();
        if (!p.hold_successor) pdl_release_successor();
    }
    // Row tiles of a group: one of up to `cap` tokens, or `step` of them each, the last one of up to `cap` where the step is a whole scale
    // atom. A tile starts on an atom or in the middle of one, and touches two at most.
    const int step = cap < 128 ? 64 : cap < 192 ? 128 : 192;
    auto row_tiles = [&](int n) { return n <= 0 ? 0 : n <= cap ? 1 : step == 128 ? 1 + (n - cap + 127) / 128 : (n + step - 1) / step; };
    if (warp == 2) {
        build_tile_table(p, tile_start, lane, [&](int, int begin, int rows) {
            if ((begin & 127) != 0 && p.error_flag != nullptr) atomicExch(p.error_flag, 2);
            return row_tiles(rows) * tiles_n;
        });
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    const int total_tiles = tile_start[G];
    volatile int* abort_flag = &s_abort;
    const long long limit = p.timeout_cycles;
    unsigned long long* note = p.trace != nullptr ? p.trace + 2 : nullptr;

    auto decode = [&](int tile, int& g, ColTile& t) {
        while (tile >= tile_start[g + 1]) ++g;
        const int local = tile - tile_start[g];
        const int m0 = p.m_offsets[g], n = group_rows(p, g, m0);
        const int tiles_m = row_tiles(n);
        const int mt = local % tiles_m;  // consecutive tiles share the weights
        t.group = g;
        t.nt = local / tiles_m;
        t.row = m0 + mt * step;
        t.valid = min(mt == tiles_m - 1 ? n - mt * step : step, p.m_total - t.row);
        t.cols = (max(t.valid, 1) + kChunk - 1) / kChunk * kChunk;
        t.w_row = g * p.n + (kSwiGLU ? t.nt * 128 : t.nt * kWeightRows);
        t.w_row2 = g * p.n + p.n / 2 + t.nt * 128;  // SwiGLU: the matching up rows
    };

    const int stride = (int)gridDim.x;
    const bool drawn = p.sched != nullptr;
    int tslot = 0, tphase = 0;
    auto next_tile = [&](int tile) {
        if (!drawn) return tile + stride;
        if (!__all_sync(0xffffffffu, mbar_wait(&tile_full[tslot], tphase, abort_flag, limit, note, wait_id(8, tile, 0, tslot)))) return total_tiles;
        const int t = s_tile[tslot];
        __syncwarp();
        if (lane == 0) mbar_arrive(&tile_free[tslot]);
        if (++tslot == kTileSlots) {
            tslot = 0;
            tphase ^= 1;
        }
        return t;
    };

    if (p.early_table) {
        if (warp == 0 && lane == 0 && (int)blockIdx.x < total_tiles) {
            int g = 0;
            ColTile t;
            decode(blockIdx.x, g, t);
            for (int kb = 0; kb < min(num_kb, kColsAheadBlocks); ++kb) {
                tma_prefetch_2d(&map_w, kb * 128, t.w_row);
                if (kSwiGLU) tma_prefetch_2d(&map_w, kb * 128, t.w_row2);
            }
        }
        pdl_wait_predecessor();
        if (!p.hold_successor) pdl_release_successor();
    }

    if (warp == 0) {
        // ================= TMA producer =================
        int stage = 0, phase = 0, g = 0, issued = 0, gated_group = -1, drawn_tile = 0;
        bool stamped = false, ok = true;
        ColTile t;
        auto hand_out = [&](int tile) {
            if (!drawn) return tile + stride;
            const int next = min(stride + __shfl_sync(0xffffffffu, drawn_tile, 0), total_tiles);
            if (!__all_sync(0xffffffffu, mbar_wait(&tile_free[tslot], tphase ^ 1, abort_flag, limit, note, wait_id(9, tile, 0, tslot)))) {
                ok = false;
                return total_tiles;
            }
            if (lane == 0) {
                s_tile[tslot] = next;
                mbar_arrive(&tile_full[tslot]);
            }
            __syncwarp();
            if (++tslot == kTileSlots) {
                tslot = 0;
                tphase ^= 1;
            }
            return next;
        };
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile = hand_out(tile)) {
            if (drawn && lane == 0) drawn_tile = atomicAdd(p.sched, 1);  // used when this tile's loads have been issued
            decode(tile, g, t);
            if (p.ready != nullptr && t.group != gated_group) {
                // the rows of this group come from other GPUs: wait until all of them have landed
                const unsigned long long want = p.expected[t.group];
                if (ld_acquire_sys_u64(p.ready + t.group) < want) {
                    const long long t0 = clock64();
                    while (ld_acquire_sys_u64(p.ready + t.group) < want) {
                        if (*abort_flag || clock64() - t0 > limit) {
                            if (!*abort_flag && note != nullptr) atomicCAS(note, 0ull, wait_id(2, tile, 0, t.group));
                            *abort_flag = 1;
                            ok = false;
                            break;
                        }
                    }
                }
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                fence_proxy_async();
                gated_group = t.group;
            }
            if (p.trace != nullptr && !stamped) {
                if (lane == 0) atomicMin(&p.trace[0], global_timer_ns());
                stamped = true;
            }
            const int atoms = (t.row & 127) + t.cols > 128 ? 2 : 1;
            const uint32_t tx = kWeightBytes + t.cols * kKBlockBytes + 512 * (2 + atoms);
            const uint8_t* sfw = p.sfb_atoms + ((size_t)t.group * tiles_n + t.nt) * num_kb * 1024;
            const uint8_t* sft = p.sfa_atoms + (size_t)(t.row >> 7) * num_kb * 512;
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1, abort_flag, limit, note, wait_id(1, tile, kb, stage)))) {
                    ok = false;
                    break;
                }
                if (elect_one()) {
                    uint8_t* sw = stage_base + (size_t)stage * stage_bytes;
                    uint8_t* st = sw + kWeightBytes;
                    mbar_expect_tx(&full[stage], tx);
                    tma_load_2d(&map_w, &full[stage], sw, kb * 128, t.w_row);
                    if (kSwiGLU) tma_load_2d(&map_w, &full[stage], sw + kWeightBytes / 2, kb * 128, t.w_row2);
                    int at = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (t.cols & (128 >> i)) {
                            tma_load_2d(&maps_t.m[i], &full[stage], st + at * kKBlockBytes, kb * 128, t.row + at);
                            at += 128 >> i;
                        }
                    }
                    uint8_t* ssf = st + cap * kKBlockBytes;
                    bulk_load_1d(ssf, sfw + (size_t)kb * 1024, 1024, &full[stage]);
                    bulk_load_1d(ssf + 1024, sft + (size_t)kb * 512, 512, &full[stage]);
                    if (atoms > 1) bulk_load_1d(ssf + 1536, sft + (size_t)(num_kb + kb) * 512, 512, &full[stage]);
                }
                __syncwarp();
                if (issued < stages) ++issued;
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        if (drawn && lane == 0) {  // the last CTA to stop drawing leaves the counter as it was found
            __threadfence();
            if (atomicAdd(p.sched + 1, 1) == stride - 1) {
                p.sched[1] = 0;
                atomicExch(p.sched, 0);
            }
        }
        if (!ok) {  // copies in flight land in this CTA's shared memory: wait (bounded) for every armed stage
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
    } else if (warp == 1) {
        // ================= MMA issuer =================
        int stage = 0, phase = 0, g = 0, win_phase = 0, sf_buf = 0;
        bool ok = true;
        ColTile t;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile = next_tile(tile)) {
            decode(tile, g, t);
            const uint32_t idesc = make_idesc_mx(t.cols, kBlockM);
            const bool two_atoms = (t.row & 127) + t.cols > 128;
            if (!__all_sync(0xffffffffu, mbar_wait(tmem_empty, win_phase ^ 1, abort_flag, limit, note, wait_id(3, tile, 0, 0)))) break;
            win_phase ^= 1;
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag, limit, note, wait_id(4, tile, kb, stage)))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sw = smem_u32(stage_base) + (uint32_t)(stage * stage_bytes);
                const uint32_t st = sw + kWeightBytes, ssf = st + cap * kKBlockBytes;
                const uint64_t wdesc = make_smem_desc(sw), tdesc = make_smem_desc(st);
                const uint32_t t_sfw = tmem_base + (uint32_t)(kSfCol0 + sf_buf * 16);
                const uint32_t t_sft = t_sfw + 8 + (uint32_t)((t.row >> 5) & 2);  // a column has the factors of 32 tokens
                if (elect_one()) {
                    tmem_cp_sf(t_sfw, make_sf_desc(ssf));
                    tmem_cp_sf(t_sfw + 4, make_sf_desc(ssf + 512));
                    tmem_cp_sf(t_sfw + 8, make_sf_desc(ssf + 1024));
                    if (two_atoms) tmem_cp_sf(t_sfw + 12, make_sf_desc(ssf + 1536));
                    // The two products take turns (144 tokens, both GEMMs of 256 experts: 2210 -> 2165 us).
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            umma_mx(tmem_base + h * kHalfCols, wdesc + (uint64_t)(h * (kWeightBytes / 2 >> 4) + j * 2), tdesc + (uint64_t)(j * 2), idesc,
                                    t_sfw + 4 * h, t_sft, (kb == 0 && j == 0) ? 0u : 1u);
                    umma_commit(&empty[stage]);
                    if (kb == num_kb - 1) umma_commit(tmem_full);
                }
                __syncwarp();
                sf_buf ^= 1;
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
    } else {
        // ================= epilogue =================
        const int q = warp & 3;            // TMEM lane quarter this warp may read
        const int half = (warp - 2) >> 2;  // takes the chunks 2c + half
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
        const int ldc = kSwiGLU ? p.n / 2 : p.n;
        const bool scatter = !kSwiGLU && p.row_info != nullptr;
        int g = 0, win_phase = 0, tiles_done = 0;
        bool ok = true;
        ColTile t;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile = next_tile(tile)) {
            decode(tile, g, t);
            int info[kSwiGLU ? 1 : kChunks];  // scatter: lane l has the destination word of the chunk's token l
            if constexpr (!kSwiGLU) {
                if (scatter) {
#pragma unroll
                    for (int c = 0; c < kChunks; ++c) {
                        const int tok = (2 * c + half) * kChunk + (lane & 15);
                        info[c] = tok < t.valid ? p.row_info[t.row + tok] : -1;
                    }
                }
            }
            if (!mbar_wait(tmem_full, win_phase, abort_flag, limit, note, wait_id(6, tile, 0, warp))) {
                ok = false;
                break;
            }
            win_phase ^= 1;
            tc_fence_after();
            // The window in registers as BF16 pairs of neighbouring tokens: SwiGLU one feature per thread, else one of each product.
            uint32_t keep[kChunks][kSwiGLU ? 8 : 16];
#pragma unroll
            for (int c = 0; c < kChunks; ++c) {
                const int t0 = (2 * c + half) * kChunk;
                if (t0 < t.cols) {
                    uint32_t v[16], u[16];
                    tmem_ld16(taddr + t0, v);
                    tmem_ld16(taddr + kHalfCols + t0, u);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if constexpr (kSwiGLU) {
                            keep[c][i] = f2_to_bf16x2(silu(__uint_as_float(v[2 * i])) * __uint_as_float(u[2 * i]),
                                                      silu(__uint_as_float(v[2 * i + 1])) * __uint_as_float(u[2 * i + 1]));
                        } else {
                            keep[c][i] = f2_to_bf16x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
                            keep[c][8 + i] = f2_to_bf16x2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1]));
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tmem_empty);

            if constexpr (kSwiGLU) {
                // A tile's 128 features are one scale block of the next GEMM's activations: power-of-two scale from the token's largest
                // BF16 magnitude (NaN does not count, as with fmaxf). Each warp reduces its 32 features, eight pairs of tokens at once:
                // every step halves the pairs a lane keeps, so lane l ends with pair l / 4. The four quarters exchange their
                // maxima through words tagged with the tile's number, two tile parities.
                const unsigned tag = (unsigned)(++tiles_done & 0xffff) << 16;
                volatile uint32_t* xs = xch + (tiles_done & 1) * (cap * 4);
#pragma unroll
                for (int c = 0; c < kChunks; ++c) {
                    const int t0 = (2 * c + half) * kChunk;
                    if (t0 < t.cols) {
                        __nv_bfloat162 m[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const uint32_t mag = keep[c][i] & 0x7fff7fffu;
                            m[i] = *reinterpret_cast<const __nv_bfloat162*>(&mag);
                        }
#pragma unroll
                        for (int step = 4; step >= 1; step >>= 1) {
                            const bool upper = (lane & (step * 4)) != 0;
#pragma unroll
                            for (int i = 0; i < step; ++i) {
                                const __nv_bfloat162 send = upper ? m[i] : m[i + step], mine = upper ? m[i + step] : m[i];
                                const uint32_t got = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const uint32_t*>(&send), step * 4);
                                m[i] = __hmax2(mine, *reinterpret_cast<const __nv_bfloat162*>(&got));
                            }
                        }
#pragma unroll
                        for (int o = 2; o >= 1; o >>= 1) {
                            const uint32_t got = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const uint32_t*>(&m[0]), o);
                            m[0] = __hmax2(m[0], *reinterpret_cast<const __nv_bfloat162*>(&got));
                        }
                        const uint32_t both = *reinterpret_cast<const uint32_t*>(&m[0]);
                        uint32_t bits = ((lane & 1) ? both >> 16 : both) & 0x7fffu;
                        if (bits > 0x7f80u) bits = 0;
                        if ((lane & 3) < 2) xs[(t0 + (lane >> 2) * 2 + (lane & 1)) * 4 + q] = tag | bits;
                    }
                }
                // Two chunks at a time: lanes 0-15 have the tokens of the first, lanes 16-31 those of the second.
#pragma unroll
                for (int c2 = 0; c2 < kChunks; c2 += 2) {
                    if ((2 * c2 + half) * kChunk < t.cols && ok) {
                        const int tok = (2 * (c2 + (lane >> 4)) + half) * kChunk + (lane & 15);
                        uint32_t most = 0;
                        if (tok < t.cols) {
                            const uint32_t slot = smem_u32(const_cast<const uint32_t*>(xs) + tok * 4);
                            uint32_t w[4];
                            auto look = [&]() {
                                asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(slot) : "memory");
                                return (((w[0] ^ tag) | (w[1] ^ tag) | (w[2] ^ tag) | (w[3] ^ tag)) >> 16) == 0;
                            };
                            if (!look()) {
                                const long long w0 = clock64();
                                while (!look()) {
                                    if (*abort_flag || clock64() - w0 > limit) {
                                        if (!*abort_flag && note != nullptr) atomicCAS(note, 0ull, wait_id(7, tile, 0, warp));
                                        *abort_flag = 1;
                                        ok = false;
                                        break;
                                    }
                                }
                            }
                            most = max(max(w[0], w[1]), max(w[2], w[3])) & 0xffffu;
                        }
                        ok = __all_sync(0xffffffffu, ok);
                        if (ok) {
                            float scale, inv;
                            fp8_scale_from_amax(__uint_as_float(most << 16), true, scale, inv);
                            if (q == 0 && tok < t.valid) {
                                const int row = t.row + tok;
                                *reinterpret_cast<uint32_t*>(p.c_atoms + ((size_t)(row >> 7) * (ldc / 128) + t.nt) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4) =
                                    ((__float_as_uint(scale) >> 23) & 0xffu) * 0x01010101u;
                            }
#pragma unroll
                            for (int c = c2; c < c2 + 2 && c < kChunks; ++c) {
                                const int t0 = (2 * c + half) * kChunk;
                                if (t0 >= t.cols) break;
                                uint8_t* dst = p.c_fp8 + (size_t)(t.row + t0 + (lane & 3)) * ldc + t.nt * 128 + q * 32 + (lane & ~3);
#pragma unroll
                                for (int i = 0; i < kChunk; i += 4) {
                                    const float2 lo = bf16x2_to_f2(keep[c][i / 2]), hi = bf16x2_to_f2(keep[c][i / 2 + 1]);
                                    const int from = (c & 1) * 16 + i;
                                    const float x0 = lo.x * __shfl_sync(0xffffffffu, inv, from), x1 = lo.y * __shfl_sync(0xffffffffu, inv, from + 1);
                                    const float x2 = hi.x * __shfl_sync(0xffffffffu, inv, from + 2), x3 = hi.y * __shfl_sync(0xffffffffu, inv, from + 3);
                                    const uint32_t w = transpose_bytes_4x4(pack_e4m3x4(x0, x1, x2, x3), lane);
                                    if (t0 + i + (lane & 3) < t.valid) *reinterpret_cast<uint32_t*>(dst + (size_t)i * ldc) = w;
                                }
                            }
                        }
                    }
                }
            } else {
                // Two lanes exchange halves, so that each has two neighbouring features of one token; eight tokens then pass through shared
                // memory, and every lane stores 16 bytes: 64 contiguous ones per token.
                uint32_t* block = reinterpret_cast<uint32_t*>(xch_base) + (warp - 2) * 128;
                const int col = t.nt * kWeightRows + q * 32 + (lane & 3) * 8;
#pragma unroll
                for (int c = 0; c < kChunks; ++c) {
                    const int t0 = (2 * c + half) * kChunk;
                    if (t0 < t.cols) {
#pragma unroll
                        for (int g8 = 0; g8 < 2; ++g8) {
                            const int tok = t0 + g8 * 8 + (lane >> 2);
                            __nv_bfloat16* dst = nullptr;
                            if (scatter) {
                                const int word = __shfl_sync(0xffffffffu, info[c], g8 * 8 + (lane >> 2));
                                if (word >= 0) dst = reinterpret_cast<__nv_bfloat16*>(p.scatter_bases[word >> 24]) + (size_t)(word & 0xffffff) * ldc + col;
                            } else if (tok < t.valid) {
                                dst = reinterpret_cast<__nv_bfloat16*>(p.c) + (size_t)(t.row + tok) * ldc + col;
                            }
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const uint32_t w = keep[c][h * 8 + g8 * 4 + i];
                                    const uint32_t o = __shfl_xor_sync(0xffffffffu, w, 1);
                                    block[(2 * i + (lane & 1)) * 16 + (lane >> 1)] = __byte_perm(w, o, (lane & 1) ? 0x3276 : 0x5410);
                                }
                                __syncwarp();
                                const int4 piece = *reinterpret_cast<const int4*>(block + lane * 4);
                                __syncwarp();
                                if (dst != nullptr) *reinterpret_cast<int4*>(dst + h * 128) = piece;
                            }
                        }
                    }
                }
            }
        }
    }

    if (warp >= 2) {
        if (p.row_info != nullptr) __threadfence_system();  // rows scattered into other GPUs' memory are performed there
        if (p.trace != nullptr && warp == 2 && lane == 0) atomicMax(&p.trace[1], global_timer_ns());
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && s_abort && p.error_flag != nullptr) atomicExch(p.error_flag, 1);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

template <bool kSwiGLU>
cudaError_t launch_cols_impl(const GroupedGemmArgs& a, cudaStream_t stream) {
    CUtensorMap map_w;
    TokenMaps maps_t;
    if (!make_map(&map_w, a.b, true, (uint64_t)a.num_groups * a.n, (uint64_t)a.k, kSwiGLU ? kWeightRows / 2 : kWeightRows)) return cudaErrorInvalidValue;
    for (int i = 0; i < 4; ++i)
        if (!make_map(&maps_t.m[i], a.a, true, (uint64_t)a.m_total, (uint64_t)a.k, 128 >> i)) return cudaErrorInvalidValue;
    const size_t fixed = 1024 /*align*/ + 256 /*barriers*/ + cols_table_bytes(a.num_groups) + cols_exchange_bytes(a.token_cap, kSwiGLU);
    const int stages = std::min(kMaxStages, (int)((kMaxSmem - 512 /*static*/ - fixed) / cols_stage_bytes(a.token_cap)));
    const size_t smem = std::max(kTensorKernelSmem, fixed + (size_t)stages * cols_stage_bytes(a.token_cap));
    auto kernel = token_cols_gemm_kernel<kSwiGLU>;
    static bool smem_opted_in[64] = {};  // per device, once: the attribute is sticky
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !smem_opted_in[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem - 512);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) smem_opted_in[dev] = true;
    }
    return launch_dependent(kernel, dim3(a.num_sms), kColsThreads, smem, stream, map_w, maps_t, a, stages);
}

}  // namespace

cudaError_t launch_token_cols_gemm(const GroupedGemmArgs& a, cudaStream_t stream) {
    if (a.num_groups < 1 || a.num_groups > kMaxGroups || a.num_sms < 1 || a.mode != 0 || !a.fp8) return cudaErrorInvalidValue;
    if (a.token_cap < 64 || a.token_cap > kMaxTokenCap || a.token_cap % 32 != 0 || a.k % 128 != 0 || a.k <= 0 || a.n % kWeightRows != 0) return cudaErrorInvalidValue;
    if (a.m_total <= 0) return cudaSuccess;  // (tensors without rows have no address)
    if (a.sfa_atoms == nullptr || a.sfb_atoms == nullptr || (a.swiglu && (a.c_fp8 == nullptr || a.c_atoms == nullptr))) return cudaErrorInvalidValue;
    return a.swiglu ? launch_cols_impl<true>(a, stream) : launch_cols_impl<false>(a, stream);
}

}  // namespace dx
