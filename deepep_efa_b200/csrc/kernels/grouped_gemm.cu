// Grouped expert GEMM for sm_100a: tcgen05.mma with the accumulator in TMEM, operands staged into
// 128-byte-swizzled shared memory by TMA (from this GPU's own memory only, never multicast), a
// persistent warp-specialised CTA per SM.
//
//   warp 0   : TMA producer   (one elected lane issues)  global -> smem ring, mbarrier complete_tx
//   warp 1   : MMA issuer     (one elected thread)  tcgen05.mma, tcgen05.commit frees smem stages and publishes
//                                         accumulator windows; also owns TMEM alloc / dealloc
//   warps 2.. : epilogue (4 warps for BF16, 8 for FP8)  tcgen05.ld -> registers -> (scale | SwiGLU) -> BF16 ->
//                                         per-warp smem transpose -> coalesced global stores
//
// A tile is 128 rows x kBlockN columns; a K block is 128 bytes per row (64 BF16 or 128 e4m3), i.e. one
// swizzle atom, consumed by four MMAs. Two accumulator windows in TMEM let the epilogue of window i
// overlap the MMAs of window i+1. BF16: a window is a whole output tile. FP8 with DeepSeek-style fp32
// scales (1x128 on activations, 128x128 on weights): a window is ONE K block; the epilogue multiplies it
// by scale_a[row, kb] * scale_b[nblock, kb] and accumulates in fp32 registers (the MMA's native block
// scaling wants power-of-two UE8M0 factors, which these scales are not). Tiles of 256 columns where there are enough of them (wide_promotion).
//
// Every mbarrier wait is bounded; when a limit runs out the CTA raises a flag, all roles leave their
// loops, TMEM is released and the kernel returns.
//
// The reference has no GEMM: its users run their expert FFN between dispatch and combine themselves.
#include <cstring>

#include "gemm_choice.h"
#include "launch.cuh"
#include "tc_prims.cuh"

namespace dx {

namespace {

constexpr int kEdgeRows = 32;          // rows of one copy when a tile of A is fetched in part
// Of the last K block of a weight gradient, where its reduction has no more left: half the bytes of a block that short reductions have two or three of (both of
// 64 experts of 4096 -> 1408 in a loop, 94 rows 518 -> 490 us).
constexpr int kTailRows = 32;
constexpr int kAheadBlocks = 10;       // K blocks of weights per CTA fetched into L2 before the predecessor ends: 48 MB of the 126 MB

__device__ __forceinline__ int4 pack8_bf16(const float* o) {
    int4 w;
    __nv_bfloat162 t0 = __floats2bfloat162_rn(o[0], o[1]), t1 = __floats2bfloat162_rn(o[2], o[3]);
    __nv_bfloat162 t2 = __floats2bfloat162_rn(o[4], o[5]), t3 = __floats2bfloat162_rn(o[6], o[7]);
    w.x = *reinterpret_cast<int*>(&t0);
    w.y = *reinterpret_cast<int*>(&t1);
    w.z = *reinterpret_cast<int*>(&t2);
    w.w = *reinterpret_cast<int*>(&t3);
    return w;
}

// Stores a 32-row x kCols BF16 block that a warp holds one row per lane. Writing it straight from registers would put
// every lane on its own 32-byte sector (half filled); instead the block is transposed through a per-warp shared
// buffer (XOR-swizzled 16-byte pieces) so that each store instruction covers whole rows: 128 contiguous bytes per row
// for kCols = 64, 64 bytes for kCols = 32.
template <int kCols>
__device__ __forceinline__ void store_block_coalesced(int4* stage, const int4 (&regs)[kCols / 8], __nv_bfloat16* gbase, int ldc,
                                                      int rows_valid, int lane) {
    constexpr int P = kCols / 8;    // 16-byte pieces per row
    constexpr int RPI = 32 / P;     // rows covered by one store instruction
    __syncwarp();
#pragma unroll
    for (int j = 0; j < P; ++j) stage[lane * P + (j ^ (lane & (P - 1)))] = regs[j];
    __syncwarp();
    int4 v[P];  // (all of them in front of the stores, behind which the compiler must not move them)
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const int row = i * RPI + lane / P, piece = lane % P;
        v[i] = stage[row * P + (piece ^ (row & (P - 1)))];
    }
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const int row = i * RPI + lane / P, piece = lane % P;
        if (row < rows_valid) *reinterpret_cast<int4*>(gbase + (size_t)row * ldc + piece * 8) = v[i];
    }
}

// 32 rows x 32 BF16 columns, one row per lane, without shared memory: lanes 2i and 2i + 1 exchange halves, so that each store instruction writes 64
// contiguous bytes of 16 rows. Every row's address is a multiple of 32 bytes, and the columns are stored at multiples of 16.
// Where the reduction is short the epilogue is the tile: 4500 cycles for 128 x 256 outputs through the staging buffer of store_block_coalesced and with the group's
// table in global memory (20 to 94 rows per expert), 3100 with these stores and the table in shared memory. Both weight gradients of 64 experts of 4096 -> 1408 in a
// loop, us, before / with that and reductions that stop at the last row: 20 rows 559 / 453, 94 rows 623 / 538, 190 rows 753 / 671, 384 rows 1061 / 1041, on pairs 768 rows
// 1563 / 1567 (what came since stands at kTailRows and kWgrad). Other forms of the store, the first of the two, 94 rows, us: these 343, whole lines of 128 bytes by two
// exchanges 343, columns read from TMEM ahead 398.
struct RowPair {
    __nv_bfloat16 *even, *odd;  // this lane's half of 32 columns of the rows of lanes 2i and 2i + 1 (nullptr: no such row)
    bool upper;
    __device__ __forceinline__ RowPair(__nv_bfloat16* mine, int lane) : upper(lane & 1) {
        __nv_bfloat16* other = reinterpret_cast<__nv_bfloat16*>(__shfl_xor_sync(0xffffffffu, reinterpret_cast<unsigned long long>(mine), 1));
        even = upper ? other : mine;
        odd = upper ? mine : other;
        if (upper && even != nullptr) even += 16;
        if (upper && odd != nullptr) odd += 16;
    }
    __device__ __forceinline__ void store(const int4 (&regs)[4], int column) const {
        uint32_t w[16], first[8], second[8];
        memcpy(w, regs, sizeof(w));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? w[j] : w[8 + j], 1);
            first[j] = upper ? got : w[j];
            second[j] = upper ? w[8 + j] : got;
        }
        st_global_256(even + column, first, even != nullptr);
        st_global_256(odd + column, second, odd != nullptr);
    }
};

// Same block, but every row goes to its own destination: lane l holds the address of row l (nullptr = drop the row).
template <int kCols>
__device__ __forceinline__ void store_block_scattered(int4* stage, const int4 (&regs)[kCols / 8], __nv_bfloat16* my_row_ptr, int lane) {
    constexpr int P = kCols / 8;
    constexpr int RPI = 32 / P;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < P; ++j) stage[lane * P + (j ^ (lane & (P - 1)))] = regs[j];
    __syncwarp();
    const unsigned long long mine = reinterpret_cast<unsigned long long>(my_row_ptr);
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const int row = i * RPI + lane / P, piece = lane % P;
        const int4 v = stage[row * P + (piece ^ (row & (P - 1)))];
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(__shfl_sync(0xffffffffu, mine, row));
        if (dst != nullptr) *reinterpret_cast<int4*>(dst + piece * 8) = v;
    }
}

// 32 rows x 256 bytes: lane l holds row l as 16 pieces of 16 bytes, and the row's destination (nullptr = drop the row). Eight rows at a
// time pass through a 2 KiB staging buffer (XOR-swizzled pieces), so that every store instruction covers two whole 256-byte rows:
// rows that leave for another GPU cross NVLink in 256-byte packets.
__device__ __forceinline__ void store_rows_256(int4* stage, const int4 (&regs)[16], __nv_bfloat16* my_row_ptr, int lane) {
    const unsigned long long mine = reinterpret_cast<unsigned long long>(my_row_ptr);
#pragma unroll
    for (int g8 = 0; g8 < 4; ++g8) {
        __syncwarp();
        if ((lane >> 3) == g8) {
#pragma unroll
            for (int j = 0; j < 16; ++j) stage[(lane & 7) * 16 + (j ^ (lane & 7))] = regs[j];
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r8 = i * 2 + (lane >> 4), piece = lane & 15;
            const int4 v = stage[r8 * 16 + (piece ^ r8)];
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(__shfl_sync(0xffffffffu, mine, g8 * 8 + r8));
            if (dst != nullptr) *reinterpret_cast<int4*>(dst + piece * 8) = v;
        }
    }
}

struct TileInfo {
    int a_row, a_k0, b_row, b_row2, b_k0, num_kb, c_row, c_col, group, nblock, nblock2;
    int c_row_end;  // first output row this tile must not write (end of its group; groups need no 128-row alignment)
    int k_rows;     // weight gradients: rows of the reduction
    int tail_kb;    // and the K block that holds at most kTailRows of them, MN-major (-1: none)
    int nt;         // n-tile index inside the group (kMx: selects the B scale atoms)
    int n_cols;     // columns of this tile: kBlockN, or half of it for the last column tile of an MN-major operand (kRagged)
    // MN-major operands: first tile row inside the tensor's contiguous dimension, and the tensor row of K index 0
    int a_mn0, a_kbase, b_mn0, b_kbase;
};

// kRowScatter: the scatter epilogue writes every output row of a 128-column tile as ONE 256-byte piece (the largest NVLink
// packet) instead of two 128-byte pieces; it needs an 8 KiB staging buffer per epilogue warp and gives up one pipeline stage.
template <int kBlockN, bool kFp8, bool kSwiGLU, bool kPair, bool kMx = false, bool kRowScatter = false>
struct Cfg {
    static constexpr bool kPromote = kFp8 && !kMx;  // FP8 with fp32 scales: every K block is promoted on the CUDA cores
    static constexpr int kSfBAtoms = kBlockN / 128;                  // 512-byte scale atoms of the B tile
    static constexpr int kSfTxBytes = kMx ? 512 * (1 + kSfBAtoms) : 0;   // per stage: scale atoms of A and of B
    static constexpr int kSfBytes = (kSfTxBytes + 1023) / 1024 * 1024;   // stages stay 1024-byte aligned (swizzle atoms)
    // B rows staged per CTA: a CTA pair splits the tile's N between its two CTAs
    static constexpr int kBRows = kPair ? kBlockN / 2 : kBlockN;
    static constexpr int kBTileBytes = kBRows * kKBlockBytes;
    static constexpr int kStageBytes = kATileBytes + kBTileBytes + kSfBytes;
    static constexpr int kStageTxBytes = kATileBytes + kBTileBytes + kSfTxBytes;  // bytes the copies of one stage deliver
    static constexpr int kStages = kMx ? ((kBlockN == 256) ? (kPair ? 5 : 4) : (kRowScatter ? 5 : 6)) : kPair ? ((kBlockN == 256) ? (kFp8 ? 5 : 6) : (kFp8 ? 6 : 8)) : ((kBlockN == 256) ? 4 : (kFp8 ? 5 : 6));
    static constexpr int kTileRows = kPair ? 2 * kBlockM : kBlockM;  // rows of one scheduled tile (both CTAs of a pair)
    // Accumulator windows in TMEM. FP8 hands the epilogue one window per K block, so the MMA warp needs to run several
    // K blocks ahead of the promotion: four 128-column windows fill TMEM. BF16 hands over one window per tile: two.
    // kMx with 256-column tiles: ONE window (two would fill TMEM and leave no room for the scale columns); the epilogue of
    // that variant drains the accumulator into registers first and releases the window before it stores.
    static constexpr int kWindows = kPromote ? (kBlockN == 256 ? 2 : 4) : ((kMx && kBlockN == 256) ? 1 : 2);
    static constexpr int kSfCol0 = kWindows * kBlockN;   // kMx: two alternating sets of (4 columns A + 4 per B atom) after the windows
    static constexpr int kSfColsPerBuf = 4 + 4 * kSfBAtoms;
    static constexpr int kTmemCols = kMx ? 512 : kWindows * kBlockN;
    static constexpr int kOutCols = kSwiGLU ? kBlockN / 2 : kBlockN;
    // (Tiles of 256 columns have two windows, and 128 accumulators per thread.)
    // FP8 promotes every K block on the CUDA cores, so it gets two epilogue warps per TMEM lane quarter (each takes half
    // of the columns); BF16 reads the accumulator once per tile and one warp per quarter is plenty.
    // The single-window wide tile also gets two warps per quarter: each drains half of the columns RAW (128 fp32 registers per
    // thread) and hands the window back at once, so the MMA issuer idles for the TMEM reads only, not for the SwiGLU arithmetic.
    static constexpr bool kSplitDrain = kMx && kBlockN == 256;
    // plain BF16 with MN-major B: a column count that is an odd multiple of 128 ends in one tile of half the width
    static constexpr bool kRagged = !kFp8 && !kSwiGLU && kBlockN == 256;
    static constexpr int kEpiWarps = (kPromote || kSplitDrain) ? 8 : 4;
    // first row and rows of every group in shared memory too: read from global memory they cost an epilogue that has little else to do 500 cycles a tile
    static constexpr bool kGroupTable = !kMx;
    static constexpr bool kWidePromote = kPromote && kBlockN == 256;
    // 128 accumulators per thread and two buffers of 32 columns do not fit the 168 registers that ten warps get: with the epilogue in warpgroups of its own, the
    // loader's and issuer's (and two warps that have nothing to do) hand theirs over. The sum is what the block was launched with: 3 x 168.
    static constexpr bool kMoveRegs = kWidePromote;
    static constexpr int kLaunchRegs = 168, kSmallRegs = 56, kEpiRegs = 224;
    static_assert(kSmallRegs + 2 * kEpiRegs <= 3 * kLaunchRegs, "a split above the launch's registers waits forever");
    static constexpr int kFirstEpi = kMoveRegs ? 4 : 2;  // first warp of the epilogue
    static constexpr int kThreads = 32 * (kFirstEpi + kEpiWarps);
    static constexpr int kOutStageBytes = kWidePromote ? 0 : kRowScatter ? 8192 : (kSplitDrain ? 2048 : 4096);    // per epilogue warp: 32 rows x 32 / 64 (128) BF16
    // kSplitDrain with quantised output: the two warps of a quarter exchange their half-row maxima here (two tile parities)
    static constexpr int kXchBytes = ((kMx || kPromote) && kSwiGLU && kBlockN == 256) ? 2 * 2 * kBlockM * 8 : 0;
    static constexpr size_t kSmemBytes =
        (size_t)kStages * kStageBytes + (size_t)kEpiWarps * kOutStageBytes + 1024 /*align*/ + 256 /*barriers*/ + (kMaxGroups + 2) * 4 + kXchBytes +
        (kGroupTable ? kMaxGroups * 8 : 0);
    static_assert(kSmemBytes >= kTensorKernelSmem, "kernels with tensor memory must not share an SM");
};

// kWgrad: weight gradients with both operands read in place. What is fixed for them costs no instructions (every launch fetches its code anew, and an MMA whose
// operands are not known costs more to issue): 8 experts, 1408 x 1024, 512 rows 15.9 -> 15.5 us, 16 experts, 2816 x 1024, 320 rows 37.2 -> 36.1.
template <int kBlockN, bool kFp8, bool kSwiGLU, bool kPair, bool kMx = false, bool kRowScatter = false, bool kWgrad = false>
__global__ void __launch_bounds__((Cfg<kBlockN, kFp8, kSwiGLU, kPair, kMx, kRowScatter>::kThreads), 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb, const GroupedGemmArgs p) {
    using C = Cfg<kBlockN, kFp8, kSwiGLU, kPair, kMx, kRowScatter>;
    static_assert(!kWgrad || (!kFp8 && !kSwiGLU), "weight gradients are BF16");
    const int mode = kWgrad ? 1 : p.mode, b_mn = kWgrad ? 1 : p.b_mn;
    constexpr int a_mn = kWgrad ? 1 : 0;  // (nothing else takes A that way)
    static_assert(!kRowScatter || (kMx && !kSwiGLU && !kPair && kBlockN == 128), "whole-row scatter: natively block-scaled 128-column tiles");
    static_assert(!kMx || (kFp8 && ((!kPair && kBlockN == 128) || (kBlockN == 256 && (kSwiGLU || !kPair)))),
                  "native block scaling: e4m3 operands; 128-column tiles, 256-column tiles, or 256-column SwiGLU tiles on a CTA pair");
    const uint32_t cta_rank = kPair ? cluster_ctarank() : 0u;   // 0 = leader (issues the MMAs of the pair)
    const int sched_id = kPair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int sched_stride = kPair ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* stage_base = smem;
    uint8_t* out_stage_base = smem + (size_t)C::kStages * C::kStageBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_stage_base + (size_t)C::kEpiWarps * C::kOutStageBytes);
    uint64_t* full = bars;                       // [kStages]
    uint64_t* empty = bars + C::kStages;         // [kStages]
    uint64_t* tmem_full = bars + 2 * C::kStages; // [kWindows]
    uint64_t* tmem_empty = tmem_full + C::kWindows;  // [kWindows]
    uint64_t* tile_full = tmem_empty + C::kWindows;   // [kTileSlots] tiles handed out by the loader (p.sched)
    uint64_t* tile_free = tile_full + kTileSlots;     // [kTileSlots]
    static_assert(2 * C::kStages + 2 * C::kWindows + 2 * kTileSlots <= 32, "barrier block");
    int* tile_start = reinterpret_cast<int*>(bars + 32);  // [G+1] first tile index of every group
    volatile unsigned long long* xch = reinterpret_cast<volatile unsigned long long*>(bars + 32 + (kMaxGroups + 2) / 2);  // [2][2][kBlockM] (tile tag << 32 | amax bits)
    int2* group_table = reinterpret_cast<int2*>(bars + 32 + (kMaxGroups + 2) / 2 + C::kXchBytes / 8);  // kGroupTable: (first row, rows)
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    __shared__ volatile int s_tile[kTileSlots];
    __shared__ volatile int s_prod_state[2];  // what the loader is doing (1 = arrival gate, 2 = free stage, 3 = loads issued) and for which tile

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = p.num_groups;
    const int elem_per_kb = kFp8 ? 128 : 64;
    constexpr bool kMnMajor = !kFp8 && !kSwiGLU;    // instantiations that take MN-major operands
    const int out_width = mode == 0 ? p.n : p.k;  // columns that the column tiles cover
    const int col_tiles = C::kRagged ? (out_width + kBlockN - 1) / kBlockN : out_width / kBlockN;

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < C::kWindows; ++a) {
            mbar_init(&tmem_full[a], 1);
            mbar_init(&tmem_empty[a], kPair ? 2 * C::kEpiWarps : C::kEpiWarps);  // the leader collects both CTAs' epilogue warps
        }
        for (int i = 0; i < kTileSlots; ++i) {
            mbar_init(&tile_full[i], 1);
            mbar_init(&tile_free[i], 1 + C::kEpiWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tma_prefetch_desc(&map_a);
        tma_prefetch_desc(&map_b);
    }
    if (!kPair && mode == 0 && p.m_ends != nullptr) {  // see `edge` below
        for (int s = 0; s < C::kStages; ++s)
            for (int i = threadIdx.x; i < kATileBytes / 16; i += C::kThreads)
                reinterpret_cast<int4*>(stage_base + (size_t)s * C::kStageBytes)[i] = make_int4(0, 0, 0, 0);
        fence_proxy_async();
    }
    if (warp == 1) {
        if constexpr (kPair) tmem_alloc_pair(&s_tmem_base, C::kTmemCols);
        else tmem_alloc(&s_tmem_base, C::kTmemCols);
    }
    if constexpr (kPair) cluster_sync_all();  // the peer's barriers exist before anything signals them
    // What precedes overlaps the end of the previous kernel (programmatic dependent launch); from here on its results are read.
    // The successor is released only now, so that a kernel that starts early finds every kernel before this one complete.
    // With p.early_table the group table is older than the predecessor, so the tile table and the first weights do not wait for it.
    if (!p.early_table) {
        pdl_wait_predecessor();
        if (!p.hold_successor) pdl_release_successor();
    }
    if (warp == 2) {
        const int tiles_n = mode == 0 ? col_tiles : 0;
        const int tiles_fixed = mode == 1 ? ((p.n + C::kTileRows - 1) / C::kTileRows) * col_tiles : 0;
        build_tile_table(p, tile_start, lane, [&](int g, int begin, int rows) {
            // native block scaling reads one scale atom per 128-row tile, so a group that does not start on a tile boundary
            // would be scaled with its neighbour's factors: flag it (value 2) instead of returning silently wrong numbers
            if (kMx && (begin & 127) != 0 && p.error_flag != nullptr) atomicExch(p.error_flag, 2);
            if (C::kGroupTable) group_table[g] = make_int2(begin, rows);
            return mode == 0 ? ((rows + C::kTileRows - 1) / C::kTileRows) * tiles_n : tiles_fixed;
        });
    }
    if constexpr (C::kXchBytes > 0) {
        for (int i = threadIdx.x; i < C::kXchBytes / 8; i += C::kThreads) xch[i] = 0ull;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    const int total_tiles = tile_start[G];
    volatile int* abort_flag = &s_abort;
    const long long limit = p.timeout_cycles;
    unsigned long long* note = p.trace != nullptr ? p.trace + 2 : nullptr;  // trace[2]: first bounded wait that gave up

    // Decodes tile index -> coordinates; `g` is a cursor that only moves forward.
    auto decode = [&](int tile, int& g, TileInfo& ti) {
        while (tile >= tile_start[g + 1]) ++g;
        const int local = tile - tile_start[g];
        int2 own;
        if constexpr (C::kGroupTable) own = group_table[g];
        else own = make_int2(p.m_offsets[g], group_rows(p, g, p.m_offsets[g]));
        const int m0 = own.x, m1 = own.x + own.y;
        ti.group = g;
        if (mode == 0) {
            const int tiles_m = (m1 - m0 + C::kTileRows - 1) / C::kTileRows;
            const int tiles_n_ = col_tiles;
            // order 0: consecutive tiles share the weight tile (n outer); order 1: they share the activation tile (m outer)
            const int nt = p.tile_order == 0 ? local / tiles_m : local % tiles_n_;
            const int mt = p.tile_order == 0 ? local % tiles_m : local / tiles_n_;
            ti.a_row = m0 + mt * C::kTileRows + (int)cta_rank * kBlockM;
            ti.nt = nt;
            ti.n_cols = C::kRagged ? min(kBlockN, out_width - nt * kBlockN) : kBlockN;
            ti.a_mn0 = ti.a_kbase = 0;                                          // mode 0: A is always K-major
            ti.b_mn0 = nt * kBlockN + (int)cta_rank * (ti.n_cols / 2);          // MN-major B: [G * K, N], N contiguous
            ti.b_kbase = g * p.k;
            ti.a_k0 = 0;
            ti.b_k0 = 0;
            ti.num_kb = p.k / elem_per_kb;
            ti.k_rows = 0;
            ti.tail_kb = -1;
            ti.c_row = ti.a_row;
            ti.c_row_end = min(m1, p.m_total);
            if (kSwiGLU) {
                const int half = kBlockN / 2, inter = p.n / 2;
                ti.b_row = g * p.n + nt * half;            // gate rows
                ti.b_row2 = g * p.n + inter + nt * half;   // up rows
                ti.c_col = nt * half;
                ti.nblock = (nt * half) / 128;
                ti.nblock2 = (inter + nt * half) / 128;
            } else {
                ti.b_row = g * p.n + nt * kBlockN + (int)cta_rank * (kBlockN / 2);  // a pair splits the tile's N
                ti.b_row2 = 0;
                ti.c_col = nt * kBlockN;
                ti.nblock = (nt * kBlockN) / 128;
                ti.nblock2 = ti.nblock;
            }
        } else {
            const int tiles_j = col_tiles;
            const int it = local / tiles_j, jt = local % tiles_j;
            ti.n_cols = C::kRagged ? min(kBlockN, out_width - jt * kBlockN) : kBlockN;
            ti.a_row = it * C::kTileRows + (int)cta_rank * kBlockM;
            ti.b_row = jt * kBlockN + (int)cta_rank * (ti.n_cols / 2);
            ti.b_row2 = 0;
            ti.a_mn0 = ti.a_row;                                                // MN-major: A is [M, N_out], B is [M, K_out]
            ti.b_mn0 = ti.b_row;
            ti.a_kbase = ti.b_kbase = m0;
            ti.a_k0 = m0;
            ti.b_k0 = m0;
            ti.k_rows = own.y;  // (with p.m_ends the rows behind it are zero in both operands)
            ti.num_kb = (ti.k_rows + elem_per_kb - 1) / elem_per_kb;
            ti.tail_kb = kWgrad && ti.num_kb * 64 - ti.k_rows >= 64 - kTailRows ? ti.num_kb - 1 : -1;
            ti.c_row = g * p.n + ti.a_row;
            ti.c_row_end = min((g + 1) * p.n, p.num_groups * p.n);
            ti.c_col = jt * kBlockN;
            ti.nblock = ti.nblock2 = 0;
        }
    };

    // Which tile comes next. Without p.sched every CTA walks its share in strides. With it the loader draws tiles from a counter and
    // passes them on through a small ring: SMs see unequal shares of the L2-to-SM bandwidth, and with equal numbers of tiles the
    // slowest of them finished tens of microseconds after the first in kernels that stream weights (one B200, decode of 128 tokens
    // through 256 experts of 7168 -> 2048: first / second GEMM 1243 / 661 -> 1209 / 622 us; the fused layer of 4096 tokens 2700 -> 2600).
    const bool drawn = !kPair && p.sched != nullptr;
    int tslot = 0, tphase = 0;  // this role's position in the ring
    auto next_tile = [&](int tile) {
        if (!drawn) return tile + sched_stride;
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

    auto next_tile_alone = [&](int tile) {  // for a single thread of a warp
        if (!drawn) return tile + sched_stride;
        if (!mbar_wait(&tile_full[tslot], tphase, abort_flag, limit, note, wait_id(8, tile, 0, tslot))) return total_tiles;
        const int t = s_tile[tslot];
        mbar_arrive(&tile_free[tslot]);
        if (++tslot == kTileSlots) {
            tslot = 0;
            tphase ^= 1;
        }
        return t;
    };

    if (p.early_table) {
        if (warp == 0 && lane == 0 && mode == 0 && sched_id < total_tiles) {
            // weights of the first tile -> L2 while the predecessor's last tiles leave most SMs idle
            int g = 0;
            TileInfo ti;
            decode(sched_id, g, ti);
            for (int kb = 0; kb < min(ti.num_kb, kAheadBlocks); ++kb) {
                if (kMnMajor && b_mn) break;
                tma_prefetch_2d(&map_b, ti.b_k0 + kb * elem_per_kb, (kSwiGLU && kPair && cta_rank == 1) ? ti.b_row2 : ti.b_row);
                if (kSwiGLU && !kPair) tma_prefetch_2d(&map_b, ti.b_k0 + kb * elem_per_kb, ti.b_row2);
            }
        }
        pdl_wait_predecessor();
        if (!p.hold_successor) pdl_release_successor();
    }

    // An epilogue warp hands an accumulator window back to the MMA issuer: in a pair that is the leader CTA's barrier.
    auto release_window = [&](uint64_t* bar) {
        if constexpr (kPair) {
            if (cta_rank == 0) mbar_arrive(bar);
            else mbar_arrive_cluster(mapa_shared(smem_u32(bar), 0));
        } else {
            mbar_arrive(bar);
        }
    };

    if (warp < C::kFirstEpi) {
        if constexpr (C::kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kSmallRegs));
        if (warp == 0) {
        // ================= TMA producer =================
        {
            int stage = 0, phase = 0, g = 0;
            int issued = 0;  // stages armed so far (saturating), for the drain on the abort path
            int gated_group = -1;
            bool stamped = false;
            TileInfo ti;
            bool ok = true;
            auto hand_out = [&](int tile, int draw) {
                if (!drawn) return tile + sched_stride;
                const int t = min(sched_stride + __shfl_sync(0xffffffffu, draw, 0), total_tiles);
                if (!__all_sync(0xffffffffu, mbar_wait(&tile_free[tslot], tphase ^ 1, abort_flag, limit, note, wait_id(9, tile, 0, tslot)))) {
                    ok = false;
                    return total_tiles;
                }
                if (lane == 0) {
                    s_tile[tslot] = t;
                    mbar_arrive(&tile_full[tslot]);
                }
                __syncwarp();
                if (++tslot == kTileSlots) {
                    tslot = 0;
                    tphase ^= 1;
                }
                return t;
            };
            int drawn_tile = 0;
            const uint32_t full_u32 = smem_u32(full), stage_u32 = smem_u32(stage_base);
            unsigned stage_rows = 0;  // four bits per stage: 32-row pieces of A that are not zero
            for (int tile = sched_id; tile < total_tiles && ok; tile = hand_out(tile, drawn_tile)) {
                if (drawn && lane == 0) drawn_tile = atomicAdd(p.sched, 1);  // used when this tile's loads have been issued
                decode(tile, g, ti);
                if (lane == 0) s_prod_state[1] = tile;
                if (!kWgrad && p.ready != nullptr && ti.group != gated_group) {
                    if (lane == 0) s_prod_state[0] = 1;
                    // the rows of this group come from other GPUs: wait until all of them have landed
                    const unsigned long long want = p.expected[ti.group];
                    if (ld_acquire_sys_u64(p.ready + ti.group) < want) {
                        const long long t0 = clock64();
                        while (ld_acquire_sys_u64(p.ready + ti.group) < want) {
                            if (*abort_flag || clock64() - t0 > limit) {
                                if (!*abort_flag && note != nullptr) atomicCAS(note, 0ull, wait_id(2, tile, 0, ti.group));
                                *abort_flag = 1;
                                ok = false;
                                break;
                            }
                        }
                    }
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    fence_proxy_async();
                    gated_group = ti.group;
                }
                if (p.trace != nullptr && !stamped) {
                    if (lane == 0) atomicMin(&p.trace[0], global_timer_ns());
                    stamped = true;
                }
                // Rows past the end of the group are not fetched when m_ends says where that is; the tensor core sees zeros instead.
                // A stage holds 16 KB of A beside 32 KB of B, and rows that are multiplied for nothing cost power, which lowers the
                // clock (decode, 20 tokens: 177 us for the first GEMM over stale bytes, 142 with all 128 rows fetched, 138 over
                // zeros). One or two copies of 32 rows replace the copy of 128; with three or four the loading lane would fall behind.
                const int valid_rows = max(1, ti.c_row_end - ti.a_row);
                const int edge = (!kPair && mode == 0 && p.m_ends != nullptr && valid_rows <= 2 * kEdgeRows) ? (valid_rows + kEdgeRows - 1) / kEdgeRows : 0;
                if constexpr (kFp8 && !kPair) {
                    // The same for e4m3 operands with everything that does not change from one K block to the next in front of the loop: what the
                    // loading lane needs per K block is part of every stage's round trip.
                    const uint8_t* sfa = kMx ? p.sfa_atoms + (size_t)(ti.a_row >> 7) * (size_t)(p.k / 128) * 512 : nullptr;
                    const uint8_t* sfb = kMx ? p.sfb_atoms + ((size_t)ti.group * (p.n / kBlockN) + ti.nt) * (size_t)(p.k / 128) * (512 * C::kSfBAtoms) : nullptr;
                    const bool whole = edge == 0 && p.m_ends == nullptr;
                    if (note != nullptr && lane == 0) s_prod_state[0] = 2;
                    for (int kb = 0; kb < ti.num_kb; ++kb) {
                        if (!__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1, abort_flag, limit, note, wait_id(1, tile, kb, stage)))) {
                            ok = false;
                            break;
                        }
                        int pieces = kBlockM / kEdgeRows;
                        if (!whole) {
                            // 32-row pieces of A to write: the valid ones, then pieces an earlier tile left in this stage (zeroed by copies from
                            // past the last row, which touch no memory)
                            const int filled = (int)(stage_rows >> (4 * stage)) & 7;
                            if (edge != 0) pieces = max(edge, filled);
                            stage_rows = (stage_rows & ~(7u << (4 * stage))) | ((unsigned)(edge == 0 ? kBlockM / kEdgeRows : edge) << (4 * stage));
                        }
                        if (elect_one()) {
                            const uint32_t bar = full_u32 + stage * 8, sa = stage_u32 + stage * C::kStageBytes, sb = sa + kATileBytes;
                            mbar_expect_tx_at(bar, C::kStageTxBytes - kATileBytes + pieces * (kEdgeRows * kKBlockBytes));
                            tma_load_2d_at(&map_b, bar, sb, kb * 128, ti.b_row);
                            if (kSwiGLU) tma_load_2d_at(&map_b, bar, sb + C::kBTileBytes / 2, kb * 128, ti.b_row2);
                            if (edge == 0) tma_load_2d_at(&map_a, bar, sa, kb * 128, ti.a_row);
                            else
                                for (int j = 0; j < pieces; ++j)
                                    tma_load_2d_at(&map_sfa, bar, sa + j * kEdgeRows * kKBlockBytes, kb * 128, j < edge ? ti.a_row + j * kEdgeRows : p.m_total);
                            if constexpr (kMx) {
                                // scale atoms: [row tile][K block][512] for A, [group][n tile][K block][512] for B
                                bulk_load_1d_at(sb + C::kBTileBytes, sfa + kb * 512, 512, bar);
                                bulk_load_1d_at(sb + C::kBTileBytes + 512, sfb + kb * (512 * C::kSfBAtoms), 512 * C::kSfBAtoms, bar);
                            }
                        }
                        __syncwarp();
                        if (issued < C::kStages) ++issued;
                        if (++stage == C::kStages) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                    continue;
                }
                for (int kb = 0; kb < ti.num_kb; ++kb) {
                    if (lane == 0) s_prod_state[0] = 2;
                    if (!__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1, abort_flag, limit, note, wait_id(1, tile, kb, stage)))) {
                        ok = false;
                        break;
                    }
                    uint8_t* sa = stage_base + (size_t)stage * C::kStageBytes;
                    uint8_t* sb = sa + kATileBytes;
                    if constexpr (kPair) {
                        // both CTAs fill their own stage and signal the LEADER's barrier, which expects the bytes of both
                        const uint32_t leader_full = mapa_shared(smem_u32(&full[stage]), 0);
                        const bool tail = kWgrad && kb == ti.tail_kb;
                        if (elect_one()) {
                            if (cta_rank == 0) mbar_expect_tx(&full[stage], tail ? C::kStageTxBytes : 2 * C::kStageTxBytes);
                            if (tail) tma_load_3d_pair(&map_sfa, leader_full, sa, ti.a_kbase + kb * 64, ti.a_mn0 / 64);
                            else if (kMnMajor && a_mn) tma_load_3d_pair(&map_a, leader_full, sa, ti.a_kbase + kb * 64, ti.a_mn0 / 64);
                            else tma_load_2d_pair(&map_a, leader_full, sa, ti.a_k0 + kb * elem_per_kb, ti.a_row);
                            if (tail) tma_load_3d_pair(&map_sfb, leader_full, sb, ti.b_kbase + kb * 64, ti.b_mn0 / 64);
                            else if (kMnMajor && b_mn) tma_load_3d_pair(&map_b, leader_full, sb, ti.b_kbase + kb * 64, ti.b_mn0 / 64);
                            else
                                tma_load_2d_pair(&map_b, leader_full, sb, ti.b_k0 + kb * elem_per_kb,
                                                 (kSwiGLU && cta_rank == 1) ? ti.b_row2 : ti.b_row);  // SwiGLU: gate half / up half
                            if constexpr (kMx) {
                                // scale atoms as rows of 32-bit words: this CTA's own 128 rows of A, and the whole tile's B columns
                                uint8_t* ssf = sb + C::kBTileBytes;
                                const int nkb = p.k / 128;
                                tma_load_2d_pair(&map_sfa, leader_full, ssf, 0, (ti.a_row >> 7) * nkb + kb);
                                tma_load_2d_pair(&map_sfb, leader_full, ssf + 512, 0, (ti.group * (p.n / kBlockN) + ti.nt) * nkb + kb);
                            }
                        }
                        __syncwarp();
                        if (issued < C::kStages) ++issued;
                        if (++stage == C::kStages) {
                            stage = 0;
                            phase ^= 1;
                        }
                        continue;
                    }
                    if (lane == 0) s_prod_state[0] = 3;
                    // 32-row pieces of A to write: the valid ones, then pieces an earlier tile left in this stage (zeroed by copies from
                    // past the last row, which touch no memory)
                    const int filled = (int)(stage_rows >> (4 * stage)) & 7;
                    const int pieces = edge == 0 ? kBlockM / kEdgeRows : max(edge, filled);
                    stage_rows = (stage_rows & ~(7u << (4 * stage))) | ((unsigned)(edge == 0 ? kBlockM / kEdgeRows : edge) << (4 * stage));
                    const bool tail = kWgrad && kb == ti.tail_kb;
                    if (elect_one()) {
                        mbar_expect_tx(&full[stage], tail ? C::kStageTxBytes / 2 : C::kStageTxBytes - kATileBytes + pieces * kEdgeRows * kKBlockBytes);
                        // (BF16 from here on)
                        if (tail) tma_load_3d(&map_sfa, &full[stage], sa, ti.a_kbase + kb * 64, ti.a_mn0 / 64);
                        else if (kMnMajor && a_mn) tma_load_3d(&map_a, &full[stage], sa, ti.a_kbase + kb * 64, ti.a_mn0 / 64);
                        else if (edge == 0) tma_load_2d(&map_a, &full[stage], sa, ti.a_k0 + kb * elem_per_kb, ti.a_row);
                        else
                            for (int j = 0; j < pieces; ++j)
                                tma_load_2d(&map_sfa, &full[stage], sa + j * kEdgeRows * kKBlockBytes, ti.a_k0 + kb * elem_per_kb,
                                            j < edge ? ti.a_row + j * kEdgeRows : p.m_total);
                        if (tail) {
                            tma_load_3d(&map_sfb, &full[stage], sb, ti.b_kbase + kb * 64, ti.b_mn0 / 64);
                        } else if (kMnMajor && b_mn) {
                            tma_load_3d(&map_b, &full[stage], sb, ti.b_kbase + kb * 64, ti.b_mn0 / 64);
                        } else if (kSwiGLU) {
                            tma_load_2d(&map_b, &full[stage], sb, ti.b_k0 + kb * elem_per_kb, ti.b_row);
                            tma_load_2d(&map_b, &full[stage], sb + C::kBTileBytes / 2, ti.b_k0 + kb * elem_per_kb, ti.b_row2);
                        } else {
                            tma_load_2d(&map_b, &full[stage], sb, ti.b_k0 + kb * elem_per_kb, ti.b_row);
                        }
                    }
                    __syncwarp();
                    if (issued < C::kStages) ++issued;
                    if (++stage == C::kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (drawn && lane == 0) {  // the last CTA to stop drawing leaves the counter as it was found
                __threadfence();
                if (atomicAdd(p.sched + 1, 1) == (int)gridDim.x - 1) {
                    p.sched[1] = 0;
                    atomicExch(p.sched, 0);
                }
            }
            // Own copies in flight land in this CTA's shared memory: before the CTA may exit, wait (bounded) for every stage
            // that was armed but whose completion this lane has not yet seen. `stage`/`phase` point at the next stage to
            // fill, so the kStages stages before it are the candidates, each with the phase it was armed in.
            if (!ok) {
                if (kPair && cta_rank == 1) {
                    // the peer's copies signal the leader's barriers, which this CTA cannot poll: give them a fixed grace time
                    const long long t0 = clock64();
                    while (clock64() - t0 < 400000) {
                    }
                } else {
                    int st = stage, ph = phase;
                    for (int i = 0; i < C::kStages && i < issued; ++i) {
                        if (--st < 0) {
                            st = C::kStages - 1;
                            ph ^= 1;
                        }
                        const long long t0 = clock64();
                        while (!mbar_try_wait(&full[st], ph) && clock64() - t0 < limit) {
                        }
                    }
                }
            }
        }
        } else if (warp == 1) {
        // ================= MMA issuer =================
        if (cta_rank == 0 && elect_one()) {
            const uint32_t idesc_full = kMx ? make_idesc_mx(kBlockN, C::kTileRows) : make_idesc<kFp8>(kBlockN, C::kTileRows, a_mn, b_mn);
            const uint32_t idesc_half = make_idesc<kFp8>(kBlockN / 2, C::kTileRows, a_mn, b_mn);
            // bytes (in 16-byte units) one K = 16 step moves the operand's start address: 32 B inside the swizzle atom when K
            // is contiguous, 16 K-steps of 128 B when the rows are
            const uint64_t a_kstep = a_mn ? 128 : 2, b_kstep = b_mn ? 128 : 2;
            int sf_buf = 0;  // native block scaling: which set of scale columns
            int stage = 0, phase = 0, g = 0;
            int win = 0, win_phase = 0;  // accumulator window ring
            TileInfo ti;
            bool ok = true;
            for (int tile = sched_id; tile < total_tiles && ok; tile = next_tile_alone(tile)) {
                decode(tile, g, ti);
                if (ti.num_kb == 0) continue;  // epilogue writes zeros on its own
                const uint32_t idesc = (C::kRagged && ti.n_cols != kBlockN) ? idesc_half : idesc_full;
                for (int kb = 0; kb < ti.num_kb; ++kb) {
                    const bool new_window = C::kPromote ? true : (kb == 0);
                    if (new_window) {
                        if (!(mbar_wait(&tmem_empty[win], win_phase ^ 1, abort_flag, limit, note, wait_id(3, tile, kb, win)))) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                    }
                    if (!(mbar_wait(&full[stage], phase, abort_flag, limit, note, wait_id(4, tile, kb, stage)))) {
                        if (note != nullptr) atomicCAS(note + 1, 0ull, ((unsigned long long)s_prod_state[0] << 32) | (unsigned)s_prod_state[1]);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(stage_base) + (uint32_t)(stage * C::kStageBytes);
                    const uint32_t sb = sa + kATileBytes;
                    const uint64_t adesc = a_mn ? make_smem_desc_mn(sa) : make_smem_desc(sa);
                    const uint64_t bdesc = b_mn ? make_smem_desc_mn(sb) : make_smem_desc(sb);
                    const uint32_t tmem_d = tmem_base + (uint32_t)(win * kBlockN);
                    const bool window_done = C::kPromote ? true : (kb == ti.num_kb - 1);
                    {
                        if constexpr (kMx) {
                            // scale atoms of this stage -> TMEM (alternating column sets), then four K=32 MMAs that read them
                            const uint32_t ssf = sb + C::kBTileBytes;
                            const uint32_t t_sfa = tmem_base + (uint32_t)(C::kSfCol0 + sf_buf * C::kSfColsPerBuf), t_sfb = t_sfa + 4;
                            if constexpr (kPair) {
                                tmem_cp_sf_pair(t_sfa, make_sf_desc(ssf));
#pragma unroll
                                for (int at = 0; at < C::kSfBAtoms; ++at) tmem_cp_sf_pair(t_sfb + 4 * at, make_sf_desc(ssf + 512 + 512 * at));
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    umma_mx_pair(tmem_d, adesc + (uint64_t)(j * 2), bdesc + (uint64_t)(j * 2), idesc, t_sfa, t_sfb,
                                                 (new_window && j == 0) ? 0u : 1u);
                            } else {
                                tmem_cp_sf(t_sfa, make_sf_desc(ssf));
#pragma unroll
                                for (int at = 0; at < C::kSfBAtoms; ++at) tmem_cp_sf(t_sfb + 4 * at, make_sf_desc(ssf + 512 + 512 * at));
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    umma_mx(tmem_d, adesc + (uint64_t)(j * 2), bdesc + (uint64_t)(j * 2), idesc, t_sfa, t_sfb,
                                            (new_window && j == 0) ? 0u : 1u);
                            }
                        } else {
                            auto step_at = [&](uint64_t adesc, uint64_t bdesc, int j) {
                                // +32 bytes along K inside the swizzle atom = +2 in the 16-byte start-address field
                                if constexpr (kPair)
                                    umma_pair<kFp8>(tmem_d, adesc + (uint64_t)j * a_kstep, bdesc + (uint64_t)j * b_kstep, idesc,
                                                    (new_window && j == 0) ? 0u : 1u);
                                else
                                    umma<kFp8>(tmem_d, adesc + (uint64_t)j * a_kstep, bdesc + (uint64_t)j * b_kstep, idesc,
                                               (new_window && j == 0) ? 0u : 1u);
                            };
                            auto step = [&](int j) { step_at(adesc, bdesc, j); };
                            // 16 K steps per MMA; those behind the last row of a weight gradient are left out, as are whole blocks of 64 (decode): both weight
                            // gradients of 64 experts of 4096 -> 1408, us, in a loop: 190 rows 781 -> 726, 384 rows 1065 -> 1044, 768 rows 1649 -> 1605.
                            // (Whole blocks keep their straight line of four: an MMA behind a branch costs three times as much to issue.)
                            if (kWgrad && kb == ti.tail_kb) {
                                const uint64_t at = make_smem_desc_mn(sa, kTailRows * 128), bt = make_smem_desc_mn(sb, kTailRows * 128);
                                step_at(at, bt, 0);
                                if (ti.k_rows - kb * 64 > 16) step_at(at, bt, 1);
                            } else if (kMnMajor && mode == 1 && ti.k_rows - kb * 64 <= 48) {
                                step(0);
                                if (ti.k_rows - kb * 64 > 16) step(1);
                                if (ti.k_rows - kb * 64 > 32) step(2);
                            } else {
#pragma unroll
                                for (int j = 0; j < 4; ++j) step(j);
                            }
                        }
                        // smem stage reusable once these MMAs have read it (in both CTAs of a pair)
                        if constexpr (kPair) {
                            umma_commit_pair(smem_u32(&empty[stage]));
                            umma_commit_pair(mapa_shared(smem_u32(&empty[stage]), 1));
                        } else {
                            umma_commit(&empty[stage]);
                        }
                        if (window_done) {
                            if constexpr (kPair) {
                                umma_commit_pair(smem_u32(&tmem_full[win]));
                                umma_commit_pair(mapa_shared(smem_u32(&tmem_full[win]), 1));
                            } else {
                                umma_commit(&tmem_full[win]);
                            }
                        }
                    }
                    sf_buf ^= 1;
                    if (window_done) {
                        if (++win == C::kWindows) {
                            win = 0;
                            win_phase ^= 1;
                        }
                    }
                    if (++stage == C::kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
        __syncwarp();
        }
    } else {
        // ================= epilogue =================
        if constexpr (C::kMoveRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kEpiRegs));
        const int q = warp & 3;                    // TMEM lane quarter this warp may read
        const int half = (warp - C::kFirstEpi) >> 2;          // FP8 only: which half of the columns this warp promotes
        const int row_in_tile = q * 32 + lane;
        int4* out_stage = reinterpret_cast<int4*>(out_stage_base + (size_t)(warp - C::kFirstEpi) * C::kOutStageBytes);
        int g = 0, win = 0, win_phase = 0;
        int xch_iter = 0;  // split drain: tiles whose row maxima went through the exchange so far
        (void)xch_iter;
        TileInfo ti;
        bool ok = true;
        __nv_bfloat16* cbase = reinterpret_cast<__nv_bfloat16*>(p.c);
        const int ldc = mode == 0 ? (kSwiGLU ? p.n / 2 : p.n) : p.k;
        const bool scatter = !kSwiGLU && mode == 0 && p.row_info != nullptr;
        // Maximum over a row's 128 columns, whose other 64 are the partner warp's of this quarter: the two exchange theirs through shared memory,
        // tagged with the tile's number, two tile parities.
        auto row_maximum = [&](float& amax, int tile) {
            const int par = xch_iter & 1;
            ++xch_iter;
            const unsigned tag = (unsigned)tile + 1u;
            xch[(par * 2 + half) * kBlockM + row_in_tile] = ((unsigned long long)tag << 32) | __float_as_uint(amax);
            volatile unsigned long long* other = xch + (par * 2 + (half ^ 1)) * kBlockM + row_in_tile;
            unsigned long long w = *other;
            bool there = true;
            if ((unsigned)(w >> 32) != tag) {
                const long long t0 = clock64();
                while ((unsigned)((w = *other) >> 32) != tag) {
                    if (*abort_flag || clock64() - t0 > limit) {
                        if (!*abort_flag && note != nullptr) atomicCAS(note, 0ull, wait_id(7, tile, 0, warp));
                        *abort_flag = 1;
                        there = false;
                        break;
                    }
                }
            }
            amax = fmaxf(amax, __uint_as_float((unsigned)w));
            return __all_sync(0xffffffffu, there) != 0;
        };
        (void)row_maximum;
        const bool direct = (reinterpret_cast<uintptr_t>(p.c) & 31) == 0;  // (rows are multiples of 256 bytes apart)
        for (int tile = sched_id; tile < total_tiles && ok; tile = next_tile(tile)) {
            decode(tile, g, ti);
            const int row = ti.c_row + row_in_tile;
            __nv_bfloat16* crow = cbase + (size_t)row * ldc + ti.c_col;
            // scatter epilogue: this lane's row goes to row (word & 0xffffff) of the matrix at scatter_bases[word >> 24]
            __nv_bfloat16* scat_ptr = nullptr;
            if (scatter && row < ti.c_row_end) {
                const int word = p.row_info[row];
                if (word >= 0)
                    scat_ptr = reinterpret_cast<__nv_bfloat16*>(p.scatter_bases[word >> 24]) + (size_t)(word & 0xffffff) * ldc + ti.c_col;
            }
            if (ti.num_kb == 0) {
                __nv_bfloat16* zrow = scatter ? scat_ptr : crow;
                if (row < ti.c_row_end && half == 0 && zrow != nullptr)
                    for (int c = 0; c < (C::kRagged ? ti.n_cols : C::kOutCols); c += 8) *reinterpret_cast<int4*>(zrow + c) = make_int4(0, 0, 0, 0);
                continue;
            }
            if constexpr (C::kWidePromote) {
                // 256 columns: a warp promotes 128 of them, with SwiGLU 64 gate columns and the matching up columns, else one scale block. A K
                // block costs its hand-overs (stage, window, scales) once for twice the columns, and twice the weights are on their way.
                const int num_kscales = p.k / 128, n_blocks = p.n / 128;
                const int c0 = half * (kSwiGLU ? 64 : 128), c1 = kSwiGLU ? 128 + half * 64 : half * 128 + 64;
                const float* sa_row = p.a_scales + (size_t)min(row, p.m_total - 1) * num_kscales;
                const float* sb0 = p.b_scales + ((size_t)ti.group * n_blocks + ti.nblock + (kSwiGLU ? 0 : half)) * num_kscales;
                const float* sb1 = p.b_scales + ((size_t)ti.group * n_blocks + ti.nblock2) * num_kscales;
                const bool warp_has_rows = ti.c_row + q * 32 < ti.c_row_end;  // else it only keeps the windows moving
                float acc[2][64];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 64; ++i) acc[h][i] = 0.f;
                // scales are fetched two K blocks ahead: with one an L2 round trip under load is part of every block
                float s_next[3] = {0.f, 0.f, 0.f}, s_far[3] = {0.f, 0.f, 0.f};
                auto fetch_scales = [&](int kb, float (&s)[3]) {
                    if (kb >= ti.num_kb) return;
                    s[0] = __ldcg(sa_row + kb);
                    s[1] = __ldg(sb0 + kb);
                    if (kSwiGLU) s[2] = __ldg(sb1 + kb);
                };
                if (warp_has_rows && p.ready == nullptr) {  // (with arrival gating the rows' scales are there after the first wait: see below)
                    fetch_scales(0, s_next);
                    fetch_scales(1, s_far);
                }
                for (int kb = 0; kb < ti.num_kb; ++kb) {
                    if (!mbar_wait(&tmem_full[win], win_phase, abort_flag, limit, note, wait_id(5, tile, kb, warp))) {
                        ok = false;
                        break;
                    }
                    if (warp_has_rows) {
                        if (kb == 0 && p.ready != nullptr) {
                            fetch_scales(0, s_next);
                            fetch_scales(1, s_far);
                        }
                        tc_fence_after();
                        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(win * kBlockN);
                        uint32_t v[2][32];
                        tmem_ld32(taddr + c0, v[0]);
                        const float s0 = s_next[0] * s_next[1], s1 = kSwiGLU ? s_next[0] * s_next[2] : s0;
#pragma unroll
                        for (int i = 0; i < 3; ++i) s_next[i] = s_far[i];
                        fetch_scales(kb + 2, s_far);
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            tmem_ld_wait();
                            if (c < 3) {  // the next 32 columns are on their way while these are added
                                tmem_ld32(taddr + (c + 1 < 2 ? c0 + 32 : c1 + (c - 1) * 32), v[(c + 1) & 1]);
                            } else {
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0) release_window(&tmem_empty[win]);
                            }
#pragma unroll
                            for (int i = 0; i < 32; ++i) acc[c / 2][(c & 1) * 32 + i] = fmaf(__uint_as_float(v[c & 1][i]), c < 2 ? s0 : s1, acc[c / 2][(c & 1) * 32 + i]);
                        }
                    } else {
                        __syncwarp();
                        if (lane == 0) release_window(&tmem_empty[win]);
                    }
                    if (++win == C::kWindows) {
                        win = 0;
                        win_phase ^= 1;
                    }
                }
                if (!ok) break;
                // Straight on, without branches: while a warp is here the tensor core runs two K blocks ahead at most, and a jump to instructions that
                // were last fetched a tile ago takes some 800 cycles. 64 experts of 4096 -> 1408, 73 rows: 7400 -> 3000 cycles a tile with SwiGLU, 8000 -> 1500
                // without; a K block 1430 -> 1150 with the columns below read ahead. Both products, us: 73 rows 227 / 223, 300 rows (second) 245 / 216.
                if (warp_has_rows) {
                    __nv_bfloat16* mine = scatter ? scat_ptr : row < ti.c_row_end ? crow : nullptr;
                    if (mine != nullptr) mine += half * (kSwiGLU ? 64 : 128);
                    auto columns = [&](int c, int4 (&regs)[4]) {
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            float o[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) o[j] = kSwiGLU ? silu(acc[0][(c + i + j) & 63]) * acc[1][(c + i + j) & 63] : acc[c / 64][(c + i + j) & 63];
                            regs[i / 8] = pack8_bf16(o);
                        }
                    };
                    bool quantised = false;
                    if constexpr (kSwiGLU) {
                        if (p.c_fp8 != nullptr) {
                            // the 128 output columns are one scale block of the next product's activations: what a cast of the BF16 rows would write
                            quantised = true;
                            int4 keep[8];
                            float amax = 0.f;
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                int4 regs[4];
                                columns(c * 32, regs);
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    keep[c * 4 + i] = regs[i];
                                    const uint32_t w4[4] = {(uint32_t)regs[i].x, (uint32_t)regs[i].y, (uint32_t)regs[i].z, (uint32_t)regs[i].w};
#pragma unroll
                                    for (int t = 0; t < 4; ++t) {
                                        const float2 f = bf16x2_to_f2(w4[t]);
                                        amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
                                    }
                                }
                            }
                            ok = row_maximum(amax, tile);
                            if (!ok) break;
                            float scale, inv;
                            fp8_scale_from_amax(amax, false, scale, inv);
                            int4 q8[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                uint32_t out[4];
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    const int4 v = keep[2 * i + h];
                                    const float2 f0 = bf16x2_to_f2((uint32_t)v.x), f1 = bf16x2_to_f2((uint32_t)v.y);
                                    const float2 f2 = bf16x2_to_f2((uint32_t)v.z), f3 = bf16x2_to_f2((uint32_t)v.w);
                                    out[2 * h] = pack_e4m3x4(f0.x * inv, f0.y * inv, f1.x * inv, f1.y * inv);
                                    out[2 * h + 1] = pack_e4m3x4(f2.x * inv, f2.y * inv, f3.x * inv, f3.y * inv);
                                }
                                q8[i] = make_int4((int)out[0], (int)out[1], (int)out[2], (int)out[3]);
                            }
                            const bool row_there = row < ti.c_row_end;
                            uint8_t* dst = row_there ? p.c_fp8 + (size_t)row * ldc + ti.c_col + half * 64 : nullptr;
                            // 64 bytes per row, like 32 BF16 columns
                            RowPair(reinterpret_cast<__nv_bfloat16*>(dst), lane).store(q8, 0);
                            if (half == 0 && row_there) p.c_scales[(size_t)row * (ldc / 128) + (ti.c_col >> 7)] = scale;
                        }
                    }
                    if (quantised) {
                    } else if (__all_sync(0xffffffffu, (reinterpret_cast<uintptr_t>(mine) & 31) == 0)) {
                        const RowPair rows(mine, lane);
#pragma unroll
                        for (int c = 0; c < (kSwiGLU ? 64 : 128); c += 32) {
                            int4 regs[4];
                            columns(c, regs);
                            rows.store(regs, c);
                        }
                    } else if (mine != nullptr) {
#pragma unroll
                        for (int c = 0; c < (kSwiGLU ? 64 : 128); c += 32) {
                            int4 regs[4];
                            columns(c, regs);
#pragma unroll
                            for (int i = 0; i < 4; ++i) reinterpret_cast<int4*>(mine + c)[i] = regs[i];
                        }
                    }
                }
            } else if constexpr (C::kPromote) {
                // One window per K block, promoted into fp32 registers with the two scales. A warp owns two 32-column
                // chunks: with SwiGLU a gate chunk and the matching up chunk, otherwise two neighbouring chunks.
                constexpr int kLo0 = 0, kHalfCols = kBlockN / 2;
                const int c_lo = kSwiGLU ? half * 32 : half * kHalfCols;
                const int c_hi = kSwiGLU ? kHalfCols + half * 32 : half * kHalfCols + 32;
                (void)kLo0;
                float acc[64];
#pragma unroll
                for (int i = 0; i < 64; ++i) acc[i] = 0.f;
                const int num_kscales = p.k / 128;
                const int n_blocks = p.n / 128;
                const float* sa_row = p.a_scales + (size_t)min(row, p.m_total - 1) * num_kscales;
                const float* sb0 = p.b_scales + ((size_t)ti.group * n_blocks + ti.nblock) * num_kscales;
                const float* sb1 = p.b_scales + ((size_t)ti.group * n_blocks + ti.nblock2) * num_kscales;
                // A warp whose 32 rows all lie past the end of the group (masked low-latency layout: a handful of valid rows
                // per expert) only keeps the window ring moving; it promotes nothing.
                const bool warp_has_rows = ti.c_row + q * 32 < ti.c_row_end;
                // Scales are fetched two K blocks ahead: loaded right before their window's wait they put an L2 round trip into
                // every K block as soon as the promotion, not the loads, is the slower side (64 experts of 4096 -> 1408, 128 rows each:
                // first / second GEMM 194 / 103 -> 187 / 93 us; 768 rows each: 1066 / 550 -> 1008 / 523 us). With arrival gating the activation
                // scales are written by other GPUs during this kernel, and only the accumulator hand-over orders this warp after
                // the loader's acquire of the group's arrival counter: the first loads then come after the tile's first wait.
                float s_cur[3] = {0.f, 0.f, 0.f}, s_next[3] = {0.f, 0.f, 0.f}, s_far[3] = {0.f, 0.f, 0.f};
                auto fetch_scales = [&](int kb, float (&s)[3]) {
                    if (kb >= ti.num_kb) return;
                    s[0] = __ldcg(sa_row + kb);
                    s[1] = __ldg(sb0 + kb);
                    if (kSwiGLU) s[2] = __ldg(sb1 + kb);
                };
                if (warp_has_rows && p.ready == nullptr) {
                    fetch_scales(0, s_next);
                    fetch_scales(1, s_far);
                }
                for (int kb = 0; kb < ti.num_kb; ++kb) {
                    if (!warp_has_rows) {
                        if (!mbar_wait(&tmem_full[win], win_phase, abort_flag, limit, note, wait_id(7, tile, kb, warp))) {
                            ok = false;
                            break;
                        }
                        __syncwarp();
                        if (lane == 0) release_window(&tmem_empty[win]);
                        if (++win == C::kWindows) {
                            win = 0;
                            win_phase ^= 1;
                        }
                        continue;
                    }
                    if (!mbar_wait(&tmem_full[win], win_phase, abort_flag, limit, note, wait_id(5, tile, kb, warp))) {
                        ok = false;
                        break;
                    }
                    if (kb == 0 && p.ready != nullptr) {
                        fetch_scales(0, s_next);
                        fetch_scales(1, s_far);
                    }
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        s_cur[i] = s_next[i];
                        s_next[i] = s_far[i];
                    }
                    fetch_scales(kb + 2, s_far);
                    const float s_lo = s_cur[0] * s_cur[1], s_hi = kSwiGLU ? s_cur[0] * s_cur[2] : s_lo;
                    tc_fence_after();
                    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(win * kBlockN);
                    uint32_t v[32], u[32];
                    tmem_ld32(taddr + c_lo, v);
                    tmem_ld32(taddr + c_hi, u);
                    tmem_ld_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) release_window(&tmem_empty[win]);  // the window is free as soon as it sits in registers
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        acc[i] = fmaf(__uint_as_float(v[i]), s_lo, acc[i]);
                        acc[32 + i] = fmaf(__uint_as_float(u[i]), s_hi, acc[32 + i]);
                    }
                    if (++win == C::kWindows) {
                        win = 0;
                        win_phase ^= 1;
                    }
                }
                if (!ok) break;
                {
                    // rows of this warp: ti.c_row + q*32 .. +32; the block base is row 0 of the warp
                    __nv_bfloat16* wbase = cbase + (size_t)(ti.c_row + q * 32) * ldc + ti.c_col;
                    const int rows_valid = min(32, ti.c_row_end - (ti.c_row + q * 32));
                    if constexpr (kSwiGLU) {
                        int4 regs[4];
#pragma unroll
                        for (int c = 0; c < 32; c += 8) {
                            float o[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) o[i] = silu(acc[c + i]) * acc[32 + c + i];
                            regs[c / 8] = pack8_bf16(o);
                        }
                        store_block_coalesced<32>(out_stage, regs, wbase + half * 32, ldc, rows_valid, lane);
                    } else {
                        int4 regs[8];
#pragma unroll
                        for (int c = 0; c < 64; c += 8) regs[c / 8] = pack8_bf16(&acc[c]);
                        if (scatter) store_block_scattered<64>(out_stage, regs, scat_ptr != nullptr ? scat_ptr + half * kHalfCols : nullptr, lane);
                        else store_block_coalesced<64>(out_stage, regs, wbase + half * kHalfCols, ldc, rows_valid, lane);
                    }
                }
            } else {
                if (!mbar_wait(&tmem_full[win], win_phase, abort_flag, limit, note, wait_id(6, tile, 0, warp))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(win * kBlockN);
                __nv_bfloat16* wbase = cbase + (size_t)(ti.c_row + q * 32) * ldc + ti.c_col;
                const int rows_valid = min(32, ti.c_row_end - (ti.c_row + q * 32));
                if constexpr (kSwiGLU && C::kWindows == 1) {
                    // Single window, two warps per lane quarter: this warp takes 64 of the tile's 128 output columns. Their gate
                    // and up accumulators go to registers raw, the window returns to the MMA issuer right away, and the
                    // arithmetic and the stores run while the next tile accumulates.
                    uint32_t v[2][32], u[2][32];
                    tmem_ld32(taddr + half * 64, v[0]);
                    tmem_ld32(taddr + half * 64 + 32, v[1]);
                    tmem_ld32(taddr + kBlockN / 2 + half * 64, u[0]);
                    tmem_ld32(taddr + kBlockN / 2 + half * 64 + 32, u[1]);
                    tmem_ld_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) release_window(&tmem_empty[win]);
                    int4 keep[2][4];
#pragma unroll
                    for (int ci = 0; ci < 2; ++ci)
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            float o[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) o[j] = silu(__uint_as_float(v[ci][i + j])) * __uint_as_float(u[ci][i + j]);
                            keep[ci][i / 8] = pack8_bf16(o);
                        }
                    if constexpr (kMx) {
                        if (p.c_fp8 != nullptr) {
                            // The tile's 128 output columns are exactly one scale block of the next GEMM's activation operand: quantise
                            // here (same arithmetic as the standalone cast applied to the BF16 values: power-of-two scale from the
                            // row's amax) and write e4m3 + the UE8M0 atom word. The row's other 64 columns sit in the partner warp
                            // of this quarter; the two exchange their maxima through shared memory, tagged with the tile number.
                            float amax = 0.f;
#pragma unroll
                            for (int ci = 0; ci < 2; ++ci)
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const int4 v4 = keep[ci][j];
                                    const uint32_t w4[4] = {(uint32_t)v4.x, (uint32_t)v4.y, (uint32_t)v4.z, (uint32_t)v4.w};
#pragma unroll
                                    for (int t = 0; t < 4; ++t) {
                                        const float2 f = bf16x2_to_f2(w4[t]);
                                        amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
                                    }
                                }
                            ok = row_maximum(amax, tile);
                            if (!ok) break;
                            float scale, inv;
                            fp8_scale_from_amax(amax, true, scale, inv);
                            int4 q8[4];
#pragma unroll
                            for (int ci = 0; ci < 2; ++ci)
#pragma unroll
                                for (int jj = 0; jj < 2; ++jj) {
                                    uint32_t outw[4];
#pragma unroll
                                    for (int h2 = 0; h2 < 2; ++h2) {
                                        const int4 v4 = keep[ci][jj * 2 + h2];
                                        const float2 f0 = bf16x2_to_f2((uint32_t)v4.x), f1 = bf16x2_to_f2((uint32_t)v4.y);
                                        const float2 f2 = bf16x2_to_f2((uint32_t)v4.z), f3 = bf16x2_to_f2((uint32_t)v4.w);
                                        outw[h2 * 2] = pack_e4m3x4(f0.x * inv, f0.y * inv, f1.x * inv, f1.y * inv);
                                        outw[h2 * 2 + 1] = pack_e4m3x4(f2.x * inv, f2.y * inv, f3.x * inv, f3.y * inv);
                                    }
                                    q8[ci * 2 + jj] = make_int4((int)outw[0], (int)outw[1], (int)outw[2], (int)outw[3]);
                                }
                            // 64 bytes per row go out like 32 BF16 columns: whole row pieces per store instruction
                            uint8_t* obase = p.c_fp8 + (size_t)(ti.c_row + q * 32) * ldc + ti.c_col + half * 64;
                            store_block_coalesced<32>(out_stage, q8, reinterpret_cast<__nv_bfloat16*>(obase), ldc / 2, rows_valid, lane);
                            if (half == 0 && row < ti.c_row_end) {
                                const uint32_t ex = (__float_as_uint(scale) >> 23) & 0xffu;
                                *reinterpret_cast<uint32_t*>(p.c_atoms + ((size_t)(row >> 7) * (ldc / 128) + (ti.c_col >> 7)) * 512 + (row & 31) * 16 +
                                                             ((row >> 5) & 3) * 4) = ex * 0x01010101u;
                            }
                            win_phase ^= 1;
                            continue;
                        }
                    }
#pragma unroll
                    for (int ci = 0; ci < 2; ++ci) store_block_coalesced<32>(out_stage, keep[ci], wbase + half * 64 + ci * 32, ldc, rows_valid, lane);
                    win_phase ^= 1;  // kWindows == 1: the same window, next phase
                    continue;
                } else if constexpr (kSwiGLU) {
#pragma unroll 1
                    for (int c = 0; c < C::kOutCols; c += 32) {
                        uint32_t v[32], u[32];
                        tmem_ld32(taddr + c, v);
                        tmem_ld32(taddr + kBlockN / 2 + c, u);
                        tmem_ld_wait();
                        int4 regs[4];
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            float o[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) o[j] = silu(__uint_as_float(v[i + j])) * __uint_as_float(u[i + j]);
                            regs[i / 8] = pack8_bf16(o);
                        }
                        store_block_coalesced<32>(out_stage, regs, wbase + c, ldc, rows_valid, lane);
                    }
                } else if constexpr (C::kSplitDrain) {
                    // 256-column tile, single window, two warps per lane quarter: this warp takes 128 of the columns. They go to
                    // registers raw, the window returns to the MMA issuer, then every row leaves as one 256-byte piece (to the
                    // output matrix, or with the scatter epilogue to the row its info word names).
                    uint32_t v[4][32];
#pragma unroll
                    for (int c4 = 0; c4 < 4; ++c4) tmem_ld32(taddr + half * 128 + c4 * 32, v[c4]);
                    tmem_ld_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) release_window(&tmem_empty[win]);
                    int4 regs[16];
#pragma unroll
                    for (int c4 = 0; c4 < 4; ++c4)
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            float o[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) o[j] = __uint_as_float(v[c4][i + j]);
                            regs[c4 * 4 + i / 8] = pack8_bf16(o);
                        }
                    __nv_bfloat16* dst = scatter ? (scat_ptr != nullptr ? scat_ptr + half * 128 : nullptr) : (row < ti.c_row_end ? crow + half * 128 : nullptr);
                    store_rows_256(out_stage, regs, dst, lane);
                    win_phase ^= 1;  // kWindows == 1: the same window, next phase
                    continue;
                } else if constexpr (kRowScatter) {
                    // the tile's 128 columns of every row leave as one 256-byte piece: both halves go through the staging buffer
                    // (32 rows x 16 pieces of 16 bytes, XOR-swizzled), then each store instruction covers two whole rows
                    __syncwarp();
#pragma unroll 1
                    for (int c = 0; c < 128; c += 64) {
                        uint32_t v[32], u[32];
                        tmem_ld32(taddr + c, v);
                        tmem_ld32(taddr + c + 32, u);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            float o[8], o2[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                o[j] = __uint_as_float(v[i + j]);
                                o2[j] = __uint_as_float(u[i + j]);
                            }
                            out_stage[lane * 16 + ((c / 8 + i / 8) ^ (lane & 15))] = pack8_bf16(o);
                            out_stage[lane * 16 + ((c / 8 + 4 + i / 8) ^ (lane & 15))] = pack8_bf16(o2);
                        }
                    }
                    __syncwarp();
                    const unsigned long long mine = reinterpret_cast<unsigned long long>(scat_ptr);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int r2 = i * 2 + (lane >> 4), piece = lane & 15;
                        const int4 val = out_stage[r2 * 16 + (piece ^ (r2 & 15))];
                        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(__shfl_sync(0xffffffffu, mine, r2));
                        if (dst != nullptr) *reinterpret_cast<int4*>(dst + piece * 8) = val;
                    }
                } else {
                    const RowPair rows(row < ti.c_row_end ? crow : nullptr, lane);
#pragma unroll 1
                    for (int c = 0; c < (C::kRagged ? ti.n_cols : C::kOutCols); c += 64) {
                        uint32_t v[32], u[32];
                        tmem_ld32(taddr + c, v);
                        tmem_ld32(taddr + c + 32, u);
                        tmem_ld_wait();
                        int4 regs[8];
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            float o[8], o2[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                o[j] = __uint_as_float(v[i + j]);
                                o2[j] = __uint_as_float(u[i + j]);
                            }
                            regs[i / 8] = pack8_bf16(o);
                            regs[4 + i / 8] = pack8_bf16(o2);
                        }
                        if (scatter) {
                            store_block_scattered<64>(out_stage, regs, scat_ptr != nullptr ? scat_ptr + c : nullptr, lane);
                        } else if (direct) {
                            rows.store(*reinterpret_cast<const int4(*)[4]>(regs), c);
                            rows.store(*reinterpret_cast<const int4(*)[4]>(regs + 4), c + 32);
                        } else {
                            store_block_coalesced<64>(out_stage, regs, wbase + c, ldc, rows_valid, lane);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) release_window(&tmem_empty[win]);
                if (++win == C::kWindows) {
                    win = 0;
                    win_phase ^= 1;
                }
            }
        }
    }

    if (warp >= C::kFirstEpi) {
        // rows scattered into other GPUs' memory are performed there before this kernel counts as finished
        if (!kWgrad && p.row_info != nullptr) __threadfence_system();
        if (p.trace != nullptr && warp == C::kFirstEpi && lane == 0) atomicMax(&p.trace[1], global_timer_ns());
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (kPair) cluster_sync_all();  // neither CTA leaves while the other may still signal it or read its operands
    if (threadIdx.x == 0 && s_abort && p.error_flag != nullptr) atomicExch(p.error_flag, 1);
    if (warp == 1) {
        tc_fence_after();
        if constexpr (kPair) tmem_dealloc_pair(tmem_base, C::kTmemCols);
        else tmem_dealloc(tmem_base, C::kTmemCols);
    }
}

// ---- host side ------------------------------------------------------------------------------
// Scale atoms as a 2-D tensor of 32-bit words: one row per (tile, K block), `words` words per row (128 per 512-byte atom).
bool make_map_sf(CUtensorMap* map, const void* ptr, uint64_t rows, uint32_t words) {
    EncodeFn fn = get_encode_fn();
    if (fn == nullptr) return false;
    cuuint64_t dims[2] = {words, rows};
    cuuint64_t strides[1] = {(cuuint64_t)words * 4};
    cuuint32_t box[2] = {words, 1};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

template <typename C, typename Kernel>
bool has_registers(Kernel kernel) {
    cudaFuncAttributes attributes;
    if (cudaFuncGetAttributes(&attributes, kernel) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return attributes.numRegs == C::kLaunchRegs;
}

template <int kBlockN, bool kFp8, bool kSwiGLU, bool kPair, bool kMx = false, bool kRowScatter = false, bool kWgrad = false>
cudaError_t launch_impl(const GroupedGemmArgs& a, cudaStream_t stream) {
    using C = Cfg<kBlockN, kFp8, kSwiGLU, kPair, kMx, kRowScatter>;
    CUtensorMap map_a, map_b, map_sfa, map_sfb;
    std::memset(&map_sfa, 0, sizeof(map_sfa));
    std::memset(&map_sfb, 0, sizeof(map_sfb));
    if constexpr (kMx && kPair) {
        const uint64_t nkb = (uint64_t)a.k / 128;
        if (!make_map_sf(&map_sfa, a.sfa_atoms, (((uint64_t)a.m_total + 127) / 128) * nkb, 128) ||
            !make_map_sf(&map_sfb, a.sfb_atoms, (uint64_t)a.num_groups * (a.n / kBlockN) * nkb, 128 * C::kSfBAtoms))
            return cudaErrorInvalidValue;
    }
    if constexpr (!kPair) {  // single CTAs read scale atoms without a map; the slot holds the map of A's partial tiles
        if (a.mode == 0 && a.m_ends != nullptr && !make_map(&map_sfa, a.a, kFp8, (uint64_t)a.m_total, (uint64_t)a.k, kEdgeRows)) return cudaErrorInvalidValue;
    }
    const uint32_t b_box_rows = (kSwiGLU || kPair) ? kBlockN / 2 : kBlockN;
    bool ok;
    if (a.mode == 0) {
        ok = make_map(&map_a, a.a, kFp8, (uint64_t)a.m_total, (uint64_t)a.k, kBlockM) &&
             (a.b_mn ? make_map_mn(&map_b, a.b, (uint64_t)a.num_groups * a.k, (uint64_t)a.n, C::kBRows)  // B given as [G, K, N]
                     : make_map(&map_b, a.b, kFp8, (uint64_t)a.num_groups * a.n, (uint64_t)a.k, b_box_rows));
    } else {
        ok = (a.a_mn ? make_map_mn(&map_a, a.a, (uint64_t)a.m_total, (uint64_t)a.n, kBlockM)   // A given as [M, N_out]
                     : make_map(&map_a, a.a, kFp8, (uint64_t)a.n, (uint64_t)a.m_total, kBlockM)) &&
             (a.b_mn ? make_map_mn(&map_b, a.b, (uint64_t)a.m_total, (uint64_t)a.k, C::kBRows)   // B given as [M, K_out]
                     : make_map(&map_b, a.b, kFp8, (uint64_t)a.k, (uint64_t)a.m_total, b_box_rows));
        if (ok && a.a_mn)  // the maps of scale atoms are free: boxes of a reduction's last rows
            ok = make_map_mn(&map_sfa, a.a, (uint64_t)a.m_total, (uint64_t)a.n, kBlockM, kTailRows) &&
                 make_map_mn(&map_sfb, a.b, (uint64_t)a.m_total, (uint64_t)a.k, C::kBRows, kTailRows);
    }
    if (!ok) return cudaErrorInvalidValue;
    auto kernel = grouped_gemm_kernel<kBlockN, kFp8, kSwiGLU, kPair, kMx, kRowScatter, kWgrad>;
    static bool smem_opted_in[64] = {};  // per device, once: the attribute is sticky (and the registers do not change)
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !smem_opted_in[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmemBytes);
        if (e != cudaSuccess) return e;
        if constexpr (C::kMoveRegs) {  // launched with fewer registers the epilogue would wait for more forever; the choice has asked (wide_promotion_fits)
            if (!has_registers<C>(kernel)) return cudaErrorLaunchOutOfResources;
        }
        if (dev >= 0 && dev < 64) smem_opted_in[dev] = true;
    }
    if constexpr (kPair) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(a.num_sms & ~1), 1, 1);  // whole CTA pairs
        cfg.blockDim = dim3(C::kThreads, 1, 1);
        cfg.dynamicSmemBytes = C::kSmemBytes;
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
        if (cfg.gridDim.x < 2) return cudaErrorInvalidValue;
        return cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, map_sfa, map_sfb, a);
    } else {
        return launch_dependent(kernel, dim3(a.num_sms), C::kThreads, C::kSmemBytes, stream, map_a, map_b, map_sfa, map_sfb, a);
    }
}

// kPair chosen at run time (GroupedGemmArgs::cta_pairs)
template <int kBlockN, bool kFp8, bool kSwiGLU, bool kWgrad = false>
cudaError_t launch_sel(const GroupedGemmArgs& a, cudaStream_t stream) {
    if (a.cta_pairs) return launch_impl<kBlockN, kFp8, kSwiGLU, true, false, false, kWgrad>(a, stream);
    return launch_impl<kBlockN, kFp8, kSwiGLU, false, false, false, kWgrad>(a, stream);
}

}  // namespace

bool wide_promotion_fits(bool swiglu) {
    if (swiglu) {  // (once each: every device runs the same code)
        static const bool fits = has_registers<Cfg<256, true, true, false>>(grouped_gemm_kernel<256, true, true, false>);
        return fits;
    }
    static const bool fits = has_registers<Cfg<256, true, false, false>>(grouped_gemm_kernel<256, true, false, false>);
    return fits;
}

cudaError_t launch_grouped_gemm(const GroupedGemmArgs& a, cudaStream_t stream) {
    if (a.num_groups < 1 || a.num_groups > kMaxGroups || a.num_sms < 1) return cudaErrorInvalidValue;
    // MN-major operands: bf16, no swiglu, single CTAs or pairs (the caller's choice); mode 0 takes B that way (input gradients read the weight in place),
    // mode 1 takes both (weight gradients read the output gradient and the activation in place)
    if ((a.a_mn || a.b_mn) && (a.fp8 || a.swiglu || (a.mode == 0 && a.a_mn) || (a.mode == 1 && !(a.a_mn && a.b_mn)) || a.n % 64 != 0))
        return cudaErrorInvalidValue;
    if (a.m_total <= 0) return cudaSuccess;
    const int kb = a.fp8 ? 128 : 64;
    if (a.mode == 0) {
        if (a.k % kb != 0) return cudaErrorInvalidValue;
        if (a.fp8 && a.sfa_atoms != nullptr) {
            // native block scaling: pre-built UE8M0 scale atoms, every group starts on a multiple of 128 rows
            if (a.sfb_atoms == nullptr || a.k % 128 != 0 || a.n % 128 != 0) return cudaErrorInvalidValue;
            if (a.swiglu) {
                if ((a.n / 2) % 128 != 0) return cudaErrorInvalidValue;  // gate/up halves start on scale-block boundaries
                if (a.mx_wide && a.cta_pairs) return launch_impl<256, true, true, true, true>(a, stream);
                if (a.mx_wide) return launch_impl<256, true, true, false, true>(a, stream);
                return launch_impl<128, true, true, false, true>(a, stream);
            }
            if (a.mx_wide) return (a.n % 256 == 0) ? launch_impl<256, true, false, false, true>(a, stream) : cudaErrorInvalidValue;
            if (a.row_info != nullptr) return launch_impl<128, true, false, false, true, true>(a, stream);
            return launch_impl<128, true, false, false, true>(a, stream);
        }
        if (a.fp8) {
            if (a.a_scales == nullptr || a.b_scales == nullptr || a.k % 128 != 0) return cudaErrorInvalidValue;
            if (a.swiglu) {
                if ((a.n / 2) % 128 != 0) return cudaErrorInvalidValue;  // gate/up halves must start on scale-block boundaries
                if (wide_promotion(a)) return launch_impl<256, true, true, false>(a, stream);
                if (a.c_fp8 != nullptr) return cudaErrorInvalidValue;  // (a narrow tile holds half of a scale block)
                return launch_sel<128, true, true>(a, stream);
            }
            if (a.n % 128 != 0) return cudaErrorInvalidValue;
            if (!a.scatter_to_peers && wide_promotion(a)) return launch_impl<256, true, false, false>(a, stream);
            return launch_sel<128, true, false>(a, stream);
        }
        if (a.swiglu) {
            if ((a.n / 2) % 128 == 0) return launch_sel<256, false, true>(a, stream);
            if ((a.n / 2) % 64 == 0) return launch_sel<128, false, true>(a, stream);
            return cudaErrorInvalidValue;
        }
        // MN-major B: 256-column tiles with one half-width tile at the end beat 128-column tiles (input gradient of 53248 rows with 64
        // experts of 4096 x 1408: 815 -> 635 us); K-major boxes would reach into the next expert's rows, so those stay at 128
        if (a.n % 256 == 0 || (a.b_mn && a.n > 256 && a.n % 128 == 0)) return launch_sel<256, false, false>(a, stream);
        if (a.n % 128 == 0) return launch_sel<128, false, false>(a, stream);
        return cudaErrorInvalidValue;
    }
    // K-grouped (weight gradients), bf16 only
    if (a.fp8 || a.swiglu || a.n % kBlockM != 0) return cudaErrorInvalidValue;
    if (a.k % 128 != 0) return cudaErrorInvalidValue;
    if (a.a_mn) {
        // 256-column tiles as above (weight gradient of the same layer: 880 -> 680 us; with 128 rows per expert 216 -> 201 us)
        if (a.k >= 256) return launch_sel<256, false, false, true>(a, stream);
        return launch_sel<128, false, false, true>(a, stream);
    }
    if (a.k % 256 == 0) return launch_sel<256, false, false>(a, stream);
    return launch_sel<128, false, false>(a, stream);
}

}  // namespace dx
