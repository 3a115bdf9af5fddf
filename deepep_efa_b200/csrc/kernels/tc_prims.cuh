// What the expert GEMM kernels share: inline PTX for mbarriers, TMA, TMEM and tcgen05 (sm_100a only), shared-memory and instruction
// descriptors, bounded waits, and the tensor maps.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "gemm_api.h"
#include "prims.cuh"
#include "sigmoid.cuh"

namespace dx {

namespace {

constexpr int kBlockM = 128;
constexpr int kKBlockBytes = 128;      // one 128B swizzle atom per row
constexpr int kATileBytes = kBlockM * kKBlockBytes;  // 16 KiB
constexpr int kTileSlots = 2;          // tiles the loader may hand to the other roles ahead of time
constexpr int kMaxGroups = 1024;

// ---- PTX wrappers ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: returns false (and raises the CTA abort flag) when the limit runs out or another role
// has already aborted.
// `note` (optional, device memory) keeps the first wait that gave up: `what` = (role code << 56 | tile << 24 | k block << 8 | slot).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, long long limit,
                                          unsigned long long* note = nullptr, unsigned long long what = 0) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (*abort_flag) return false;
        if (clock64() - t0 > limit) {
            *abort_flag = 1;
            if (note != nullptr) atomicCAS(note, 0ull, what);
            return false;
        }
    }
    return true;
}
// True in one lane of a converged warp. The loader and the issuer run their loops with the whole warp and leave only the issue of
// TMA copies and tcgen05 instructions to this lane.
__device__ __forceinline__ bool elect_one() {
    uint32_t yes;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(yes));
    return yes != 0;
}
__device__ __forceinline__ unsigned long long wait_id(int role, int tile, int kb, int slot) {
    return ((unsigned long long)role << 56) | ((unsigned long long)(tile & 0xffffffff) << 24) | ((unsigned long long)(kb & 0xffff) << 8) |
           (unsigned long long)(slot & 0xff);
}

__device__ __forceinline__ void tma_load_2d(const CUtensorMap* map, uint64_t* bar, void* dst, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int c0, int c1) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1) : "memory");
}
// The same with shared-memory addresses as they are: inside loops that issue copies every K block the conversion of pointers counts.
__device__ __forceinline__ void mbar_expect_tx_at(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d_at(const CUtensorMap* map, uint32_t bar, uint32_t dst, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}
// An MN-major operand tile in one copy: its chunks of 64 rows are the third dimension of the map (see make_map_mn).
__device__ __forceinline__ void tma_load_3d(const CUtensorMap* map, uint64_t* bar, void* dst, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Kernels allocate tensor memory in front of their wait for the predecessor, and an allocation blocks, without a limit, until the columns are free. Were a CTA
// of the predecessor still to allocate on the same SM, each would wait for the other; a predecessor's other warps may release the successor before that. So no
// two of these kernels share an SM: each takes at least this much of its 228 KB of shared memory (1 KB more per CTA is the system's).
constexpr size_t kTensorKernelSmem = 114 * 1024;
static_assert(2 * (kTensorKernelSmem + 1024) > 228 * 1024, "two kernels with tensor memory must not fit one SM");

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
template <bool kFp8>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (kFp8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K-major operand tile in 128B-swizzled shared memory: rows are 128 bytes apart, 8-row groups 1024 bytes
// apart (stride byte offset), descriptor version 1 (Blackwell), layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);   // start address, 16-byte units
    d |= (uint64_t)1 << 16;                        // leading byte offset (unused with swizzle)
    d |= (uint64_t)(1024 >> 4) << 32;              // stride byte offset
    d |= (uint64_t)1 << 46;                        // descriptor version
    d |= (uint64_t)2 << 61;                        // SWIZZLE_128B
    return d;
}
// MN-major operand tile (the tensor's contiguous dimension is the tile's row index, not K): the tile is stored as chunks of
// 64 rows; a chunk is 64 K-steps of 128 bytes (64 BF16 row elements), 128B-swizzled in groups of 8 K-steps. Stride byte
// offset = distance between 8-K-step groups (1024), leading byte offset = distance between 64-row chunks (8192).
__device__ __forceinline__ uint64_t make_smem_desc_mn(uint32_t smem_addr, uint32_t chunk_bytes = 8192) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)(chunk_bytes >> 4) << 16;       // leading byte offset: next 64-row chunk
    d |= (uint64_t)(1024 >> 4) << 32;              // stride byte offset: next group of 8 K-steps
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;                        // SWIZZLE_128B
    return d;
}
// Instruction descriptor: fp32 accumulate, M = 128, N = n; bit 15 / 16 = A / B is MN-major instead of K-major.
template <bool kFp8>
__device__ __forceinline__ uint32_t make_idesc(int n, int m = kBlockM, int a_mn = 0, int b_mn = 0) {
    uint32_t d = 0;
    d |= 1u << 4;                          // D format = F32
    d |= (kFp8 ? 0u : 1u) << 7;            // A format: E4M3 (f8f6f4) or BF16 (f16)
    d |= (kFp8 ? 0u : 1u) << 10;           // B format
    d |= (a_mn ? 1u : 0u) << 15;           // A major
    d |= (b_mn ? 1u : 0u) << 16;           // B major
    d |= (uint32_t)(n >> 3) << 17;         // N / 8
    d |= (uint32_t)(m >> 4) << 24;         // M / 16 (256 for a CTA pair)
    return d;
}

// ---- CTA pairs (cta_group::2): two CTAs of a cluster share one 256-row MMA; each stages its own 128 rows of A and HALF
// of the B tile, so the bytes every SM pulls from L2 per FLOP drop by a third. No load here is a multicast: each CTA's TMA
// writes only its own shared memory and signals the leader CTA's mbarrier.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t cta_rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta_rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(const CUtensorMap* map, uint32_t bar_cluster_addr, void* dst, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(const CUtensorMap* map, uint32_t bar_cluster_addr, void* dst, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(0), "r"(c1), "r"(c2)
        : "memory");
}
// The same with the shared-memory address as it is.
__device__ __forceinline__ void tma_load_2d_pair_at(const CUtensorMap* map, uint32_t bar_cluster_addr, uint32_t dst, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair_at(const CUtensorMap* map, uint32_t bar_cluster_addr, uint32_t dst, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t addr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint32_t bar_cluster_addr) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr) : "memory");
}
template <bool kFp8>
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (kFp8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}

// ---- native block scaling (kind::mxf8f6f4.block_scale): UE8M0 scale factors live in TMEM, one byte per 32 K-elements and
// row. A 128-row x 128-K scale tile is a 512-byte atom in shared memory: the byte of row (m0 + 32*m1), K sub-block kb sits at
// m0*16 + m1*4 + kb; tcgen05.cp moves it to four TMEM columns (lane m0, column m1, byte kb), replicated to all four lane
// quarters. With one scale per 128 K-elements the four bytes of a word are equal.
__device__ __forceinline__ void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src),
                 "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void bulk_load_1d_at(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// 32 rows of 16 bytes, contiguous: no swizzle, 8-row groups 128 bytes apart
__device__ __forceinline__ uint64_t make_sf_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;            // leading byte offset (one 16-byte column only)
    d |= (uint64_t)(128 >> 4) << 32;   // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;            // descriptor version
    return d;                          // layout type 0: no swizzle
}
__device__ __forceinline__ void tmem_cp_sf(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void umma_mx(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
}
// Instruction descriptor of the block-scaled kind: E4M3 operands (format 0), K-major, UE8M0 scales, scale-factor ids 0.
__device__ __forceinline__ uint32_t make_idesc_mx(int n, int m = kBlockM) {
    uint32_t d = 0;
    d |= (uint32_t)(n >> 3) << 17;         // N / 8
    d |= 1u << 23;                         // scale format: E8M0
    d |= (uint32_t)(m >> 4) << 24;         // M / 16 (256 for a CTA pair)
    return d;
}
// CTA-pair forms: one instruction makes BOTH CTAs copy their own scale atoms (same shared-memory offset) into their own TMEM,
// and one MMA covers the 256 rows of the pair; every CTA holds the scale factors of its own 128 rows of A and of ALL columns.
__device__ __forceinline__ void tmem_cp_sf_pair(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void umma_mx_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
}

__device__ __forceinline__ unsigned long long ld_acquire_sys_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
// Orders what this thread observed through ordinary loads (the arrival counter) before its later TMA reads of the rows.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// 32 bytes per lane where `on`; the address is a multiple of 32
__device__ __forceinline__ void st_global_256(void* p, const uint32_t (&v)[8], bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %9, 0;\n\t@p st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n\t}" ::"l"(p), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"((uint32_t)on)
                 : "memory");
}

// Four lanes hold one byte of each of four tokens (byte t of the word) for neighbouring features: afterwards lane j of the four holds
// the four features of token j.
__device__ __forceinline__ uint32_t transpose_bytes_4x4(uint32_t w, int lane) {
    uint32_t o = __shfl_xor_sync(0xffffffffu, w, 1);
    w = __byte_perm(w, o, (lane & 1) ? 0x3715 : 0x6240);
    o = __shfl_xor_sync(0xffffffffu, w, 2);
    return __byte_perm(w, o, (lane & 2) ? 0x3276 : 0x5410);
}

// Rows of group g (mode 0), which starts at row `begin`.
__device__ __forceinline__ int group_rows(const GroupedGemmArgs& p, int g, int begin) {
    if (p.m_ends == nullptr) return max(p.m_offsets[g + 1] - begin, 0);
    return max(p.m_ends_are_counts ? p.m_ends[g] : p.m_ends[g] - begin, 0);
}

// Tile table, by one warp: tile_start[g] = tiles of the groups before g, tile_start[G] = all; tiles(g, first row, rows) says how many a group has.
template <typename Tiles>
__device__ __forceinline__ void build_tile_table(const GroupedGemmArgs& p, int* tile_start, int lane, Tiles&& tiles) {
    const int G = p.num_groups;
    int run = 0;
#pragma unroll 1
    for (int g0 = 0; g0 < G; g0 += 32) {
        const int g = g0 + lane;
        int n = 0;
        if (g < G) {
            const int begin = p.m_offsets[g];
            n = tiles(g, begin, group_rows(p, g, begin));
        }
        const int incl = warp_incl_scan(n);
        if (g < G) tile_start[g] = run + incl - n;
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) tile_start[G] = run;
}

// ---- host side ------------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn get_encode_fn() {
    static EncodeFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeFn>(p);
    }
    return fn;
}

// 2-D row-major [rows, cols] tensor, box = 128 bytes of columns x box_rows rows, 128B swizzle.
bool make_map(CUtensorMap* map, const void* ptr, bool fp8, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    EncodeFn fn = get_encode_fn();
    if (fn == nullptr) return false;
    const uint64_t esz = fp8 ? 1 : 2;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {cols * esz};
    cuuint32_t box[2] = {(cuuint32_t)(kKBlockBytes / esz), box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims,
                          strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Row-major [k_rows, mn_cols] bf16 tensor whose contiguous dimension is the operand's row index (MN-major operand), seen as
// [mn_cols / 64, k_rows, 64]: a box of `box_rows` operand rows x 64 K-steps lands as chunks of 64 rows (8 KiB each, 128B swizzle),
// the order the matrix descriptor expects, in one copy. One copy per 64-row chunk cost the loading lane up to six instructions per
// stage. Chunks past the last column read as zeros and touch no memory.
bool make_map_mn(CUtensorMap* map, const void* ptr, uint64_t k_rows, uint64_t mn_cols, uint32_t box_rows, uint32_t k_steps = 64) {
    EncodeFn fn = get_encode_fn();
    if (fn == nullptr) return false;
    cuuint64_t dims[3] = {64, k_rows, mn_cols / 64};
    cuuint64_t strides[2] = {mn_cols * 2, 128};
    cuuint32_t box[3] = {64, k_steps, box_rows / 64};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

}  // namespace

}  // namespace dx
