// Launch API of the grouped expert GEMM (tcgen05 / TMEM / TMA, sm_100a). No torch headers.
//
//   C[m, n] = sum_k A[m, k] * B[n, k]        (both operands K-major, fp32 accumulation in TMEM)
//
// mode 0, "M-grouped" (expert forward and input gradients): A is [M_total, K]; rows
//   [m_offsets[g], m_offsets[g+1]) belong to expert g and use weight block B[g*N : (g+1)*N, :].
//   Group boundaries must be multiples of 128 (dispatch's expert alignment / the permute pads).
// mode 1, "K-grouped" (weight gradients): A is [N_out, M_total], B is [K_out, M_total]; expert g
//   reduces over columns [m_offsets[g], m_offsets[g+1]) and writes C[g*N_out : (g+1)*N_out, :].
//
// Operand types: BF16 (kind::f16) or FP8 e4m3 with DeepSeek-style scales (one fp32 per 1x128 of A and
// per 128x128 of B): every 128-deep K block is accumulated in its own TMEM window and promoted into
// fp32 registers with the product of the two scales.
// swiglu = 1: B holds [gate; up] stacked per expert ([G, 2*I, K]); a tile computes matching gate and up
//   columns and writes silu(gate) * up, so C is [M_total, I].
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace dx {

struct GroupedGemmArgs {
    const void* a;            // operand A (see mode)
    const void* b;            // operand B
    void* c;                  // bf16 output
    const float* a_scales;    // fp8 only: [M_total, K/128]
    const float* b_scales;    // fp8 only: [G, N/128, K/128]
    // fp8 with native block scaling (power-of-two scales; mode 0, group starts on multiples of 128 rows): UE8M0 scale atoms,
    // 512 bytes per (128 rows, 128 K): [ceil(M/128)][K/128][512] and [G][N/128 tiles (swiglu: N/2/64 tiles)][K/128][512];
    // when sfa_atoms is set the fp32 scale pointers are ignored
    const uint8_t* sfa_atoms;
    const uint8_t* sfb_atoms;
    int mx_wide;              // swiglu only: 1 = 256-column tiles (one accumulator window; large groups), 0 = 128-column tiles
    const int* m_offsets;     // [G+1] device memory
    const int* m_ends;        // optional [G]: group g covers rows [m_offsets[g], m_ends[g]) instead of up to m_offsets[g+1]
                              // (the low-latency layout has fixed group starts and a count per expert). mode 1, MN-major operands: the rows
                              // behind it are zero in both, and the reduction may stop there or go over them
    int zero_tail;            // launch_token_pairs_gemm, with m_ends: 1 = rows from m_ends[g] to m_offsets[g+1] are zero in A, and in C they are
                              // written as zeros; 0 = they are not touched
    int m_ends_are_counts;    // 1 = m_ends[g] is the number of rows of group g instead of its end
    int num_groups;
    int mode;                 // 0 = M-grouped, 1 = K-grouped
    int fp8;                  // 0 = bf16 operands, 1 = e4m3 operands (mode 0 only)
    int swiglu;               // mode 0 only
    int m_total;              // rows of A (mode 0) / reduction length (mode 1)
    int n;                    // mode 0: rows of B per expert (2*I when swiglu); mode 1: N_out (rows of A)
    int k;                    // mode 0: reduction length; mode 1: K_out (rows of B)
    int num_sms;              // persistent grid size
    int rows_hint;            // how many rows all groups have together, where that is less than m_total (0 = not known)
    int tile_order;           // mode 0: 0 = weight tile shared by consecutive CTAs, 1 = activation tile shared
    int cta_pairs;            // 1 = two CTAs of a cluster share one 256-row MMA (cta_group::2), each staging half of the B tile
    int narrow_promotion;     // 1 = this build's 256-column promotion cannot run (wide_promotion_fits), 128 columns take its place
    int* error_flag;          // device int, set non-zero when a bounded pipeline wait ran out
    long long timeout_cycles;
    // Arrival gating (mode 0): the rows of group g are written by other GPUs while this kernel runs. Before the first tile
    // of a group is loaded, the loader waits (bounded) until ready[g] >= expected[g]; `ready` is advanced with system-scope
    // release reductions by the senders, `expected` is rank-local. Both null = no gating.
    const unsigned long long* ready;
    const unsigned long long* expected;
    // Scatter epilogue (mode 0, no swiglu): output row m is not stored to c[m] but to row (row_info[m] & 0xffffff) of the
    // [rows, n] bf16 matrix at scatter_bases[row_info[m] >> 24] (a peer's symmetric memory or this GPU's); rows whose word
    // is negative are dropped. Null = ordinary output.
    const int* row_info;
    const unsigned long long* scatter_bases;
    int scatter_to_peers;     // 1 = some of them are other GPUs': pieces of a row should be long (FP8 with fp32 scales keeps tiles that store 128 bytes)
    unsigned long long* trace;  // optional [4]: earliest first-tile load / latest epilogue end (global timer, ns) / first wait that
                                // gave up (role << 56 | tile << 24 | k block << 8 | slot; 0 = none) / what the loader was doing
                                // then (state << 32 | tile; state 1 = arrival gate, 2 = waiting for a free stage, 3 = loads issued; e4m3 single CTAs: 2 from a tile's first wait on)
    // MN-major operands (bf16, no swiglu): the operand is read from a tensor whose contiguous dimension is the operand's row
    // index instead of K, so gradients need no transposed copies. mode 0: b_mn = 1, B given as [G, K, N] (input gradients:
    // the forward weight as it is). mode 1: a_mn = b_mn = 1, A given as [M_total, N_out], B as [M_total, K_out] (weight
    // gradients: output gradient and activation as they are).
    int a_mn, b_mn;
    // Quantised output (natively block-scaled kernel with 256-column SwiGLU tiles only): instead of bf16 rows in `c`, write
    // e4m3 rows [M_total, N/2] to c_fp8 and their power-of-two scales as UE8M0 scale atoms [ceil(M/128)][N/2/128][512] to
    // c_atoms: the activation operand of the next natively block-scaled GEMM, without a cast pass in between.
    uint8_t* c_fp8;
    uint8_t* c_atoms;
    float* c_scales;          // fp32 scales [M_total, N/2/128] instead of atoms, where tiles are promoted in 256 columns; c_fp8 32-byte aligned then
    // Optional [2], zero: tiles are drawn from a counter instead of dealt out in strides (single CTAs only; pairs ignore it). The
    // kernel leaves both words zero. Launches that may run at the same time need words of their own.
    int* sched;
    // 1 = m_offsets and m_ends were final before the kernel in front of this one in the stream began, and that kernel started only
    // after everything before it had ended: the tile table is then built without waiting for it (programmatic dependent launch).
    int early_table;
    // 1 = the next kernel in the stream gets no SM before this one has ended, also where it is a programmatic dependent launch: the SMs
    // that this launch leaves free are meant for another stream.
    int hold_successor;
    int token_pairs;          // the caller's choice: launch_token_pairs_gemm takes this product (gemm_choice.h; never with gates, the scatter epilogue, a
                              // trace, a tile counter, early_table or hold_successor, which that kernel does not have: a traced product takes rows)
    // launch_token_cols_gemm, launch_token_pairs_gemm: tokens of one tile at most (a multiple of 32 from 64 to 224, of 64 up to 256)
    int token_cap;
};

// Returns cudaErrorInvalidValue for unsupported shapes (divisibility rules are in grouped_gemm.cu).
cudaError_t launch_grouped_gemm(const GroupedGemmArgs& args, cudaStream_t stream);
// Whether the compiler gave the 256-column promotion the registers that its warps move between them (another toolkit, -G or -maxrregcount may not).
bool wide_promotion_fits(bool swiglu);
// The same product for groups of few to some hundred rows (gemm_cols.cu): natively block-scaled operands with 256-column weight atoms,
// mode 0, n % 256 == 0; SwiGLU writes c_fp8 and c_atoms, otherwise bf16 rows to c or through the scatter epilogue.
cudaError_t launch_token_cols_gemm(const GroupedGemmArgs& args, cudaStream_t stream);

// BF16 with the tokens as columns on CTA pairs (gemm_pairs.cu): mode 0, B [G, N, K] or with b_mn [G, K, N], n % 128 == 0, k % 64 == 0, any
// group boundaries.
cudaError_t launch_token_pairs_gemm(const GroupedGemmArgs& args, cudaStream_t stream);

// Expert-major plan from local expert ids [N, K] (-1 = unselected) and 128-aligned group offsets [L+1] on the host:
// m_offsets [L+1] (the offsets on the device), m_ends [L] (end of every group's rows in front of its padding), pos [N*K], src_row [m_pad]
// (-1 = padding), src_k [m_pad] (0 there).
constexpr int kPlanMaxExperts = 1024;  // local experts of one launch; the offsets travel as kernel arguments (4 KiB)
cudaError_t launch_build_plan(const int64_t* topk_idx, const int* host_offsets, int* m_offsets, int* m_ends, int* pos, int* src_row, int* src_k,
                              int num_rows, int num_topk, int num_local_experts, cudaStream_t stream);

// Row gathers between receive order and the expert-major, 128-row-aligned layout (permute.cu).
//   dst[m] = scale * src[src_row[m]]   (src_row[m] < 0 -> zero row; scale may be null; bf16 rows when scaled, one scale per row m). Rows
//   are multiples of 4 bytes (of 16 when scaled).
cudaError_t launch_gather_rows(const void* src, void* dst, const int* src_row, const float* scale, int num_dst_rows, int row_bytes,
                               cudaStream_t stream);
// The same without a scale for a plan's two maps: src_row, which decides, and pos [num_src_rows, num_k] (may be null), where each row goes (-1: nowhere).
cudaError_t launch_permute_rows(const void* src, void* dst, const int* pos, const int* src_row, int num_src_rows, int num_k, int num_dst_rows, int row_bytes, cudaStream_t stream);
// Rows of e4m3 with their fp32 scales per 128 channels (hidden % 128 == 0), gathered in one launch: scales as they are [num_dst_rows, hidden/128], or with
// `atoms` as scale atoms (powers of two; whole tiles of 128 rows). Clears the two words at `sched` (may be null), for the products behind it.
cudaError_t launch_gather_quantised(const void* src, const float* src_scales, void* dst, float* scales, uint8_t* atoms, const int* src_row, int num_dst_rows, int hidden,
                                    int* sched, cudaStream_t stream);
//   dst[n] = sum_k w[n,k] * src[pos[n,k]]  (bf16 rows, fp32 accumulate; pos < 0 skipped; w may be null = 1)
cudaError_t launch_gather_reduce_rows(const void* src, void* dst, const int* pos, const float* w, int num_dst_rows, int num_k, int hidden,
                                      cudaStream_t stream);

// Training-step helpers (train_ops.cu). All tensors bf16 unless noted.
//   out[b, c, r] = in[b, r, c]                     rows and cols multiples of 8
cudaError_t launch_transpose_bf16(const void* in, void* out, int batch, int rows, int cols, cudaStream_t stream);
//   h[m, i] = silu(h13[m, i]) * h13[m, inter + i]
cudaError_t launch_logistic(const float* x, float* out, long long n, cudaStream_t stream);
cudaError_t launch_swiglu_fwd(const void* h13, void* h, long long rows, int inter, cudaStream_t stream);
//   dh13 = d/dh13 of the above given dh
cudaError_t launch_swiglu_bwd(const void* h13, const void* dh, void* dh13, long long rows, int inter, cudaStream_t stream);
//   gradient of y[n] = sum_k w[n, k] * a[pos[n, k]]: da[m] = w[n, k] * g[n] for the (n, k) with pos[n, k] = m, 0 where src_row[m] < 0;
//   dw[n, k] = <a[pos[n, k]], g[n]>, 0 where pos < 0
cudaError_t launch_unpermute_bwd(const void* a, const void* g, const float* w, const int* pos, const int* src_row, void* da, float* dw, int n_rows,
                                 int num_k, int m_rows, int hidden, cudaStream_t stream);
//   out[n, k] = <a[pos[n, k]], b[n]>  (f32 out, 0 where pos < 0)
cudaError_t launch_rowdot(const void* a, const void* b, const int* pos, float* out, int n_rows, int num_k, int hidden, cudaStream_t stream);

// Scale atoms of the natively block-scaled FP8 GEMM (sf_atoms.cu); scales must be powers of two.
// With group_counts only the rows r with r % rows_per_group < group_counts[r / rows_per_group] are looked at (rows_per_group % 128 == 0).
cudaError_t launch_build_sfa_atoms(const float* scales, uint8_t* atoms, int rows, int num_kb, const int* group_counts, int rows_per_group,
                                   cudaStream_t stream);
cudaError_t launch_build_sfb_atoms(const float* scales, uint8_t* atoms, int groups, int n, int num_kb, int swiglu, int wide,
                                   cudaStream_t stream);

}  // namespace dx
