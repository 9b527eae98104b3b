// Internal interface between the C-ABI layer and the MoE kernels.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>

namespace rf {

// ---- routing / data movement (moe_route.cu); `overlap`: programmatic dependent launch
// Row ranges [offsets[g], offsets[g + 1]) -> list of row tiles for the grouped GEMM.  With alt_rows > 0 the list
// starts with the tiles of one more group, number n_groups, of rows [0, alt_rows) of a matrix of its own (the
// shared expert's).  At most alt_rows / kMoeTileRows + rows / kMoeTileRows + n_groups + 1 tiles.
struct MoeTile {
    int group;      // weight set
    int row0;       // first row
    int rows;       // valid rows, 1 .. kMoeTileRows
    int chunk;      // (first tile of the tile's chunk << 8) | tiles in the chunk
};
// counters: [0] = number of tiles, [1 .. kMoeItemCounters] = 0, the item counters of as many grouped GEMMs.
constexpr int kMoeItemCounters = 2;

// block_counts (moe_topk_counts_bytes, or nullptr): the counts that moe_permute_launch needs.
cudaError_t moe_topk_launch(const void* scores, int n_tokens, int n_experts, int top_k, void* index, void* weight,
                            void* source_rows, int* block_counts, bool overlap, cudaStream_t stream);
size_t moe_topk_counts_bytes(int n_tokens, int n_experts);
size_t moe_permute_scratch_bytes(int n_items, int n_experts);
// counted: `scratch` holds the counts that moe_topk_launch left for the same tokens; else it has
// moe_permute_scratch_bytes.  tiles / counters (or nullptr): the
// row tiles of the experts' rows and of alt_rows rows of an alt group, as moe_tile_list_launch gives them.
cudaError_t moe_permute_launch(const void* experts, const void* source_rows, const void* weights, int n_tokens, int top_k,
                               int n_experts, void* permuted_experts, void* permuted_rows, void* first_token_offset,
                               void* rev_permuted_rows, void* expanded_softmax, void* scratch, bool counted, int alt_rows,
                               MoeTile* tiles, int* counters, bool overlap, cudaStream_t stream);
cudaError_t moe_gather_rows_launch(const void* src, const int* row_map, int row_mod, int n_rows, int row_bytes,
                                   void* dst, int num_sms, bool overlap, cudaStream_t stream);
cudaError_t moe_combine_launch(const void* y, const void* shared_out, const int* rev, const void* expanded_softmax,
                               int n_tokens, int top_k, int row_bytes, void* out, bool overlap, cudaStream_t stream);
cudaError_t moe_tile_list_launch(const int* offsets, int n_groups, int alt_rows, MoeTile* tiles, int* counters,
                                 cudaStream_t stream);

// ---- expert-parallel exchange over peer memory (moe_ep.cu)
struct PeerPtrs {
    void* p[8];
};
#ifdef __CUDACC__
// One of the (at most 8) peer pointers, selected without indexing the kernel-parameter struct dynamically
// (which would force a copy of the struct into local memory).
__device__ __forceinline__ void* pick_peer(const PeerPtrs& pp, int q) {
    void* r = pp.p[0];
#pragma unroll
    for (int i = 1; i < 8; ++i)
        if (q == i) r = pp.p[i];
    return r;
}
#endif
// counts_all [world][n_experts] (row s = pairs per global expert on source rank s).  Writes
//   send_base[e]      row, inside the owner rank's receive buffer, of this rank's first pair for expert e
//   recv_offsets[j]   j = 0..n_experts/world: row range of local expert j in this rank's receive buffer
// Row ranges are clipped to `capacity` (rows of the receive buffers); an overflow ORs kDiagEpOverflow into
// the diagnostics word of `status`.
cudaError_t moe_ep_layout_launch(const int* counts_all, int rank, int world, int n_experts, int capacity,
                                 int* send_base, int* recv_offsets, int* status, cudaStream_t stream);
// Copies the token row of every local (token, expert) pair into the owner rank's receive buffer
// (peer stores) and records where it went (pair_rank, pair_row).  With `recv_meta` != nullptr it also
// writes, beside every row it sends, the return address of the row's result: (this rank << 28) | p, p = the
// pair's position in this rank's expert-sorted order (kEpMetaSlotBits bits).
// A pair whose destination row is >= `capacity` is not sent: pair_rank = -1, kDiagEpOverflow is raised, and
// with `drop_fill` != nullptr (this rank's fp16 [n_pairs, row] result matrix) its result row is zeroed.
// `max_blocks` > 0 caps the grid (to leave SMs to a GEMM running beside it).
constexpr int kEpMetaSlotBits = 28;
cudaError_t moe_ep_dispatch_launch(const void* x, const int* permuted_experts, const int* permuted_rows,
                                   const int* first_token_offset, const int* send_base, int n_tokens, int n_pairs,
                                   int row_bytes, int experts_per_rank, int rank, int world, int capacity,
                                   const PeerPtrs& recv_x, const PeerPtrs* recv_meta, int* pair_rank, int* pair_row,
                                   void* drop_fill, int* status, int num_sms, int max_blocks, cudaStream_t stream);
// out[t] = fp16(sum_i w_i * Y_{rank_i}[row_i] + shared[t]) with Y rows read from the owner ranks (peer loads).
cudaError_t moe_ep_combine_launch(const PeerPtrs& y, const void* shared_out, const int* rev, const void* weights,
                                  const int* pair_rank, const int* pair_row, int n_tokens, int top_k, int row_bytes,
                                  void* out, cudaStream_t stream);

// out[i] = fp16(out[i] + add[i]) over n_elems fp16 values (n_elems % 8 == 0)
cudaError_t moe_add_rows_launch(void* out, const void* add, size_t n_elems, int num_sms, cudaStream_t stream);

// Cross-GPU rendezvous through peer memory.  `sync` = every rank's sync area (int32): words [0, 8) are
// arrival flags (slot s is written by rank s), words [8, 8 + world * n_counts) an all-gather area.
// Each rank stores `epoch` into its slot on every peer and waits (bounded) until its own slots hold
// `epoch`; with `counts` != nullptr it first publishes its n_counts values into row `rank` of every
// peer's gather area.  One launch per rank, every rank on its own GPU.
// `from_offsets`: `counts` holds n_counts + 1 ascending offsets and their differences are published.
cudaError_t moe_ep_rendezvous_launch(const PeerPtrs& sync, const int* counts, int n_counts, bool from_offsets,
                                     int rank, int world, int epoch, int* status, cudaStream_t stream);

// ---- grouped fp16 GEMM (moe_gemm.cu)
// plain:  out[r, n] = fp16(X[r,:] . W_g[:, n]); W_g is [K, N] row-major (N contiguous)
// SwiGLU: out[r, n] = fp16(SiLU(fp16(X.Wa_g)) * fp16(X.Wb_g))

// Rows of one tile of the grouped GEMM (the MMA's N), and the largest run of tiles of one group that the grouped
// GEMM walks together (see tile_list_kernel).
constexpr int kMoeTileRows = 256;
constexpr int kMoeChunkTiles = 8;

// Tensor maps of a fp16 row-major [rows, k] matrix whose rows are the GEMM's tokens: box[i] is 16 (i + 1) rows x 64
// columns, so that half a tile of any height is one load.
struct MoeRowMaps {
    CUtensorMap box[kMoeTileRows / 32];
};

struct MoeGemmParams {
    const MoeTile* tiles;       // row tiles (device)
    const int* tile_count;      // [1]
    int* next_item;             // [1] items drawn so far beyond each pair's first; 0 at the launch
    const CUtensorMap* w_maps;  // device array, one tensor map per group (first weight)
    const CUtensorMap* w2_maps; // second weight per group (SwiGLU mode), else unused
    void* out;                  // fp16 [rows, n_out]
    // Group `alt_group` (-1: none) reads its rows from the `alt` maps and writes to alt_out: the shared expert, whose
    // rows are the tokens themselves, runs in the same launch as the routed experts.
    int alt_group;
    void* alt_out;
    // Plain mode only, optional: row r of the result is stored to row (scatter_meta[r] & slot mask) of the
    // fp16 [*, n_out] matrix scatter_dst.p[scatter_meta[r] >> kEpMetaSlotBits] instead of out[r] (peer stores:
    // the expert outputs travel back to the GPUs that own the tokens from the GEMM's own epilogue).
    const int* scatter_meta;
    PeerPtrs scatter_dst;
    int n_out;                  // output columns
    int k;                      // reduction length (multiple of 64)
    int* status;                // device status area (status_words.h)
    int launch_tag;             // tag recorded with an expired wait
};

// x: the operand rows; alt: the alt group's rows.  `num_sms` = most CTAs to launch (two per cluster).
cudaError_t moe_gemm_launch(bool swiglu, const MoeRowMaps& x, const MoeRowMaps& alt, const MoeGemmParams& p,
                            int num_sms, bool overlap, cudaStream_t stream);

// ---- router GEMM (moe_router.cu); tma_w: boxes of n_out rounded up to 16 rows x 64 columns
// out[r, n] = fp16(X[r,:] . W[n,:] + bias[n]); W is [N, K] row-major (K contiguous), N <= 256
struct MoeRouterParams {
    const float* bias;          // optional fp32 [n_out]
    void* out;                  // fp16 [n_rows, n_out]
    int n_rows;
    int n_out;
    int k;
    int tma_store;              // 1: full 32-row slabs leave through the output tensor map
    int* status;
    int launch_tag;
};
cudaError_t moe_router_launch(const CUtensorMap& tma_x, const CUtensorMap& tma_w, const CUtensorMap& tma_out,
                              const MoeRouterParams& p, int num_sms, bool overlap, cudaStream_t stream);

}  // namespace rf
