// MoE routing and data-movement kernels (all HBM/latency bound, no tensor cores):
//   topk_kernel          softmax + k rounds of warp arg-max, counts per block and expert
//                                                                            (src/moe/moe_topk_kernel.cpp:15-150)
//   count/scatter        stable counting sort of (expert, source_row) pairs, replacing the radix sort,
//                        the binary-search offsets and the index half of expand_input
//                        (src/moe/moe.cpp:119-126, src/moe/moe_topk_kernel.cpp:152-172, :199-201)
//   gather_rows_kernel   expanded_seq_input[dest] = x[permuted_rows[dest] % T]  (:174-213)
//   combine_kernel       out[t] = sum_i w * Y[rev[i*T+t]] + shared[t]           (:215-251)
//   tile_list_kernel     per-expert row ranges -> list of row tiles for the grouped GEMM
#include "moe_kernels.h"
#include "ptx.cuh"

#include <cuda_fp16.h>
#include <stdint.h>

namespace rf {

// Kernels that may start before the one in front of them has finished take what it writes through plain pointers (a load
// from const __restrict__ memory may be moved in front of griddep_wait()).
namespace {

// exp(x), x <= 0, as a fixed sequence of fp32 operations with no fused multiply-add, so a CPU
// restatement reproduces it bit for bit: t = max(x,-80)*log2e; n = rint(t); f = t-n; degree-7
// Horner for 2^f; exact scaling by 2^n.
__device__ __forceinline__ float det_exp(float x) {
    x = fmaxf(x, -80.0f);
    const float t = __fmul_rn(x, 1.4426950408889634f);
    const float n = rintf(t);
    const float f = __fsub_rn(t, n);
    float p = 1.5252733804059840e-05f;
    p = __fadd_rn(__fmul_rn(p, f), 0.0001540353039338161f);
    p = __fadd_rn(__fmul_rn(p, f), 0.0013333558146428443f);
    p = __fadd_rn(__fmul_rn(p, f), 0.009618129107628477f);
    p = __fadd_rn(__fmul_rn(p, f), 0.05550410866482158f);
    p = __fadd_rn(__fmul_rn(p, f), 0.2402265069591007f);
    p = __fadd_rn(__fmul_rn(p, f), 0.6931471805599453f);
    p = __fadd_rn(__fmul_rn(p, f), 1.0f);
    return __uint_as_float(__float_as_uint(p) + (static_cast<int>(n) << 23));   // p in [0.7, 1.42], result normal
}

// The sort's blocks: block b of `n_blocks` holds the items [b * items, (b + 1) * items), those of whole tokens where the
// counts come from topk_kernel.  At most 256 blocks: every block of the scatter reads all blocks' counts.
struct SortBlocks {
    int items, n_blocks;
};
SortBlocks sort_blocks(int n, int least) {
    int per = (n + 255) / 256;
    if (per < least) per = least;
    return {per, (n + per - 1) / per};
}
constexpr int kLeastTokens = 8;         // per block: one warp each
constexpr int kLeastItems = 1024;

// One warp per token row.  Lane l owns experts [l*VPT, (l+1)*VPT); for E < 32 lanes >= E are idle.  A block takes the
// tokens of one sort block and leaves its number of items per expert in block_counts[block][expert] (nullptr: not asked
// for).
// A round's winner is the largest key (fp16 probability, then lower index first) over the warp, by one redux instruction:
// 32768 tokens x 256 experts, top-8 take 41 us (80 with ten shuffles a round).
template <int VPT>
__global__ void __launch_bounds__(1024)
topk_kernel(const __half* scores, int n_tokens, int n_experts, int top_k, int tokens_per_block,
            int* __restrict__ out_index, __half* __restrict__ out_weight, int* __restrict__ source_rows,
            int* __restrict__ block_counts) {
    __shared__ int hist[256];
    griddep_launch_dependents();
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) hist[e] = 0;
    __syncthreads();
    griddep_wait();
    const int lane = threadIdx.x & 31;
    const int first = lane * VPT;
    const bool active = first < n_experts;
    const int t0 = blockIdx.x * tokens_per_block, t1 = min(t0 + tokens_per_block, n_tokens);
    for (int token = t0 + (threadIdx.x >> 5); token < t1; token += blockDim.x >> 5) {
        const __half* row = scores + (size_t)token * n_experts;
        float logit[VPT];
        if (active) {
            if (VPT == 8) {
                const uint4 q = *reinterpret_cast<const uint4*>(row + first);
                const __half* h = reinterpret_cast<const __half*>(&q);
#pragma unroll
                for (int j = 0; j < VPT; ++j) logit[j] = __half2float(h[j]);
            } else {
#pragma unroll
                for (int j = 0; j < VPT; ++j) logit[j] = __half2float(row[first + j]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < VPT; ++j) logit[j] = -65504.0f;
        }
        // row maximum (exact in any order; the reference takes it in fp16, same value)
        float mx = logit[0];
#pragma unroll
        for (int j = 1; j < VPT; ++j) mx = fmaxf(mx, logit[j]);
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));

        float e[VPT];
        float part = 0.f;
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            e[j] = active ? det_exp(__fsub_rn(logit[j], mx)) : 0.f;
            part = (j == 0) ? e[0] : __fadd_rn(part, e[j]);
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) part = __fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, s));
        const float recip = __fdiv_rn(1.0f, part);

        // The selection runs on fp16 probabilities (ties are frequent at fp16 resolution).  They lie in [0, 1], so their
        // bits order like their values; below them the complement of the expert's number, so that of equal ones the lowest
        // wins.  A key of 0 stands for no expert.
        uint32_t key[VPT];
#pragma unroll
        for (int j = 0; j < VPT; ++j)
            key[j] = active ? ((uint32_t)__half_as_ushort(__float2half_rn(__fmul_rn(e[j], recip))) << 16) |
                                  (0xFFFFu - (uint32_t)(first + j))
                            : 0u;
        uint32_t mine = 0;      // lane k holds the k-th winner
        for (int k = 0; k < top_k; ++k) {
            uint32_t best = key[0];
#pragma unroll
            for (int j = 1; j < VPT; ++j) best = max(best, key[j]);
            best = __reduce_max_sync(0xffffffffu, best);
            if (lane == k) mine = best;
#pragma unroll
            for (int j = 0; j < VPT; ++j)
                if (key[j] == best) key[j] = 0u;
        }
        if (lane < top_k) {
            const size_t o = (size_t)token * top_k + lane;
            const int index = (int)(0xFFFFu - (mine & 0xFFFFu));
            out_index[o] = index;
            out_weight[o] = __ushort_as_half((unsigned short)(mine >> 16));
            source_rows[o] = lane * n_tokens + token;
            if (block_counts != nullptr) atomicAdd(&hist[index], 1);
        }
    }
    if (block_counts == nullptr) return;
    __syncthreads();
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) block_counts[blockIdx.x * n_experts + e] = hist[e];
}

constexpr int kSortThreads = 256;       // of a counting block, and of a scatter block with few counts to add up
constexpr int kMaxExperts = 1024;

// block_counts[b * n_experts + e] = number of items of sort block b routed to expert e
__global__ void __launch_bounds__(kSortThreads)
sort_count_kernel(const int* __restrict__ experts, int n_items, int n_experts, int items_per_block,
                  int* __restrict__ block_counts) {
    __shared__ int hist[kMaxExperts];
    for (int e = threadIdx.x; e < n_experts; e += kSortThreads) hist[e] = 0;
    __syncthreads();
    const int lo = blockIdx.x * items_per_block, hi = min(lo + items_per_block, n_items);
    for (int g = lo + threadIdx.x; g < hi; g += kSortThreads) atomicAdd(&hist[experts[g]], 1);
    __syncthreads();
    for (int e = threadIdx.x; e < n_experts; e += kSortThreads) block_counts[blockIdx.x * n_experts + e] = hist[e];
}

// Exclusive sum of v over the first `n` threads' values (n <= blockDim.x, a multiple of 32 threads in the block);
// *total = the sum of all.  Every thread of the block calls it; warp_sums: 33 ints of shared memory.
__device__ __forceinline__ int block_exclusive_sum(int v, int* warp_sums, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    int incl = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, s);
        if (lane >= s) incl += o;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int w = lane < n_warps ? warp_sums[lane] : 0;
        int wi = w;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, wi, s);
            if (lane >= s) wi += o;
        }
        if (lane < n_warps) warp_sums[lane] = wi - w;
        if (lane == 31) warp_sums[32] = wi;
    }
    __syncthreads();
    *total = warp_sums[32];
    return warp_sums[warp] + incl - v;
}

// Row ranges [offsets[g], offsets[g+1]) (shared or global memory) -> list of row tiles (and, first, the tiles of the alt
// group's alt_rows rows).  A group's rows are cut into the fewest tiles of at most kMoeTileRows rows, all of one height (a
// multiple of 16, the step of the MMA's N) but the last: 1056 rows become four tiles of 224 and one of 160, not four of
// 256 and one of 32 whose weight traffic would count in full.  A chunk is a run of at most kMoeChunkTiles consecutive tiles
// of ONE group (a group's tiles are split into equal chunks); the grouped GEMM walks a chunk column block by column block,
// so the pairs that run at the same time share one group's weight column block and the chunk's row tiles.
// Every thread of one block calls it; starts: kMaxTileGroups + 1 ints of shared memory.  The tiles are dealt out over the
// threads, each of which looks its tile's group up (one thread per group took 33 us for a group of 128 tiles).
constexpr int kMaxTileGroups = 1024;        // the alt group included
__device__ void build_tile_list(const int* offsets, int n_groups, int alt_rows, MoeTile* __restrict__ tiles,
                                int* __restrict__ counters, int* starts, int* warp_sums) {
    const int alt = alt_rows > 0 ? 1 : 0, n_sets = n_groups + alt;      // set 0 is the alt group, if there is one
    auto rows_of = [&](int set) { return set < alt ? alt_rows : offsets[set - alt + 1] - offsets[set - alt]; };
    int total = 0;
    for (int base = 0; base < n_sets; base += blockDim.x) {
        const int set = base + (int)threadIdx.x;
        const int n = set < n_sets ? (rows_of(set) + kMoeTileRows - 1) / kMoeTileRows : 0;
        int sum;
        const int before = block_exclusive_sum(n, warp_sums, &sum);
        if (set < n_sets) starts[set] = total + before;
        total += sum;
        __syncthreads();
    }
    if (threadIdx.x == 0) starts[n_sets] = total;
    __syncthreads();
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int lo = 0, hi = n_sets;            // the last set that starts at or before t (sets without tiles start where the
        while (hi - lo > 1) {               // next one does)
            const int mid = (lo + hi) >> 1;
            if (starts[mid] <= t) lo = mid;
            else hi = mid;
        }
        const int start = starts[lo], i = t - start, n = starts[lo + 1] - start;
        const int rows = rows_of(lo), row0 = lo < alt ? 0 : offsets[lo - alt];
        const int height = ((rows + n - 1) / n + 15) & ~15;
        const int n_chunks = (n + kMoeChunkTiles - 1) / kMoeChunkTiles;
        const int size = n / n_chunks, rem = n % n_chunks;      // the first `rem` chunks hold size + 1 tiles
        int c_first, c_size;
        if (i < rem * (size + 1)) {
            c_size = size + 1;
            c_first = i / c_size * c_size;
        } else {
            c_size = size;
            c_first = rem * (size + 1) + (i - rem * (size + 1)) / size * size;
        }
        tiles[t] = MoeTile{lo < alt ? n_groups : lo - alt, row0 + i * height, min(height, rows - i * height),
                           ((start + c_first) << 8) | c_size};
    }
    if (threadIdx.x == 0) counters[0] = total;
    if (threadIdx.x < kMoeItemCounters) counters[1 + threadIdx.x] = 0;
}

// Stable scatter: item g (expert e) of sort block b goes to (items of experts below e) + (items of e in blocks before b) +
// (earlier items of e in b).  Every block adds the counts of all blocks up for itself, which a launch of one block that
// scans them would keep the chip waiting for (65536 counts took it 100 us); block 0 writes first_token_offset and, with
// `tiles`, the row tiles of the grouped GEMMs (build_tile_list).
// 32768 tokens x top-8, 256 experts: 26 us (118 in three launches, and 34 for the tiles).
__global__ void __launch_bounds__(1024)
sort_scatter_kernel(const int* experts, const int* source_rows, const __half* weights, int n_items, int n_experts,
                    int items_per_block, const int* block_counts, int* __restrict__ permuted_experts,
                    int* __restrict__ permuted_rows, int* __restrict__ rev_permuted_rows,
                    __half* __restrict__ expanded_softmax, int* __restrict__ first_token_offset, int alt_rows,
                    MoeTile* __restrict__ tiles, int* __restrict__ counters) {
    // [warps][E] running positions, later the tile list's starts; [E] items of all blocks before this one; [E + 1]
    // items of all blocks, then the experts' offsets
    extern __shared__ int next[];
    const int n_threads = blockDim.x, n_warps = n_threads >> 5;
    int* before = next + n_warps * n_experts;
    int* offsets = before + n_experts;
    __shared__ int warp_sums[33];
    griddep_launch_dependents();
    for (int i = threadIdx.x; i < (n_warps + 2) * n_experts; i += n_threads) next[i] = 0;
    __syncthreads();
    griddep_wait();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_blocks = gridDim.x, block = blockIdx.x;
    // (a thread's share of the counts: one expert and every `slices`-th block, or several experts and every block)
    const int slices = n_experts < n_threads ? n_threads / n_experts : 1;
    for (int i = threadIdx.x; i < slices * n_experts; i += n_threads) {
        const int slice = i / n_experts, e = i - slice * n_experts;
        int all = 0, mine = 0;
#pragma unroll 8
        for (int b = slice; b < n_blocks; b += slices) {
            const int c = block_counts[b * n_experts + e];
            all += c;
            if (b < block) mine += c;
        }
        atomicAdd(&offsets[e], all);
        atomicAdd(&before[e], mine);
    }
    // pass 1: counts per warp of this block; a warp takes consecutive items
    const int lo = block * items_per_block, hi = min(lo + items_per_block, n_items);
    const int per_warp = ((hi - lo + n_warps - 1) / n_warps + 31) & ~31;
    const int w0 = lo + warp * per_warp, w1 = min(w0 + per_warp, hi);
    int* mine = next + warp * n_experts;
    for (int g0 = w0; g0 < w1; g0 += 32) {
        const int g = g0 + lane;
        const int e = g < w1 ? experts[g] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && (peers & ((1u << lane) - 1)) == 0) mine[e] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        const int per = (n_experts + n_threads - 1) / n_threads;          // experts of a thread, consecutive
        const int e0 = min((int)threadIdx.x * per, n_experts), e1 = min(e0 + per, n_experts);
        int items = 0, sum;
        for (int e = e0; e < e1; ++e) items += offsets[e];
        int base = block_exclusive_sum(items, warp_sums, &sum);
        for (int e = e0; e < e1; ++e) {
            const int n = offsets[e];
            offsets[e] = base;
            int run = base + before[e];
            base += n;
            for (int w = 0; w < n_warps; ++w) {
                const int c = next[w * n_experts + e];
                next[w * n_experts + e] = run;
                run += c;
            }
        }
        if (threadIdx.x == 0) offsets[n_experts] = sum;
    }
    __syncthreads();
    // pass 2: ranks inside each group of 32 by match_any, groups in order
    for (int g0 = w0; g0 < w1; g0 += 32) {
        const int g = g0 + lane;
        const int e = g < w1 ? experts[g] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        if (e >= 0) {
            const int pos = mine[e] + __popc(peers & ((1u << lane) - 1));
            const int src = source_rows[g];
            permuted_experts[pos] = e;
            permuted_rows[pos] = src;
            rev_permuted_rows[src] = pos;
            expanded_softmax[pos] = weights[g];
        }
        __syncwarp();
        if (e >= 0 && (peers & ((1u << lane) - 1)) == 0) mine[e] += __popc(peers);
        __syncwarp();
    }
    if (block == 0) {
        for (int e = threadIdx.x; e <= n_experts; e += n_threads) first_token_offset[e] = offsets[e];
        __syncthreads();
        if (tiles != nullptr) build_tile_list(offsets, n_experts, alt_rows, tiles, counters, next, warp_sums);
    }
}

// dest row r <- src row (row_map[r] % row_mod); one 16-byte vector per thread-iteration
__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* src, const int* row_map, int row_mod, int n_rows, int vec_per_row, uint4* dst) {
    griddep_launch_dependents();
    griddep_wait();
    const size_t total = (size_t)n_rows * vec_per_row;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / vec_per_row);
        const int v = (int)(i - (size_t)r * vec_per_row);
        const int s = row_map[r] % row_mod;
        dst[i] = src[(size_t)s * vec_per_row + v];
    }
}

// out[t, :] = fp16( sum_i w_i * Y[rev[i*T+t], :] + S[t, :] ), fp32 accumulation in rank order
template <int MAX_K>
__global__ void __launch_bounds__(256)
combine_kernel(const uint4* y, const uint4* shared_out, const int* rev, const __half* expanded_softmax, int n_tokens,
               int top_k, int vec_per_row, uint4* out) {
    griddep_launch_dependents();
    griddep_wait();
    const int t = blockIdx.x;
    __shared__ int pos_s[MAX_K];
    __shared__ float w_s[MAX_K];
    if (threadIdx.x < top_k) {
        const int pos = rev[threadIdx.x * n_tokens + t];
        pos_s[threadIdx.x] = pos;
        w_s[threadIdx.x] = __half2float(expanded_softmax[pos]);
    }
    __syncthreads();
    for (int v = threadIdx.x; v < vec_per_row; v += blockDim.x) {
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
        // all k row segments are requested before the first is used
        uint4 qv[MAX_K];
#pragma unroll
        for (int i = 0; i < MAX_K; ++i)
            if (i < top_k) qv[i] = y[(size_t)pos_s[i] * vec_per_row + v];
#pragma unroll
        for (int i = 0; i < MAX_K; ++i) {
            if (i >= top_k) continue;
            const uint4 q = qv[i];
            const __half2* h = reinterpret_cast<const __half2*>(&q);
            const float w = w_s[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __half22float2(h[j]);
                acc[2 * j] = fmaf(w, f.x, acc[2 * j]);
                acc[2 * j + 1] = fmaf(w, f.y, acc[2 * j + 1]);
            }
        }
        const uint4 sq = shared_out[(size_t)t * vec_per_row + v];
        const __half2* sh = reinterpret_cast<const __half2*>(&sq);
        uint4 o;
        __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = __half22float2(sh[j]);
            oh[j] = __floats2half2_rn(acc[2 * j] + f.x, acc[2 * j + 1] + f.y);
        }
        out[(size_t)t * vec_per_row + v] = o;
    }
}

// build_tile_list for ranges in global memory; one block, at most kMaxTileGroups groups, the alt group included.
__global__ void __launch_bounds__(1024)
tile_list_kernel(const int* __restrict__ offsets, int n_groups, int alt_rows, MoeTile* __restrict__ tiles,
                 int* __restrict__ counters) {
    __shared__ int starts[kMaxTileGroups + 1], warp_sums[33];
    build_tile_list(offsets, n_groups, alt_rows, tiles, counters, starts, warp_sums);
}

}  // namespace

namespace {
// Launch, with `overlap` as a programmatic dependent of the kernel before it in the stream.
template <class... Params, class... Args>
cudaError_t launch(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream, bool overlap,
                   Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
}  // namespace

cudaError_t moe_topk_launch(const void* scores, int n_tokens, int n_experts, int top_k, void* index, void* weight,
                            void* source_rows, int* block_counts, bool overlap, cudaStream_t stream) {
    const SortBlocks sb = sort_blocks(n_tokens, kLeastTokens);
    const unsigned threads = 32u * (sb.items < 32 ? sb.items : 32);
    const __half* s = static_cast<const __half*>(scores);
    int* oi = static_cast<int*>(index);
    __half* ow = static_cast<__half*>(weight);
    int* sr = static_cast<int*>(source_rows);
    const int vpt = n_experts <= 32 ? 1 : n_experts / 32;
    auto kernel = vpt == 1 ? topk_kernel<1> : vpt == 2 ? topk_kernel<2> : vpt == 4 ? topk_kernel<4> : topk_kernel<8>;
    if (vpt != 1 && vpt != 2 && vpt != 4 && vpt != 8) return cudaErrorInvalidValue;
    return launch(kernel, (unsigned)sb.n_blocks, threads, 0, stream, overlap, s, n_tokens, n_experts, top_k, sb.items, oi, ow,
                  sr, block_counts);
}

size_t moe_permute_scratch_bytes(int n_items, int n_experts) {
    return (size_t)n_experts * (n_items > 0 ? sort_blocks(n_items, kLeastItems).n_blocks : 1) * sizeof(int);
}
size_t moe_topk_counts_bytes(int n_tokens, int n_experts) {
    return (size_t)n_experts * (n_tokens > 0 ? sort_blocks(n_tokens, kLeastTokens).n_blocks : 1) * sizeof(int);
}

cudaError_t moe_permute_launch(const void* experts, const void* source_rows, const void* weights, int n_tokens, int top_k,
                               int n_experts, void* permuted_experts, void* permuted_rows, void* first_token_offset,
                               void* rev_permuted_rows, void* expanded_softmax, void* scratch, bool counted, int alt_rows,
                               MoeTile* tiles, int* counters, bool overlap, cudaStream_t stream) {
    const int n_items = n_tokens * top_k;
    SortBlocks sb;
    int* counts = static_cast<int*>(scratch);
    if (counted) {
        sb = sort_blocks(n_tokens, kLeastTokens);
        sb.items *= top_k;
    } else {
        sb = sort_blocks(n_items, kLeastItems);
        const cudaError_t e = launch(sort_count_kernel, (unsigned)sb.n_blocks, kSortThreads, 0, stream, false,
                                     static_cast<const int*>(experts), n_items, n_experts, sb.items, counts);
        if (e != cudaSuccess) return e;
    }
    // many counts to add up: more threads to do it (the warps' positions have to fit 48 KB of shared memory)
    const unsigned threads = n_experts <= 256 && (size_t)sb.n_blocks * n_experts > 2048 ? 1024 : kSortThreads;
    const size_t smem = ((threads / 32 + 2) * (size_t)n_experts + 1) * sizeof(int);
    return launch(sort_scatter_kernel, (unsigned)sb.n_blocks, threads, smem, stream, overlap && counted,
                  static_cast<const int*>(experts), static_cast<const int*>(source_rows),
                  static_cast<const __half*>(weights), n_items, n_experts, sb.items, counts,
                  static_cast<int*>(permuted_experts), static_cast<int*>(permuted_rows),
                  static_cast<int*>(rev_permuted_rows), static_cast<__half*>(expanded_softmax),
                  static_cast<int*>(first_token_offset), alt_rows, tiles, counters);
}

cudaError_t moe_gather_rows_launch(const void* src, const int* row_map, int row_mod, int n_rows, int row_bytes,
                                   void* dst, int num_sms, bool overlap, cudaStream_t stream) {
    const int vec = row_bytes / 16;
    const size_t total = (size_t)n_rows * vec;
    size_t blocks = (total + 255) / 256;
    const size_t cap = (size_t)num_sms * 16;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) return cudaSuccess;
    return launch(gather_rows_kernel, (unsigned)blocks, 256, 0, stream, overlap, static_cast<const uint4*>(src), row_map,
                  row_mod, n_rows, vec, static_cast<uint4*>(dst));
}

cudaError_t moe_combine_launch(const void* y, const void* shared_out, const int* rev, const void* expanded_softmax,
                               int n_tokens, int top_k, int row_bytes, void* out, bool overlap, cudaStream_t stream) {
    if (n_tokens == 0) return cudaSuccess;
    return launch(combine_kernel<8>, (unsigned)n_tokens, 256, 0, stream, overlap, static_cast<const uint4*>(y),
                  static_cast<const uint4*>(shared_out), rev, static_cast<const __half*>(expanded_softmax), n_tokens, top_k,
                  row_bytes / 16, static_cast<uint4*>(out));
}

cudaError_t moe_tile_list_launch(const int* offsets, int n_groups, int alt_rows, MoeTile* tiles, int* counters,
                                 cudaStream_t stream) {
    tile_list_kernel<<<1, 1024, 0, stream>>>(offsets, n_groups, alt_rows, tiles, counters);
    return cudaGetLastError();
}

}  // namespace rf
