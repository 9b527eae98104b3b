// Grouped fp16 GEMM for the MoE layer on sm_100a: per-expert row ranges, no padding rows.
//
// Replaces the hipBLASLt grouped / dense GEMM calls and the separate SwiGLU pass of the reference
// (src/moe/gemm_thirdparty.cpp:65-115, :261-288; src/moe/moe_gemm_pipeline_kernel.cpp:377-405).
//
// The product is computed transposed, out^T = W^T X^T: the weight's columns are the MMA's M and the token rows its N.
// W [K, N] row-major is then an M-major A operand, X [rows, K] a K-major B operand, both as they lie in memory.  A row
// tile has any height up to 256 in steps of 16 (the MMA's N), so a ragged expert pays for the rows it has, and a few
// rows of a decode step cost a 16-wide MMA beside the weight stream instead of a 128-row tile.
//
// One persistent CTA pair (2-CTA cluster) per two SMs, tcgen05.mma.cta_group::2, M = 256: each CTA loads its own 128
// weight columns (SwiGLU: 64 of W_gate and the same 64 of W_up) and half of the token rows, 32 KB per 64-deep K step
// of a full tile for 512 cycles of MMA.  A work item is (row tile, block of output columns); tiles come from a
// device-built list, so per-expert counts never visit the host, and a pair's items after its first from a counter, so
// that the pairs at work at any moment hold neighbouring items.  (Dealt out round-robin, tiles of unequal height let
// the pairs drift apart until they no longer met in L2: 32 groups of about 1024 rows, K = 7168, N = 2 x 2048 read
// 5.84 GB from HBM for 2.35 GB of operands.)  Warps of each CTA:
//   warp 0     TMA producer into a six-stage ring; the leader's barrier counts the bytes of both CTAs; the leader's
//              draws the next item a few K steps before it needs it and tells every role of both CTAs
//   warp 1     (leader CTA) MMA issuer: 4 x tcgen05.mma.kind::f16 per stage, accumulating the whole K range in one of
//              two 256-column TMEM buffers; one multicast commit per stage frees it in both CTAs, one per tile
//              publishes the accumulator
//   warps 4-11 epilogue of the previous tile while the next tile's MMAs run: 32 token rows at a time, tcgen05.ld in
//              mma-fragment layout, fp16 rounding, stmatrix transposed into [row][column] order, then (SwiGLU:
//              SiLU(fp16 G) * fp16 U) whole 128-byte row segments to global memory; rows past the tile's end masked
//
// What bounds it: the tensor pipe under the power cap for large batches, the weight stream from HBM for small ones.
#include "ptx.cuh"
#include "moe_kernels.h"

namespace rf {

namespace {

constexpr int BK = 64;                      // 128 bytes of fp16: one swizzle row
constexpr int UMMA_K = 16;
constexpr int STAGES = 6;
constexpr int W_BYTES = 128 * BK * 2;       // this CTA's 128 weight columns: two boxes [64 K x 64 columns]
constexpr int W_BOX_BYTES = 64 * BK * 2;
constexpr int X_BYTES = 128 * BK * 2;       // this CTA's half of the token rows, at most 128
constexpr int X_ROW_BYTES = BK * 2;
constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
constexpr int NUM_NON_EPI_WARPS = 4;
constexpr int EPI_WARPS = 8;                // two sets of four warps (one per TMEM lane quadrant)
constexpr int THREADS = 32 * (NUM_NON_EPI_WARPS + EPI_WARPS);
constexpr int NBUF = 2;
constexpr int BUF_COLS = kMoeTileRows;      // TMEM columns of one accumulator buffer
constexpr int TMEM_COLS = NBUF * BUF_COLS;
constexpr int EPI_ROWS = 32;                // token rows per epilogue step
constexpr int OUT_SLAB_BYTES = EPI_ROWS * 256;   // [32 rows][128 accumulator lanes] fp16
constexpr int OUT_BYTES = 2 * 2 * OUT_SLAB_BYTES;      // per warp set, double buffered
// Slots of drawn items (a barrier and a number each, in both CTAs).  The producer is at most 8 items ahead of the
// epilogue: with one K step per item, the six stages, plus the two accumulator buffers; so a slot has always been read
// by every role before it is written again.
constexpr int ITEM_SLOTS = 16;
constexpr int DRAW_AHEAD = 12;              // K steps before a tile's end at which the next item is drawn
constexpr int BAR_BYTES = (2 * STAGES + 2 * NBUF + ITEM_SLOTS) * 8 + 4 * ITEM_SLOTS + 16;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + OUT_BYTES + BAR_BYTES + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");

__device__ __forceinline__ float silu_fp16_rounded(float g) {
    // SiLU evaluated in fp32 on an fp16 input, result rounded to fp16 (scripts/problems/moe/reference.py:23)
    const float s = g / (1.0f + __expf(-g));
    return __half2float(__float2half_rn(s));
}

// SiLU(g) * u on a pair of fp16 values
__device__ __forceinline__ uint32_t swiglu_pair(uint32_t g, uint32_t u) {
    const float2 gf = __half22float2(*reinterpret_cast<const __half2*>(&g));
    const float2 uf = __half22float2(*reinterpret_cast<const __half2*>(&u));
    return pack_f16x2(silu_fp16_rounded(gf.x) * uf.x, silu_fp16_rounded(gf.y) * uf.y);
}

// Work item -> (row tile, column block).  Items walk one chunk (up to kMoeChunkTiles row tiles of one
// group, built by tile_list_kernel) for one column block, then the next column block of the same chunk:
// the pairs running at the same time share that group's weight column block, and the chunk's token rows stay
// in L2 across all column blocks.  The chunk of work item w is the chunk of tile w / nbn, because the
// chunks before it hold exactly (first tile of the chunk) * nbn items.
__device__ __forceinline__ MoeTile decode_item(int w, const MoeTile* tiles, int nbn, int* nb) {
    const int info = ld_global_s32(&tiles[w / nbn].chunk);
    const int first = info >> 8;
    const int n = info & 0xff;
    const int r = w - first * nbn;
    *nb = r / n;
    const int4 t = ld_global_v4_s32(tiles + first + r % n);
    return MoeTile{t.x, t.y, t.z, t.w};
}

// MMA N of a tile: its rows rounded up to the step that M = 256 allows
__device__ __forceinline__ int mma_rows(int rows) { return (rows + 15) & ~15; }

template <bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
moe_gemm_kernel(const __grid_constant__ MoeRowMaps x, const __grid_constant__ MoeRowMaps alt, const MoeGemmParams p) {
    constexpr int TILE_N = SWIGLU ? 128 : 256;     // output columns per work item
    constexpr int CTA_N = TILE_N / 2;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t out_base = smem_base + STAGES * STAGE_BYTES;
    const uint32_t bar_base = out_base + OUT_BYTES;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };                 // leader's: bytes of both CTAs
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto tmem_full_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + b); };
    auto tmem_empty_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + NBUF + b); };   // leader's: both CTAs
    // slot of the pair's j-th drawn item, j = 1, 2, ...
    auto item_bar = [&](uint32_t j) { return bar_base + 8u * (2 * STAGES + 2 * NBUF + (j - 1) % ITEM_SLOTS); };
    auto item_slot = [&](uint32_t j) {
        return bar_base + 8u * (2 * STAGES + 2 * NBUF + ITEM_SLOTS) + 4u * ((j - 1) % ITEM_SLOTS);
    };
    const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 2 * NBUF + ITEM_SLOTS) + 4u * ITEM_SLOTS;
    uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    griddep_launch_dependents();
    const int rank = (int)cluster_ctarank();       // 0 = leader of the pair
    const int unit = (int)(blockIdx.x >> 1);
    const int n_units = (int)(gridDim.x >> 1);

    if (threadIdx.x == 0) {
        tma_prefetch_desc(x.box);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < NBUF; ++b) {
            mbar_init(tmem_full_bar(b), 1);
            mbar_init(tmem_empty_bar(b), 2 * EPI_WARPS);
        }
        for (int j = 1; j <= ITEM_SLOTS; ++j) mbar_init(item_bar(j), 1);
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc_2cta(tmem_slot, TMEM_COLS);
        tmem_relinquish_2cta();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();      // both CTAs' barriers exist before any remote arrive, byte count or commit
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot_ptr);

    griddep_wait();      // the tile list, the rows and the counters come from the kernels before this one

    const int nbn = (p.n_out + TILE_N - 1) / TILE_N;
    const int total_work = ld_global_s32(p.tile_count) * nbn;
    const int k_steps = p.k / BK;
    // The j-th item of this pair: the first by its number, the later ones as the leader's producer drew them.
    auto wait_item = [&](uint32_t j) {
        return mbar_wait<true>(item_bar(j), ((j - 1) / ITEM_SLOTS) & 1, p.status, kErrSchedWait, p.launch_tag);
    };

    if (warp == 0) {
        // ------------------------------------------------------ TMA producer
        uint32_t it = 0, j = 0;
        bool ok = true;
        for (int w = unit; w < total_work;) {
            int nb;
            const MoeTile t = decode_item(w, p.tiles, nbn, &nb);
            int drawn = 0;
            const int half = mma_rows(t.rows) >> 1;             // token rows per CTA, a multiple of 8
            const int first = rank * half;                      // of this CTA's rows inside the tile
            const CUtensorMap* mw = p.w_maps + t.group;
            const CUtensorMap* mw2 = SWIGLU ? p.w2_maps + t.group : mw;
            const int n0 = nb * TILE_N + rank * CTA_N;
            const int n1 = SWIGLU ? n0 : n0 + 64;               // columns of the second box
            // one box holds the CTA's rows, or eight more (one load a stage: with boxes of 16 rows, seven for a tile
            // of 224, a layer of 8 x 896 rows took 360 us instead of 318)
            const int box = (half + 15) >> 4;
            const CUtensorMap* mx = (t.group == p.alt_group ? alt.box : x.box) + (box - 1);
            const uint32_t bytes = 2u * (W_BYTES + 16 * box * X_ROW_BYTES);
            const int row0 = t.row0 + first;
            for (int ks = 0; ks < k_steps; ++ks, ++it) {
                const int s = it % STAGES;
                const uint32_t ph = (it / STAGES) & 1;
                // (the counter's answer is first looked at after the tile's last load)
                if (rank == 0 && lane == 0 && ks == max(k_steps - DRAW_AHEAD, 0)) drawn = atomicAdd(p.next_item, 1);
                ok = __all_sync(0xffffffffu, mbar_wait(empty_bar(s), ph ^ 1, p.status, kErrProducerWait, p.launch_tag));
                if (!ok) break;
                const uint32_t sw = smem_base + s * STAGE_BYTES;
                const uint32_t sx = sw + W_BYTES;
                const uint32_t bar = mapa_cluster(full_bar(s), 0);
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(full_bar(s), bytes);
                    tma_load_2d_pair(sw, mw, bar, n0, ks * BK);
                    tma_load_2d_pair(sw + W_BOX_BYTES, mw2, bar, n1, ks * BK);
                    tma_load_2d_pair(sx, mx, bar, ks * BK, row0);
                }
                __syncwarp();
            }
            if (!ok) break;
            ++j;
            if (rank == 0) {
                w = n_units + __shfl_sync(0xffffffffu, drawn, 0);
                if (lane < 2) {
                    st_cluster_u32(mapa_cluster(item_slot(j), lane), (uint32_t)w);
                    mbar_arrive_cluster(mapa_cluster(item_bar(j), lane));
                }
            } else {
                ok = __all_sync(0xffffffffu, wait_item(j));
                if (!ok) break;
                w = (int)ld_shared_u32(item_slot(j));
            }
        }
        // (the leader's commits arrive on this CTA's stage barriers)
        finish_producer(ok, it, STAGES, empty_bar(0), p.status, kErrProducerWait, p.launch_tag);
    } else if (warp == 1 && rank == 0) {
        // -------------------------------------------------------- MMA issuer
        uint32_t it = 0, tcount = 0;
        bool ok = true;
        for (int w = unit; w < total_work;) {
            int nb;
            const MoeTile t = decode_item(w, p.tiles, nbn, &nb);
            const uint32_t idesc = make_idesc(256, mma_rows(t.rows), /*f16*/ 0, /*f16*/ 0, /*A M-major*/ 1, /*B K-major*/ 0);
            const int buf = tcount & 1;
            const uint32_t bph = (tcount >> 1) & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(tmem_empty_bar(buf), bph ^ 1, p.status, kErrMmaWaitTmem, p.launch_tag));
            if (!ok) break;
            const uint32_t d = tmem_base + buf * BUF_COLS;
            for (int ks = 0; ks < k_steps; ++ks, ++it) {
                const int s = it % STAGES;
                const uint32_t ph = (it / STAGES) & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(full_bar(s), ph, p.status, kErrMmaWaitFull, p.launch_tag));
                if (!ok) break;
                tc_fence_after();
                const uint32_t sw = smem_base + s * STAGE_BYTES;
                const uint64_t adesc = smem_desc_mnmajor_sw128(sw, W_BOX_BYTES, 1024);
                const uint64_t bdesc = smem_desc_kmajor_sw128(sw + W_BYTES);
                if (elect_one()) {
#pragma unroll
                    for (int j = 0; j < BK / UMMA_K; ++j)
                        // M-major A: +16 K-rows = 2048 bytes; K-major B: +32 bytes along K
                        umma_f16_2cta(d, adesc + 128 * j, bdesc + 2 * j, idesc, (ks > 0 || j > 0) ? 1u : 0u);
                    umma_commit_2cta_multicast(empty_bar(s), 0x3);
                    if (ks == k_steps - 1) umma_commit_2cta_multicast(tmem_full_bar(buf), 0x3);
                }
                __syncwarp();
            }
            if (!ok) break;
            ++tcount;
            ok = __all_sync(0xffffffffu, wait_item(tcount));
            if (!ok) break;
            w = (int)ld_shared_u32(item_slot(tcount));
        }
    } else if (warp >= NUM_NON_EPI_WARPS) {
        // ---------------------------------------------------------- epilogue
        const int quad = warp & 3;
        const int set = (warp - NUM_NON_EPI_WARPS) >> 2;       // rows 32 * (set, set + 2, ...) of the tile
        const int tid = quad * 32 + lane;                      // thread of the warp set
        const int bar_id = 1 + set;
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
        const uint32_t slab0 = out_base + set * 2 * OUT_SLAB_BYTES;
        // where this lane's stmatrix row address lies: matrix lane / 8 (8 accumulator lanes each), row lane % 8;
        // 16-byte chunks of a 128-byte half row are swizzled by the row
        const int st_chunk = quad * 4 + (lane >> 3);
        const uint32_t st_off = (uint32_t)(lane & 7) * 256u + (uint32_t)(st_chunk >> 3) * 128u +
                                (uint32_t)(((st_chunk & 7) ^ (lane & 7)) << 4);
        uint32_t tcount = 0, steps = 0;
        for (int w = unit; w < total_work;) {
            int nb;
            const MoeTile t = decode_item(w, p.tiles, nbn, &nb);
            const int n_mma = mma_rows(t.rows);
            const int n0 = nb * TILE_N + rank * CTA_N;
            __half* out = static_cast<__half*>(t.group == p.alt_group ? p.alt_out : p.out);
            const bool scatter = !SWIGLU && p.scatter_meta != nullptr;
            const int buf = tcount & 1;
            const uint32_t bph = (tcount >> 1) & 1;
            bool ok = mbar_wait(tmem_full_bar(buf), bph, p.status, kErrEpilogueWait, p.launch_tag);
            // (the next item was announced when this one's last loads were issued)
            ok = ok && wait_item(++tcount);
            // the warps of a set leave the loop together: they meet at barriers below
            ok = named_barrier_all(bar_id, 128, ok);
            if (!ok) break;
            w = (int)ld_shared_u32(item_slot(tcount));
            tc_fence_after();
            const uint32_t tbase = lane_addr + buf * BUF_COLS;

            // this set's last step is the last that reads the accumulator
            int c0 = set * EPI_ROWS;
            bool released = false;
            auto release = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster_relaxed(mapa_cluster(tmem_empty_bar(buf), 0));
                released = true;
            };
            for (; c0 < n_mma; c0 += 2 * EPI_ROWS, ++steps) {
                float a[16], b[16];
                tmem_ld_16x256b_x4_async(tbase + c0, a);
                tmem_ld_16x256b_x4_async(tbase + (16u << 16) + c0, b);
                tmem_ld_wait16(a, b);
                if (c0 + 2 * EPI_ROWS >= n_mma) release();
                const uint32_t slab = slab0 + (steps & 1) * OUT_SLAB_BYTES;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    stmatrix_x4_trans(slab + i * 8 * 256 + st_off, pack_f16x2(a[4 * i], a[4 * i + 1]),
                                      pack_f16x2(a[4 * i + 2], a[4 * i + 3]), pack_f16x2(b[4 * i], b[4 * i + 1]),
                                      pack_f16x2(b[4 * i + 2], b[4 * i + 3]));
                // one barrier per step: the slab of two steps ago was read before its readers reached the last one
                named_barrier(bar_id, 128);
                const int rows_left = t.rows - c0;
                if (SWIGLU) {
                    // 8 lanes per row: 64 output columns
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int r = j * 16 + (tid >> 3), c = tid & 7;
                        const uint32_t src = slab + r * 256 + ((c ^ (r & 7)) << 4);
                        const uint4 g = ld_shared_v4(src);
                        const uint4 u = ld_shared_v4(src + 128);
                        const uint4 o = make_uint4(swiglu_pair(g.x, u.x), swiglu_pair(g.y, u.y), swiglu_pair(g.z, u.z),
                                                   swiglu_pair(g.w, u.w));
                        const int col = n0 + 8 * c;
                        if (r < rows_left && col < p.n_out)
                            *reinterpret_cast<uint4*>(out + (size_t)(t.row0 + c0 + r) * p.n_out + col) = o;
                    }
                } else {
                    // 16 lanes per row: 128 output columns
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int r = j * 8 + (tid >> 4), c = tid & 15;
                        const uint4 o = ld_shared_v4(slab + r * 256 + (c >> 3) * 128 + (((c & 7) ^ (r & 7)) << 4));
                        const int col = n0 + 8 * c;
                        if (r < rows_left && col < p.n_out) {
                            __half* row;
                            if (scatter) {
                                const int meta = p.scatter_meta[t.row0 + c0 + r];
                                row = static_cast<__half*>(pick_peer(p.scatter_dst, meta >> kEpMetaSlotBits)) +
                                      (size_t)(meta & ((1 << kEpMetaSlotBits) - 1)) * p.n_out;
                            } else {
                                row = out + (size_t)(t.row0 + c0 + r) * p.n_out;
                            }
                            *reinterpret_cast<uint4*>(row + col) = o;
                        }
                    }
                }
            }
            if (!released) release();      // (a tile of 32 rows has no step for the second set)
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();      // the peer no longer touches this CTA's barriers, shared memory or TMEM
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_2cta(tmem_base, TMEM_COLS);
    }
}

template <bool SWIGLU>
cudaError_t launch_mode(const MoeRowMaps& x, const MoeRowMaps& alt, const MoeGemmParams& p, int num_sms, bool overlap,
                        cudaStream_t stream) {
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kernel = moe_gemm_kernel<SWIGLU>;
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    const int pairs = num_sms >= 2 ? num_sms / 2 : 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs, 1, 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, x, alt, p);
}

}  // namespace

cudaError_t moe_gemm_launch(bool swiglu, const MoeRowMaps& x, const MoeRowMaps& alt, const MoeGemmParams& p,
                            int num_sms, bool overlap, cudaStream_t stream) {
    return swiglu ? launch_mode<true>(x, alt, p, num_sms, overlap, stream) : launch_mode<false>(x, alt, p, num_sms, overlap, stream);
}

}  // namespace rf
