// FP8 block-scaled GEMM on CTA pairs for sm_100a (block_n 512: 256 x 256 tiles, 384: 256 x 128).
//
// The product and its fp32 promotion are those of fp8_gemm_kernel (fp8_gemm.cu), K block by K block in the same order,
// so the results are the same bits.  What differs is how a tile is shared out.  One 2-CTA cluster computes a tile with
// cta_group::2 MMAs (M = 256): each CTA loads its own 128 rows of A and half of the tile's rows of B, 32 KB per K block of
// 256 columns instead of the 48 KB of a 128 x 256 tile.  The tile's columns are computed as two halves of HN columns, each
// with accumulator buffers and epilogue warps of its own: the halves' MMAs alternate, so one half's epilogue works while
// the other's waits for its next K block, and a buffer comes back 1.5 K blocks before it is needed (with 256-column
// buffers that both warp groups read in step, 1 K block).  Warps of each CTA:
//   warp 0      TMA producer; the leader's barrier counts the bytes of both CTAs
//   warp 1      (leader CTA) MMA issuer: per K block and half 4 x tcgen05.mma, one multicast commit that publishes the
//               half's buffer; one more that frees the stage in both CTAs
//   warps 2, 3  scales of one half each: the fp32 products a_s * b_s of this CTA's 128 rows, into shared memory
//   warps 4-11  epilogue, four per half: tcgen05.ld, one FMA per element into 128 (64) register accumulators per thread
//
// What bounds it: the power cap on long calls, else the epilogue's K block (barrier, TMEM load, FMAs: about 740 cycles
// where the tensor cores need 512).  Calls one after the other through custom_kernel, one box, two runs each, us, against the
// 128 x 256 tile of fp8_gemm.cu as it is now: 6144 x 4608 x 7168 196.6, 200.3 / 207.9, 207.0; 6144 x 7168 x 2048 102.0,
// 100.3 / 108.5, 108.7; 16384 x 28672 x 7168 3269, 3265 / 3538, 3535.  On the way there, in short runs on another box that gave
// 190.9 and 96.0 us for the first two shapes: producer and issuer as whole warps that vote and elect at every step 222 and
// 113 (their instructions queue behind the epilogue's on the shared schedulers); the scales loaded by the epilogue threads,
// at the cost of registers that spill, 230 and 114; other register splits, without a spill to show for it and for reasons not
// traced, 64 / 216 194 and 96, 120 / 192 277 and 120, 40 / 232 336 and 154.
#include "ptx.cuh"
#include "fp8_gemm.h"
#include "fp8_tiles.cuh"

#include <cstdlib>

namespace rf {

namespace {

constexpr int BM = 128;          // rows per CTA
constexpr int BK = 128;          // one scale block, one 128-byte swizzle row of fp8
constexpr int UMMA_K = 32;
constexpr int NUM_NON_EPI_WARPS = 4;
constexpr int EPI_WARPS = 8;     // four per column half
constexpr int THREADS = 32 * (NUM_NON_EPI_WARPS + EPI_WARPS);
// registers per thread after set-up; 128 * kRegsLo + 256 * kRegsHi is what the CTA was launched with (168 each)
constexpr int kRegsLo = 88, kRegsHi = 208;
static_assert(128 * kRegsLo + 256 * kRegsHi <= 64512, "register split");

// Two fp32 values in a 64-bit register pair, the form the accumulators are kept in.
using F32x2 = unsigned long long;
__device__ __forceinline__ F32x2 pack_f32x2(float lo, float hi) {
    F32x2 r;
    asm volatile("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo_f32(F32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_f32(F32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ void fma_f32x2(F32x2& acc, float x, float y, F32x2 s2) {
    const float2 r = __ffma2_rn(make_float2(x, y), make_float2(lo_f32(s2), hi_f32(s2)), make_float2(lo_f32(acc), hi_f32(acc)));
    acc = (F32x2)__float_as_uint(r.x) | ((F32x2)__float_as_uint(r.y) << 32);
}
__device__ __forceinline__ uint32_t to_bf16x2(F32x2 v) { return pack_bf16x2(lo_f32(v), hi_f32(v)); }

template <int HN_>
struct PairCfg {
    static constexpr int kHN = HN_;                           // columns of a half: one accumulator buffer
    static constexpr int kBN = 2 * HN_;
    static constexpr int kBRows = HN_ / 2;                    // rows of B that this CTA loads for each half
    static constexpr int kABytes = BM * BK;
    static constexpr int kBHalfBytes = kBRows * BK;
    static constexpr int kStageBytes = kABytes + 2 * kBHalfBytes;
    static constexpr int kBufs = 512 / kBN;                   // accumulator buffers of each half
    static constexpr int kChunks = HN_ / 64;                  // 64-column store chunks, one slab each
    static constexpr int kSlabBytes = 32 * 128;
    static constexpr int kStages = HN_ == 128 ? 4 : 6;
    static constexpr int kScaleBytes = 2 * kBufs * BM * 4;    // scale products: one slot beside each accumulator buffer
    static constexpr int kBarBytes = (2 * kStages + 6 * kBufs) * 8 + 16;
    static constexpr int kSmemBytes =
        kStages * kStageBytes + EPI_WARPS * kChunks * kSlabBytes + kScaleBytes + kBarBytes + 1024;
    static_assert(HN_ == 64 || HN_ == 128, "a half holds at most one scale block");
    static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
};

template <class Cfg, bool SPLIT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
fp8_gemm_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                     const __grid_constant__ CUtensorMap tma_c, const __grid_constant__ CUtensorMap tma_p,
                     const __grid_constant__ GemmDestMaps dests, const GemmParams p) {
    constexpr int HN = Cfg::kHN;
    constexpr int STAGES = Cfg::kStages;
    constexpr int NB = Cfg::kBufs;
    constexpr int B_ROWS = Cfg::kBRows;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t slab_base = smem_base + STAGES * Cfg::kStageBytes;
    const uint32_t scale_base = slab_base + EPI_WARPS * Cfg::kChunks * Cfg::kSlabBytes;
    const uint32_t bar_base = scale_base + Cfg::kScaleBytes;
    auto full_bar = [&](uint32_t s) { return bar_base + 8u * s; };                // leader's: bytes of both CTAs
    auto empty_bar = [&](uint32_t s) { return bar_base + 8u * (STAGES + s); };
    auto tmem_full_bar = [&](uint32_t b) { return bar_base + 8u * (2 * STAGES + b); };           // b = half * NB + i
    auto tmem_empty_bar = [&](uint32_t b) { return bar_base + 8u * (2 * STAGES + 2 * NB + b); };  // leader's: both CTAs
    auto scale_empty_bar = [&](uint32_t b) { return bar_base + 8u * (2 * STAGES + 4 * NB + b); };
    const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 6 * NB);
    uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    griddep_launch_dependents();
    const int rank = (int)cluster_ctarank();       // 0 = leader of the pair
    const int unit = (int)(blockIdx.x >> 1);
    const int n_units = (int)(gridDim.x >> 1);

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tma_a);
        tma_prefetch_desc(&tma_b);
        tma_prefetch_desc(SPLIT ? &tma_p : &tma_c);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < 2 * NB; ++b) {
            mbar_init(tmem_full_bar(b), 2);                // the MMAs' commit and the scale warp
            mbar_init(tmem_empty_bar(b), EPI_WARPS);       // four warps of each CTA
            mbar_init(scale_empty_bar(b), EPI_WARPS / 2);  // the half's four
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc_2cta(tmem_slot, 512);
        tmem_relinquish_2cta();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();      // both CTAs' barriers exist before any remote arrive, byte count or commit
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot_ptr);
    griddep_wait();

    const int kb_total = p.k / BK;

    if (warp < NUM_NON_EPI_WARPS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kRegsLo));
        // (The producer and the issuer run on one lane: a step of theirs is a serial chain, and the warps that share their
        // schedulers make every instruction of it dear.)
        if (warp == 0) {
            if (elect_one()) {
                // -------------------------------------------------- TMA producer
                uint32_t it = 0, s = 0, ph = 1;
                bool ok = true;
                PlainWalker walk(p, unit, n_units, kb_total);
                Piece pc;
                while (ok && walk.next(pc, p, n_units, kb_total)) {
                    const TileCoord t = decode_tile(SPLIT ? pc.item / p.splits : pc.item, p.tiles_m, p.tiles_n);
                    const int a_row0 = (t.m_blk * 2 + rank) * BM;
                    const int b_row0 = t.n_blk * Cfg::kBN + rank * B_ROWS;
                    int x = pc.kb0 * BK;
                    for (const uint32_t end = it + (SPLIT ? pc.kb1 - pc.kb0 : kb_total); it != end; ++it, x += BK) {
                        ok = mbar_wait(empty_bar(s), ph, p.status, kErrProducerWait, p.launch_tag);
                        if (!ok) break;
                        const uint32_t sa = smem_base + s * Cfg::kStageBytes;
                        const uint32_t bar = mapa_cluster(full_bar(s), 0);
                        if (rank == 0) mbar_expect_tx(full_bar(s), 2 * Cfg::kStageBytes);
                        tma_load_2d_pair(sa, &tma_a, bar, x, a_row0);
                        tma_load_2d_pair(sa + Cfg::kABytes, &tma_b, bar, x, b_row0);
                        tma_load_2d_pair(sa + Cfg::kABytes + Cfg::kBHalfBytes, &tma_b, bar, x, b_row0 + HN);
                        if (++s == STAGES) { s = 0; ph ^= 1; }
                    }
                }
                // (the leader's commits arrive on this CTA's stage barriers)
                finish_producer(ok, it, STAGES, empty_bar(0), p.status, kErrProducerWait, p.launch_tag);
            }
            __syncwarp();
        } else if (warp == 1) {
            if (rank == 0 && elect_one()) {
                // ---------------------------------------------------- MMA issuer
                constexpr uint32_t idesc = make_idesc(2 * BM, HN, /*e4m3*/ 0, /*e4m3*/ 0, 0, 0);
                const uint64_t desc0 = smem_desc_kmajor_sw128(smem_base);
                uint32_t it = 0, s = 0, ph = 0;
                bool ok = true;
                PlainWalker walk(p, unit, n_units, kb_total);
                Piece pc;
                while (ok && walk.next(pc, p, n_units, kb_total)) {
                    const TileCoord t = decode_tile(SPLIT ? pc.item / p.splits : pc.item, p.tiles_m, p.tiles_n);
                    const bool both = t.n_blk * Cfg::kBN + HN < p.n;        // else the second half has no columns to compute
                    for (const uint32_t end = it + (SPLIT ? pc.kb1 - pc.kb0 : kb_total); it != end; ++it) {
                        const uint32_t buf = it % NB;
                        const uint32_t bph = ((it / NB) & 1) ^ 1;
                        const uint64_t adesc = desc0 + s * (Cfg::kStageBytes / 16);
                        const uint32_t d = tmem_base + buf * HN;
                        ok = mbar_wait(full_bar(s), ph, p.status, kErrMmaWaitFull, p.launch_tag);
                        if (!ok) break;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            ok = mbar_wait(tmem_empty_bar(h * NB + buf), bph, p.status, kErrMmaWaitTmem, p.launch_tag);
                            if (!ok) break;
                            tc_fence_after();
                            const uint64_t bdesc = adesc + (Cfg::kABytes + h * Cfg::kBHalfBytes) / 16;
                            if (h == 0 || both) {
#pragma unroll
                                for (int j = 0; j < BK / UMMA_K; ++j)
                                    umma_f8_2cta(d + h * (NB * HN), adesc + 2 * j, bdesc + 2 * j, idesc, j > 0 ? 1u : 0u);
                            }
                            umma_commit_2cta_multicast(tmem_full_bar(h * NB + buf), 0x3);
                        }
                        if (!ok) break;
                        umma_commit_2cta_multicast(empty_bar(s), 0x3);
                        if (++s == STAGES) { s = 0; ph ^= 1; }
                    }
                }
            }
            __syncwarp();
        } else if (warp >= 2) {
            // ------------------------------------------------------ scales
            // One warp per half: the fp32 products a_s * b_s of this CTA's 128 rows, one K block at a time, into the slot
            // of the block's accumulator buffer.  Its loads run PF K blocks ahead, across tiles.
            const int half = warp - 2;
            constexpr int PF = 4;
            PlainWalker walk(p, unit, n_units, kb_total);
            Piece pc;
            uint32_t ar[4], br = 0;            // element offsets of the rows' and the column block's next scales
            int left = 0;
            auto next_piece = [&] {
                if (!walk.next(pc, p, n_units, kb_total)) return false;
                const TileCoord t = decode_tile(SPLIT ? pc.item / p.splits : pc.item, p.tiles_m, p.tiles_n);
                const int col0 = t.n_blk * Cfg::kBN + half * HN;
                const int row0 = (t.m_blk * 2 + rank) * BM + 4 * lane;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    ar[i] = (uint32_t)(row0 + i < p.m ? row0 + i : 0) * (uint32_t)kb_total + pc.kb0;
                br = (uint32_t)(col0 < p.n ? col0 >> 7 : 0) * (uint32_t)kb_total + pc.kb0;
                left = pc.kb1 - pc.kb0;
                return true;
            };
            bool more = next_piece();
            float qa[PF][4], qb[PF];
            uint32_t n_loaded = 0;
            auto load = [&](int d) {
                if (!more) return;
#pragma unroll
                for (int i = 0; i < 4; ++i) qa[d][i] = ld_global_f32(p.a_scale + ar[i]++);
                qb[d] = ld_global_f32(p.b_scale + br++);
                ++n_loaded;
                if (--left == 0) more = next_piece();
            };
#pragma unroll
            for (int d = 0; d < PF; ++d) load(d);
            bool ok = true;
            for (uint32_t q = 0; ok && q < n_loaded;) {
#pragma unroll
                for (int d = 0; d < PF; ++d) {
                    if (q >= n_loaded) break;
                    // The epilogue has read the slot for K block q - NB (an order that the hand-back of the accumulator
                    // does not give: it goes by a relaxed arrive and a commit, which order no shared-memory read).  It
                    // had then seen that block's arrivals on tmem_full, so this one counts for block q.
                    const uint32_t buf = half * NB + q % NB;
                    if (q >= NB) {
                        ok = __all_sync(0xffffffffu, mbar_wait(scale_empty_bar(buf), (q / NB - 1) & 1, p.status,
                                                               kErrSchedWait, p.launch_tag));
                        if (!ok) break;
                    }
                    const uint32_t slot = scale_base + buf * (BM * 4);
                    st_shared_v4(slot + lane * 16, __float_as_uint(qa[d][0] * qb[d]), __float_as_uint(qa[d][1] * qb[d]),
                                 __float_as_uint(qa[d][2] * qb[d]), __float_as_uint(qa[d][3] * qb[d]));
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tmem_full_bar(buf));
                    load(d);
                    ++q;
                }
            }
        }
    } else {
        // ---------------------------------------------------------- epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kRegsHi));
        const int ew = warp - NUM_NON_EPI_WARPS;
        const int quad = warp & 3;            // TMEM lane quadrant this warp may access
        const int half = ew >> 2;
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * (NB * HN);
        const uint32_t slab0 = slab_base + ew * Cfg::kChunks * Cfg::kSlabBytes;
        const uint32_t my_scale = scale_base + half * NB * (BM * 4) + (quad * 32 + lane) * 4;
        PlainWalker walk(p, unit, n_units, kb_total);
        Piece pc;
        uint32_t it = 0;
        F32x2 acc[HN / 2];
#pragma unroll
        for (int j = 0; j < HN / 2; ++j) acc[j] = 0;
        while (walk.next(pc, p, n_units, kb_total)) {
            const TileCoord t = decode_tile(SPLIT ? pc.item / p.splits : pc.item, p.tiles_m, p.tiles_n);
            const int cur_col0 = t.n_blk * Cfg::kBN + half * HN;
            const int cur_row0 = (t.m_blk * 2 + rank) * BM + quad * 32;
            bool ok = true;
#pragma unroll 1
            for (uint32_t end = it + (SPLIT ? pc.kb1 - pc.kb0 : kb_total); it != end; ++it) {
                const uint32_t buf = half * NB + it % NB;
                if (!mbar_wait(tmem_full_bar(buf), (it / NB) & 1, p.status, kErrEpilogueWait, p.launch_tag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t taddr = lane_addr + (it % NB) * HN;
                float v[2][32];
                tmem_ld32_async(taddr, v[0]);
                const float s = __uint_as_float(ld_shared_u32(my_scale + (it % NB) * (BM * 4)));
                const F32x2 s2 = pack_f32x2(s, s);
#pragma unroll
                for (int c = 0; c < HN / 32; ++c) {
                    tmem_ld_fence(v[c % 2]);
                    if (c + 1 < HN / 32) tmem_ld32_async(taddr + (c + 1) * 32, v[(c + 1) % 2]);
                    if (c + 1 == HN / 32) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive_cluster_relaxed(mapa_cluster(tmem_empty_bar(buf), 0));
                            mbar_arrive(scale_empty_bar(buf));
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        fma_f32x2(acc[c * 16 + j], v[c % 2][2 * j], v[c % 2][2 * j + 1], s2);
                }
            }
            if (!ok) break;
            const int cur_split = SPLIT ? pc.item % p.splits : 0;
            // Tile store: 32 rows x 128 bytes slabs, swizzled, handed to the TMA, which clips rows >= m and columns >= n.
            if (!SPLIT) {
                if (lane == 0) tma_store_wait_read<0>();       // (issued a tile ago)
                __syncwarp();
#pragma unroll
                for (int ch = 0; ch < Cfg::kChunks; ++ch) {
                    const uint32_t my_row = slab0 + ch * Cfg::kSlabBytes + lane * 128;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int a0 = ch * 32 + j * 4;
                        st_shared_v4(my_row + ((j ^ (lane & 7)) << 4),
                                     to_bf16x2(acc[a0 + 0]), to_bf16x2(acc[a0 + 1]),
                                     to_bf16x2(acc[a0 + 2]), to_bf16x2(acc[a0 + 3]));
                    }
                }
#pragma unroll
                for (int j = 0; j < HN / 2; ++j) acc[j] = 0;
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    for (int ch = 0; ch < Cfg::kChunks; ++ch) {
                        const int col = cur_col0 + ch * 64;
                        if (col >= p.n) break;
                        if (p.n_dest <= 1) {
                            tma_store_2d(&tma_c, slab0 + ch * Cfg::kSlabBytes, col, cur_row0);
                        } else {
                            // N-split GEMM: own copy first, then rank + 1, rank + 2, ...
                            for (int dd = 0; dd < p.n_dest; ++dd) {
                                int dst = p.dest_first + dd;
                                if (dst >= p.n_dest) dst -= p.n_dest;
                                tma_store_2d(&dests.m[dst], slab0 + ch * Cfg::kSlabBytes, p.c_col_offset + col, cur_row0);
                            }
                        }
                    }
                    tma_store_commit();
                }
            } else {
#pragma unroll
                for (int ch = 0; ch < HN / 32; ++ch) {
                    const uint32_t slab = slab0 + (ch % Cfg::kChunks) * Cfg::kSlabBytes;
                    if (lane == 0) tma_store_wait_read<Cfg::kChunks - 1>();
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int a0 = ch * 16 + j * 2;
                        st_shared_v4(slab + lane * 128 + ((j ^ (lane & 7)) << 4), (uint32_t)acc[a0],
                                     (uint32_t)(acc[a0] >> 32), (uint32_t)acc[a0 + 1], (uint32_t)(acc[a0 + 1] >> 32));
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (cur_col0 + ch * 32 < p.n) tma_store_3d(&tma_p, slab, cur_col0 + ch * 32, cur_row0, cur_split);
                        tma_store_commit();
                    }
                }
#pragma unroll
                for (int j = 0; j < HN / 2; ++j) acc[j] = 0;
            }
        }
        // Before exit the warp's slabs must have been read by its last stores; with several destinations the barrier
        // that follows the GEMM is taken after the data has landed.
        if (lane == 0) {
            if (p.n_dest > 1) tma_store_wait_all<0>();
            else tma_store_wait_read<0>();
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();      // the peer no longer touches this CTA's barriers, shared memory or TMEM
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_2cta(tmem_base, 512);
    }
}

// One pass of 256 x 256 tiles is what the planner chooses.  The other three are there for a caller that asks for them (K
// slices by a plan entry or argument, 256 x 128 tiles by RF_FP8_GEMM_BN): no shape was found where they are the fastest.
// us in a graph of launches, the plan / 256 x 256 in 2, 3, 4 slices: 1024 x 1536 x 7168 17.6 / 26.0, 21.7, 29.9; 1024 x 512 x
// 7168 10.1 / 21.9, 17.5, 16.3; 2048 x 2048 x 4096 20.0 / 33.9, 37.6, 44.6.  256 x 128: 1024 x 7168 x 256 7.7 (the plan 7.8),
// 6144 x 4096 x 512 21.9 (22.2), 1024 x 1536 x 7168 21.6 (17.6), 6144 x 4608 x 7168 221 (200).
using Pair256 = PairCfg<128>;     // 256 x 256 tiles
using Pair128 = PairCfg<64>;      // 256 x 128 tiles

template <class Cfg, bool SPLIT>
cudaError_t launch_split(const CUtensorMap& tma_a, const CUtensorMap& tma_b, const CUtensorMap& tma_c,
                       const CUtensorMap& tma_p, const GemmDestMaps& dests, const GemmParams& p, int num_sms,
                       bool overlap, cudaStream_t stream) {
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kernel = fp8_gemm_pair_kernel<Cfg, SPLIT>;
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    const int total = p.tiles_m * p.tiles_n * p.splits;
    const int pairs = total < num_sms / 2 ? total : num_sms / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs, 1, 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, tma_a, tma_b, tma_c, tma_p, dests, p);
}

template <class Cfg>
cudaError_t launch_cfg(const CUtensorMap& tma_a, const CUtensorMap& tma_b, const CUtensorMap& tma_c,
                       const CUtensorMap& tma_p, const GemmDestMaps& dests, const GemmParams& p, int num_sms,
                       bool overlap, cudaStream_t stream) {
    return p.splits > 1 ? launch_split<Cfg, true>(tma_a, tma_b, tma_c, tma_p, dests, p, num_sms, overlap, stream)
                        : launch_split<Cfg, false>(tma_a, tma_b, tma_c, tma_p, dests, p, num_sms, overlap, stream);
}

template <class Cfg>
cudaError_t prepare_cfg() {
    cudaError_t e = cudaFuncSetAttribute(fp8_gemm_pair_kernel<Cfg, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(fp8_gemm_pair_kernel<Cfg, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                Cfg::kSmemBytes);
}

}  // namespace

cudaError_t fp8_gemm_pair_launch(const CUtensorMap& tma_a, const CUtensorMap& tma_b, const CUtensorMap& tma_c,
                                 const CUtensorMap& tma_p, const GemmDestMaps& dests, const GemmParams& p, int block_n,
                                 int num_sms, bool overlap, cudaStream_t stream) {
    return block_n == 512 ? launch_cfg<Pair256>(tma_a, tma_b, tma_c, tma_p, dests, p, num_sms, overlap, stream)
                          : launch_cfg<Pair128>(tma_a, tma_b, tma_c, tma_p, dests, p, num_sms, overlap, stream);
}

cudaError_t fp8_gemm_pair_prepare() {
    const cudaError_t e = prepare_cfg<Pair256>();
    return e != cudaSuccess ? e : prepare_cfg<Pair128>();
}

}  // namespace rf
