// FP8 (e4m3) block-scaled GEMM for sm_100a.
//
//   C[m,n] = bf16( sum_kb a_s[m,kb] * b_s[n/128,kb] * sum_{j<128} A[m,128kb+j] * B[n,128kb+j] )
//
// Replaces the reference's transpose + pipelined MFMA kernel + split-K reduce
// (src/gemm/gemm_launcher.cpp:43-101, src/gemm/gemm_kernel.cpp:334-562, :288-303).
//
// One persistent CTA per SM, warp-specialised:
//   warp 0      TMA producer: A [128 x 128 B] and B [BN x 128 B] tiles, 128-byte
//               swizzle, into a STAGES-deep shared-memory ring (mbarrier tx counts)
//   warp 1      MMA issuer: per 128-deep K block, 4 x tcgen05.mma.kind::f8f6f4
//               (K = 32 each) into one of 512/BN TMEM accumulator buffers, then a
//               tcgen05.commit that publishes the buffer
//   warps 4..   epilogue: tcgen05.ld the K block's fp32 partial sums, scale by
//               the exact fp32 product a_s*b_s and add into a register
//               accumulator (packed fma.rn.f32x2) while the next K blocks' MMAs run
//               in the other TMEM buffers; finally round to bf16 (or store fp32
//               split-K slices)
//
// The scales are arbitrary fp32 numbers, so the hardware block-scaled MMA
// (ue8m0 scales) cannot be used; promotion is one FMA per element per K block,
// exactly the ratio of the reference's `frag_r += s * frag_c`
// (src/gemm/gemm_kernel.cpp:173-207).
#include "ptx.cuh"
#include "fp8_gemm.h"
#include "fp8_tiles.cuh"

#include <atomic>
#include <cstdio>
#include <cstdlib>

namespace rf {

#ifdef RF_WAIT_STATS
// Debug build only: cycles each role spent inside its barrier waits, summed over CTAs.
__device__ unsigned long long g_wait_stats[12];
#define RF_STAT_BEGIN() const long long _t0 = clock64()
#define RF_STAT_END(acc) (acc) += clock64() - _t0
#define RF_STAT_FLUSH(idx, acc) atomicAdd(&g_wait_stats[idx], (unsigned long long)(acc))
#else
#define RF_STAT_BEGIN()
#define RF_STAT_END(acc)
#define RF_STAT_FLUSH(idx, acc)
#endif

namespace {

constexpr int BM = 128;
constexpr int BK = 128;          // one scale block, one 128-byte swizzle row of fp8
constexpr int UMMA_K = 32;       // K per tcgen05.mma for 8-bit operands
constexpr int NUM_NON_EPI_WARPS = 4;
constexpr int kMaxClusterSlices = 8;     // the portable cluster size

// MN_MAJOR: operands stored [k][m] and [k][n] (M / N contiguous), the reference's physical layout
// (src/gemm/gemm_kernel_legacy.cpp:264-268); consumed directly as MN-major UMMA operands, so the
// reference's transpose pass (src/gemm/gemm_launcher.cpp:55-56) has no counterpart here.
// SLABS: store slabs per epilogue warp.  With two, the second 64-column chunk of a tile is staged while the
// TMA is still reading the first; worth its 32 KB of shared memory (one pipeline stage fewer) only when K is
// short and the per-tile store is a large share of the tile's time.
template <int BN, int STAGES, bool MN_MAJOR = false, int SLABS = 1>
struct GemmCfg {
    static constexpr int kBN = BN;
    static constexpr int kStages = STAGES;
    static constexpr bool kMnMajor = MN_MAJOR;
    static constexpr int kEpiGroups = 2;                       // column groups, 4 warps each
    static constexpr int kColsPerThread = BN / kEpiGroups;     // 64 or 128: one scale block at most
    static constexpr int kEpiWarps = 4 * kEpiGroups;
    static constexpr int kThreads = 32 * (NUM_NON_EPI_WARPS + kEpiWarps);   // 384
    static constexpr int kABytes = BM * BK;
    static constexpr int kBBytes = BN * BK;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr bool kCommitFreesStage = BN == 128;      // who gives a stage back: the MMAs' commit, or the epilogue
    static constexpr int kTmemBufs = 512 / BN;                // accumulator buffers in flight
    static constexpr int kTmemCols = kTmemBufs * BN;          // all 512 TMEM columns
    // full / empty per stage, full / empty per accumulator buffer, the two stream-K barriers, the TMEM address slot
    // (16 bytes)
    static constexpr int kBarBytes = (2 * STAGES + 2 * kTmemBufs + 2) * 8 + 16;
    static constexpr int kSlabBytes = 32 * 128;               // one slab: 32 rows x 128 B, swizzled
    static constexpr int kSlabs = SLABS;                      // slabs per epilogue warp
    static_assert(SLABS == 1 || SLABS == 2, "one or two store slabs per warp");
    static constexpr int kSmemBytes =
        STAGES * kStageBytes + kEpiWarps * kSlabs * kSlabBytes + kBarBytes + 1024;       // + alignment slack
    // The epilogue (64 or 128 accumulators per thread plus staging) wants more than the 168 registers a
    // 384-thread CTA starts with, the producer warpgroup far fewer: registers are rebalanced after set-up
    // (128 * kRegsLo + 256 * kRegsHi <= 64512, the CTA's allocation at 168 per thread).  The splits are measured ones, each
    // a build of its own: others are slower without a spill to show for it, for reasons not traced.  256 wide, 6144 x 4608 x
    // 7168: 64 / 216 242 us, 72 / 216 247, 88 / 208 224; 56 / 224, 104 / 200 and 120 / 192 176, of which the last is the
    // fastest of the three on short calls.  128 wide, 68 x 6464 x 3456 in 2 slices: 120 / 192 9.8, no rebalancing 10.1,
    // 56 / 224 9.5.
    static constexpr bool kRebalanceRegs = true;
#if defined(RF_REGS_LO) && defined(RF_REGS_HI)
    static constexpr int kRegsLo = RF_REGS_LO, kRegsHi = RF_REGS_HI;
#else
    static constexpr int kRegsLo = BN == 128 ? 56 : 120, kRegsHi = BN == 128 ? 224 : 192;
#endif
    static_assert(128 * kRegsLo + 256 * kRegsHi <= 64512 && kRegsLo % 8 == 0 && kRegsHi % 8 == 0, "register split");
    static_assert(kColsPerThread == 64 || kColsPerThread == 128, "epilogue handles 64 or 128 columns per thread");
    static_assert(kTmemCols == 512, "TMEM columns: power of two, at most 512");
    static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
};

// OR of the words the e4m3fnuz conversion pass left: 1 = A, 2 = B holds a byte that reads differently as e4m3fn.
// (Called by whole warps.)
__device__ __forceinline__ uint32_t fnuz_special(const uint32_t* words) {
    const int lane = threadIdx.x & 31;
    uint32_t v = 0;
#pragma unroll
    for (int i = 0; i < kFnuzWords / 128; ++i) {
        const uint4 q = ld_global_cg_v4(words + 4 * (32 * i + lane));
        v |= q.x | q.y | q.z | q.w;
    }
    return __reduce_or_sync(0xffffffffu, v);
}

// First K-block unit of CTA j's share of the stream-K region (`total` units over `n_units` CTAs).
__host__ __device__ __forceinline__ int sk_share_begin(long long total, int j, int n_units) {
    return (int)(total * j / n_units);
}

// Contributors of the tile whose first unit is `base` and whose owner is CTA `unit`: the CTAs j < unit whose
// share overlaps [base, owner's first unit).  sk_first_contributor gives the lowest candidate; candidates with an
// empty share or one that ends at or below `base` contribute nothing.
__host__ __device__ __forceinline__ int sk_first_contributor(long long total, int unit, int n_units, int base) {
    int j = unit - 1;
    while (j > 0 && sk_share_begin(total, j, n_units) > base) --j;
    return j < 0 ? 0 : j;
}
__host__ __device__ __forceinline__ bool sk_contributes(long long total, int j, int n_units, int base) {
    const int hi = sk_share_begin(total, j + 1, n_units);
    return hi > base && hi > sk_share_begin(total, j, n_units);
}

// First tile of the stream-K region.
__host__ __device__ __forceinline__ int sk_tile0(const GemmParams& p) { return p.tiles_m * p.tiles_n - p.sk_tiles; }

// The walker of plain launches (PlainWalker) and of stream-K launches.
//
// Stream-K launches (p.sk_tiles > 0): the LAST p.sk_tiles tiles form a region whose K blocks, numbered
// tile-major, are cut into n_units equal contiguous shares, so that no SM idles in a ragged last wave.  A CTA
// takes its share from the TOP down (so a tile that continues in the next CTA's share is started first and
// the tile it finishes for the previous CTA comes last) and then its plain tiles.  A share boundary inside a
// tile makes the lower CTA a contributor (it leaves its fp32 partial sums in its scratch slot and raises its
// flag at the very beginning of its run) and the upper CTA, which holds the tile's last K block, the owner
// (it adds the slots of the contributors, all of LOWER block index and long finished with them, and stores
// the tile).  Waiting only ever goes to lower block indices, which are scheduled no later than the waiter.
// (p.splits == 1, so a work item is a tile.)
template <bool STREAM_K>
struct WorkWalker : PlainWalker {
    using PlainWalker::PlainWalker;
};
template <>
struct WorkWalker<true> {
    int u_lo, u_hi;            // stream-K units of this CTA not yet done: [u_lo, u_hi), taken from the top
    int w;                     // next plain tile
    __host__ __device__ __forceinline__ WorkWalker(const GemmParams& p, int unit, int n_units, int kb_total) {
        const long long total = (long long)p.sk_tiles * kb_total;
        u_lo = sk_share_begin(total, unit, n_units);
        u_hi = sk_share_begin(total, unit + 1, n_units);
        w = unit;
    }
    __host__ __device__ __forceinline__ bool next(Piece& pc, const GemmParams& p, int n_units, int kb_total) {
        if (u_hi > u_lo) {
            const int t = (u_hi - 1) / kb_total;
            const int base = t * kb_total;
            const int lo = u_lo > base ? u_lo : base;
            pc.item = sk_tile0(p) + t;
            pc.kb0 = lo - base;
            pc.kb1 = u_hi - base;
            u_hi = lo;
            return true;
        }
        if (w < sk_tile0(p)) {
            pc.item = w;
            pc.kb0 = 0;
            pc.kb1 = kb_total;
            w += n_units;
            return true;
        }
        return false;
    }
};

// STREAM_K: the instantiation that stream-K launches (p.sk_tiles > 0) run; plain launches run the other one, which
// contains none of the stream-K code.
// CLUSTER_K: split-K with the K slices of a tile in one cluster, every CTA with one slice.  The slices meet in shared
// memory: each CTA leaves its fp32 tile in the stage ring, which its last K block has emptied, and sums its share of
// the tile's rows over the cluster in ascending slice order (the order, and so the bits, of splitk_reduce_kernel).
// That replaces the slices' round trip through memory and the second launch: 64 x 576 x 7168 in 8 slices takes 7.4 us
// (8.6 before), 1024 x 512 x 7168 in 4 10.4 (11.5).  128-wide tiles only: 256-wide ones reach 22.2 us on 1024 x 1536 x
// 7168 in 2 slices where 3 slices through memory take 18.3.
template <class Cfg, bool STREAM_K = false, bool CLUSTER_K = false>
__global__ void __launch_bounds__(Cfg::kThreads, 1)
fp8_gemm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                const __grid_constant__ CUtensorMap tma_c, const __grid_constant__ CUtensorMap tma_p,
                const __grid_constant__ GemmDestMaps dests, const GemmParams p) {
    constexpr int BN = Cfg::kBN;
    constexpr int STAGES = Cfg::kStages;
    constexpr int CPT = Cfg::kColsPerThread;
    constexpr int NBUF = Cfg::kTmemBufs;
    static_assert(!CLUSTER_K || (BN == 128 && !STREAM_K), "cluster split-K: 128 x 128 tiles");

    extern __shared__ uint8_t smem_raw[];
    // 128-byte-swizzled tiles need 1024-byte alignment.
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t slab_base = smem_base + STAGES * Cfg::kStageBytes;
    const uint32_t bar_base = slab_base + Cfg::kEpiWarps * Cfg::kSlabs * Cfg::kSlabBytes;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto tmem_full_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + b); };
    auto tmem_empty_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + NBUF + b); };
    // stream-K: "this CTA's partial sums are stored" (8 epilogue warps -> warp 3) and "the partial sums this CTA's
    // owner piece needs have arrived" (warp 3 -> epilogue warps); each is used at most once per launch
    const uint32_t sk_stored_bar = bar_base + 8u * (2 * STAGES + 2 * NBUF);
    const uint32_t sk_ready_bar = sk_stored_bar + 8u;
    const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 2 * NBUF + 2);
    uint32_t* tmem_slot_ptr =
        reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    // The next kernel in the stream may be scheduled onto SMs as this grid's CTAs leave them; it blocks in
    // its own griddep_wait() until this grid has completed.
    griddep_launch_dependents();
    const int unit = (int)blockIdx.x;          // work-loop index
    const int unit_stride = (int)gridDim.x;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tma_a);
        tma_prefetch_desc(&tma_b);
        tma_prefetch_desc(p.splits == 1 ? &tma_c : &tma_p);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        if (STREAM_K) {
            mbar_init(sk_stored_bar, Cfg::kEpiWarps);
            mbar_init(sk_ready_bar, 1);
        }
        for (int b = 0; b < NBUF; ++b) {
            mbar_init(tmem_full_bar(b), 1);
            mbar_init(tmem_empty_bar(b), Cfg::kEpiWarps);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, Cfg::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot_ptr);
    // Barriers, TMEM and descriptors are set up; everything below reads or writes global memory that the
    // previous kernel in the stream may still be producing.
    griddep_wait();

    const int kb_total = p.k / BK;

    if (warp < NUM_NON_EPI_WARPS) {
    // Register split after set-up: the 4 producer / MMA warps shrink to kRegsLo, the 8 epilogue warps grow
    // to kRegsHi.
    if (Cfg::kRebalanceRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(Cfg::kRegsLo));
    // Producer and MMA issuer each run on one lane: a step of theirs is a serial chain, and every instruction of it
    // queues behind those of the epilogue warps on the same scheduler.  (1024 x 1536 x 7168 in one pass of 128-wide tiles
    // 18.3 us as whole warps that vote and elect at every step, two of them issuing MMAs in turn; now 17.8.  1024 x 4096 x
    // 512: 6.36, now 6.09.)
    bool producer = false, loads_ok = true;      // the producer's lane; what it leaves for its end, below
    uint32_t loads = 0;
    if (warp == 0) {
        // ------------------------------------------------------ TMA producer
        uint32_t it = 0;  // running K-block counter across work items
        bool ok = true;
        long long w_empty = 0; (void)w_empty;
        // e4m3fnuz operands (reference-layout configurations only): an operand that holds +-240 or NaN bytes
        // is read from its converted copy (the conversion pass that ran before this kernel left the words)
        const CUtensorMap* map_a = &tma_a;
        const CUtensorMap* map_b = &tma_b;
        if (Cfg::kMnMajor && p.fnuz_words != nullptr) {
            const uint32_t special = fnuz_special(p.fnuz_words);
            if (special & 1u) map_a = &dests.m[0];
            if (special & 2u) map_b = &dests.m[1];
        }
        if (elect_one()) {
            WorkWalker<STREAM_K> walk(p, unit, unit_stride, kb_total);
            Piece pc;
            while (ok && walk.next(pc, p, unit_stride, kb_total)) {
                const TileCoord t = decode_tile(p.splits == 1 ? pc.item : pc.item / p.splits, p.tiles_m, p.tiles_n);
                const int a_row0 = t.m_blk * BM;
                const int b_row0 = t.n_blk * BN;
                for (int kb = pc.kb0; kb < pc.kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    { RF_STAT_BEGIN();
                    ok = mbar_wait(empty_bar(s), ph ^ 1, p.status, kErrProducerWait, p.launch_tag);
                    RF_STAT_END(w_empty); }
                    if (!ok) break;
                    mbar_expect_tx(full_bar(s), Cfg::kStageBytes);
                    const uint32_t sa = smem_base + s * Cfg::kStageBytes;
                    if (Cfg::kMnMajor) {
                        // boxes of 128 K-rows x 128 bytes of M (or N); B needs one box per 128 columns
                        tma_load_2d(sa, map_a, full_bar(s), a_row0, kb * BK);
#pragma unroll
                        for (int j = 0; j < BN / 128; ++j)
                            tma_load_2d(sa + Cfg::kABytes + j * (BK * 128), map_b, full_bar(s), b_row0 + 128 * j,
                                        kb * BK);
                    } else {
                        tma_load_2d(sa, &tma_a, full_bar(s), kb * BK, a_row0);
                        tma_load_2d(sa + Cfg::kABytes, &tma_b, full_bar(s), kb * BK, b_row0);
                    }
                }
            }
            RF_STAT_FLUSH(0, w_empty);
            producer = true;
            loads = it;
            loads_ok = ok;
        }
        __syncwarp();
    } else if (warp == 1) {
        // -------------------------------------------------------- MMA issuer
        constexpr uint32_t idesc = make_idesc(BM, BN, /*e4m3*/ 0, /*e4m3*/ 0,
                                              Cfg::kMnMajor ? 1 : 0, Cfg::kMnMajor ? 1 : 0);
        // descriptor advance per MMA (K = 32): 32 bytes inside the swizzled row for K-major operands,
        // 32 K-rows of 128 bytes for MN-major ones (address field is in 16-byte units)
        constexpr uint32_t kstep = Cfg::kMnMajor ? (UMMA_K * 128) / 16 : UMMA_K / 16;
        uint32_t it = 0;
        bool ok = true;
        long long w_tmem = 0, w_full = 0, w_issue = 0; (void)w_tmem; (void)w_full; (void)w_issue;
        if (elect_one()) {
            WorkWalker<STREAM_K> walk(p, unit, unit_stride, kb_total);
            Piece pc;
            while (ok && walk.next(pc, p, unit_stride, kb_total)) {
                for (int kb = pc.kb0; kb < pc.kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    const int buf = it % NBUF;
                    const uint32_t bph = (it / NBUF) & 1;
                    { RF_STAT_BEGIN();
                    ok = mbar_wait(tmem_empty_bar(buf), bph ^ 1, p.status, kErrMmaWaitTmem, p.launch_tag);
                    RF_STAT_END(w_tmem); }
                    if (!ok) break;
                    { RF_STAT_BEGIN();
                    ok = mbar_wait(full_bar(s), ph, p.status, kErrMmaWaitFull, p.launch_tag);
                    RF_STAT_END(w_full); }
                    if (!ok) break;
                    tc_fence_after();
                    RF_STAT_BEGIN();
                    const uint32_t sa = smem_base + s * Cfg::kStageBytes;
                    const uint64_t adesc = Cfg::kMnMajor ? smem_desc_mnmajor_sw128(sa, BK * 128, 1024)
                                                         : smem_desc_kmajor_sw128(sa);
                    const uint64_t bdesc = Cfg::kMnMajor ? smem_desc_mnmajor_sw128(sa + Cfg::kABytes, BK * 128, 1024)
                                                         : smem_desc_kmajor_sw128(sa + Cfg::kABytes);
                    const uint32_t d = tmem_base + buf * BN;
#pragma unroll
                    for (int j = 0; j < BK / UMMA_K; ++j)
                        umma_f8(d, adesc + kstep * j, bdesc + kstep * j, idesc, j > 0 ? 1u : 0u);
                    // One commit per K block publishes the accumulator buffer.  128-wide tiles free the smem stage with a
                    // second one; 256-wide ones leave that to the epilogue, which observes the first (with a second commit,
                    // and without the arrive in the epilogue's K loop, 6144 x 4608 x 7168 takes 222 us instead of 187, with no
                    // spill to show for it).
                    umma_commit(tmem_full_bar(buf));
                    if (Cfg::kCommitFreesStage) umma_commit(empty_bar(s));
                    RF_STAT_END(w_issue);
                }
            }
            RF_STAT_FLUSH(1, w_tmem); RF_STAT_FLUSH(2, w_full); RF_STAT_FLUSH(6, w_issue);
        }
        __syncwarp();
    } else if (STREAM_K && warp == 3) {
        // ------------------------------------------------- stream-K flag keeper
        // The fence that publishes this CTA's partial sums and the acquiring polls on other CTAs' flags cost
        // microseconds; this otherwise idle warp pays them, so the epilogue warps only store, load and pass two
        // shared-memory barriers.  (Memory order: epilogue stores -> mbarrier arrive [release.cta] -> this warp's
        // wait [acquire.cta] -> fence.acq_rel.gpu -> flag store; and on the other side flag load [acquire.gpu]
        // -> mbarrier arrive -> epilogue wait -> loads.  Both chains are causality-ordered.)
        const unsigned long long token = p.sk_token;
        unsigned long long* sk_flags = reinterpret_cast<unsigned long long*>(
            reinterpret_cast<char*>(p.partial) + (size_t)unit_stride * (BM * BN * sizeof(float)));
        const long long total = (long long)p.sk_tiles * kb_total;
        const int u_lo = sk_share_begin(total, unit, unit_stride);
        const int u_hi = sk_share_begin(total, unit + 1, unit_stride);
        bool ok = true;
        if (u_hi > u_lo && u_hi % kb_total != 0) {
            // the top of the share stops inside a tile: the first piece leaves partial sums
            ok = __all_sync(0xffffffffu, mbar_wait(sk_stored_bar, 0, p.status, kErrSchedWait, p.launch_tag));
            if (ok) {
                __threadfence();
                if (lane == 0) st_release_gpu_u64(sk_flags + unit, token);
            }
        }
        const int base = u_lo / kb_total * kb_total;       // first unit of the tile the share starts in
        if (ok && u_lo != base && u_hi >= base + kb_total) {
            // the bottom of the share starts inside a tile and reaches that tile's end: the last piece owns the
            // tile.  Its contributors are the CTAs below whose shares overlap the tile.
            for (int j = sk_first_contributor(total, unit, unit_stride, base); j < unit && ok; ++j) {
                if (!sk_contributes(total, j, unit_stride, base)) continue;
                ok = __all_sync(0xffffffffu, flag_wait_u64(sk_flags + j, token, p.status, kErrSchedWait, p.launch_tag));
                // consumed: cleared for the next launch that uses this scratch (a replayed graph carries the
                // same number every time)
                if (ok && lane == 0) sk_flags[j] = 0ull;
            }
            if (ok && lane == 0) mbar_arrive(sk_ready_bar);
        }
    }
    if (CLUSTER_K) cluster_sync_all();     // pairs with the epilogue warps' one in front of the sums
    // (behind the cluster's barrier, which the sums wait for: in front of it 64 x 576 x 7168 in 8 slices takes 7.59 us, here
    // 7.29.  In 256-wide tiles, whose stages the epilogue frees, it only makes sure that every copy has landed: 1024 x 4096 x
    // 512 6.40 us, without it 6.36.)
    if (producer) finish_producer(loads_ok, loads, STAGES, empty_bar(0), p.status, kErrProducerWait, p.launch_tag);
    __syncwarp();
    } else {
        // ---------------------------------------------------------- epilogue
        if (Cfg::kRebalanceRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(Cfg::kRegsHi));
        const int ew = warp - NUM_NON_EPI_WARPS;
        const int quad = warp & 3;            // TMEM lane quadrant this warp may access
        const int grp = ew >> 2;              // column group
        const int row_in_tile = quad * 32 + lane;
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
        uint32_t it = 0;
        uint32_t n_stores = 0;        // tile-store chunks issued by this warp so far
        bool ok = true;
        long long w_acc = 0, w_total = 0, w_rel = 0; (void)w_acc; (void)w_total; (void)w_rel;
        long long w_skw = 0, w_skf = 0, w_skr = 0; (void)w_skw; (void)w_skf; (void)w_skr;
#ifdef RF_WAIT_STATS
        const long long t_begin = clock64();
#endif
        // K-major scale tables have unit stride along K (a compile-time fact the address arithmetic of the
        // prefetch queue depends on); only the reference's [k/128][m] tables stride by m
        const int as_ks = Cfg::kMnMajor ? (int)p.as_k_stride : 1;
        const int bs_ks = Cfg::kMnMajor ? (int)p.bs_k_stride : 1;
        // out_scale (reference-layout configurations only): 1 for e4m3fn bytes.  e4m3fnuz bytes read as
        // e4m3fn are twice their value, so each operand that is consumed unconverted contributes 1/2; an
        // operand read from its converted copy (true values) contributes 1.  A power of two commutes
        // exactly with every rounding of the fp32 accumulation.
        float out_scale = 1.0f;
        if (Cfg::kMnMajor && p.fnuz_words != nullptr) {
            const uint32_t special = fnuz_special(p.fnuz_words);
            out_scale = ((special & 1u) ? 1.0f : 0.5f) * ((special & 2u) ? 1.0f : 0.5f);
        }
        // Scale loads run PF K blocks ahead of their use so their latency (L2 or HBM) never sits on the
        // per-K-block critical path.  (Requesting a tile's first scales before the previous tile is stored was
        // measured: no gain on long K, 8 % slower on K <= 512.)
        constexpr int PF = 4;
        float qa[PF], qb[PF];
        int kb0 = 0, kb1 = 0;
        const float* as_row = p.a_scale;
        const float* bs_row = p.b_scale;
        auto begin_piece = [&](const Piece& pc) {
            const TileCoord t = decode_tile(p.splits == 1 ? pc.item : pc.item / p.splits, p.tiles_m, p.tiles_n);
            kb0 = pc.kb0;
            kb1 = pc.kb1;
            const int row = t.m_blk * BM + row_in_tile;
            const int col0 = t.n_blk * BN + grp * CPT;
            as_row = p.a_scale + (long long)(row < p.m ? row : 0) * p.as_row_stride;
            bs_row = p.b_scale + (long long)(col0 < p.n ? (col0 >> 7) : 0) * p.bs_row_stride;
#pragma unroll
            for (int d = 0; d < PF; ++d) {
                const int kk = min(kb0 + d, kb1 - 1);
                qa[d] = ld_global_f32(as_row + kk * as_ks);
                qb[d] = ld_global_f32(bs_row + kk * bs_ks);
            }
        };
        // The next piece is drawn (tile decoded, scale pointers set, first scales requested) in the middle of the
        // current tile's store, between its first and second chunk, where the warp would otherwise wait for the
        // TMA to have read the slab it is about to rewrite (about 240 cycles per chunk, measured).
        WorkWalker<STREAM_K> walk(p, unit, unit_stride, kb_total);
        Piece pc;
        bool have = walk.next(pc, p, unit_stride, kb_total);
        if (have) begin_piece(pc);
        auto advance = [&] {
            have = walk.next(pc, p, unit_stride, kb_total);
            if (have) begin_piece(pc);
        };
        float2 acc[CPT / 2];
        bool zeroed = false;      // the tile store of the previous tile left every accumulator cleared
        while (ok && have) {
            const int cur_item = pc.item;     // `pc` moves on to the next piece during the store
            bool fresh = true;        // the accumulators still have to be cleared
            if (STREAM_K && kb0 > 0 && kb1 == kb_total) {
                // Stream-K owner piece (the tile's last K blocks; always this CTA's last piece of the region):
                // the accumulators start from the partial sums that lower CTAs left in their scratch slots at
                // the very beginning of their runs, added in ascending K order (a fixed order for a given grid,
                // so results do not depend on timing).  The loads are in flight while the pipeline fills.
                { RF_STAT_BEGIN();
                ok = __all_sync(0xffffffffu, mbar_wait(sk_ready_bar, 0, p.status, kErrSchedWait, p.launch_tag));
                RF_STAT_END(w_skf); }
                if (!ok) break;
                RF_STAT_BEGIN();
                const long long total = (long long)p.sk_tiles * kb_total;
                const int base = (pc.item - sk_tile0(p)) * kb_total;      // the tile's first unit
                for (int j = sk_first_contributor(total, unit, unit_stride, base); j < unit; ++j) {
                    if (!sk_contributes(total, j, unit_stride, base)) continue;
                    const float4* src = reinterpret_cast<const float4*>(p.partial) + (size_t)j * (BM * BN / 4) +
                                        ((int)threadIdx.x - 32 * NUM_NON_EPI_WARPS);
                    if (fresh) {
#pragma unroll
                        for (int q = 0; q < CPT / 4; ++q) {
                            const float4 t4 = ld_global_cg_v4_f32(src + q * (32 * Cfg::kEpiWarps));
                            acc[2 * q] = make_float2(t4.x, t4.y);
                            acc[2 * q + 1] = make_float2(t4.z, t4.w);
                        }
                        fresh = false;
                    } else {
#pragma unroll
                        for (int q0 = 0; q0 < CPT / 4; q0 += 8) {
                            float4 t4[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) t4[i] = ld_global_cg_v4_f32(src + (q0 + i) * (32 * Cfg::kEpiWarps));
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                acc[2 * (q0 + i)].x += t4[i].x;
                                acc[2 * (q0 + i)].y += t4[i].y;
                                acc[2 * (q0 + i) + 1].x += t4[i].z;
                                acc[2 * (q0 + i) + 1].y += t4[i].w;
                            }
                        }
                    }
                }
                RF_STAT_END(w_skr);
            }
            if (fresh && !zeroed) {
#pragma unroll
                for (int j = 0; j < CPT / 2; ++j) acc[j] = make_float2(0.f, 0.f);
            }
            zeroed = false;
#pragma unroll 4
            for (int kb = kb0; kb < kb1; ++kb, ++it) {
                const float s = Cfg::kMnMajor ? qa[0] * qb[0] * out_scale : qa[0] * qb[0];
#pragma unroll
                for (int d = 0; d + 1 < PF; ++d) { qa[d] = qa[d + 1]; qb[d] = qb[d + 1]; }
                {
                    const int kk = min(kb + PF, kb1 - 1);
                    qa[PF - 1] = ld_global_f32(as_row + kk * as_ks);
                    qb[PF - 1] = ld_global_f32(bs_row + kk * bs_ks);
                }
                const float2 s2 = make_float2(s, s);
                const int buf = it % NBUF;
                const uint32_t bph = (it / NBUF) & 1;
                { RF_STAT_BEGIN();
                if (!mbar_wait(tmem_full_bar(buf), bph, p.status, kErrEpilogueWait, p.launch_tag)) { ok = false; break; }
                RF_STAT_END(w_acc); }
                tc_fence_after();
                // The MMAs that wrote this buffer have finished reading their smem stage.
                if (!Cfg::kCommitFreesStage && ew == 0 && lane == 0) mbar_arrive(empty_bar(it % STAGES));
                const uint32_t taddr = lane_addr + buf * BN + grp * CPT;
                constexpr int NCH = CPT / 32;
                auto release_buffer = [&] {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tmem_empty_bar(buf));
                };
                RF_STAT_BEGIN();
                // Staging registers: two 32-column buffers (the load of chunk c+1 overlaps the FMAs of
                // chunk c) when a thread owns 64 columns; one buffer when it owns 128, because 128
                // accumulators leave no room for a second one (the other epilogue warp on the same
                // scheduler covers the load latency instead).
                constexpr int NV = CPT > 64 ? 1 : 2;
                float v[NV][32];
                tmem_ld32_async(taddr, v[0]);
#pragma unroll
                for (int c = 0; c < NCH; ++c) {
                    tmem_ld_fence(v[c % NV]);   // waits for every load issued so far
                    if (NV == 2 && c + 1 < NCH) tmem_ld32_async(taddr + (c + 1) * 32, v[(c + 1) % NV]);
#ifndef RF_LATE_RELEASE
                    if (c + 1 == NCH) { release_buffer(); RF_STAT_END(w_rel); }
#endif
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        acc[c * 16 + j] =
                            __ffma2_rn(make_float2(v[c % NV][2 * j], v[c % NV][2 * j + 1]), s2, acc[c * 16 + j]);
                    if (NV == 1 && c + 1 < NCH) tmem_ld32_async(taddr + (c + 1) * 32, v[0]);
                }
#ifdef RF_LATE_RELEASE
                release_buffer(); RF_STAT_END(w_rel);
#endif
            }
            if (!ok) break;
            if (STREAM_K && kb1 < kb_total) {
                // Stream-K contributor piece (always this CTA's first piece): the 128 x BN fp32 partial sums go to
                // this CTA's scratch slot, laid out [float4 number][epilogue thread] so that writer and reader,
                // which map threads to elements alike, move whole 512-byte lines.  Warp 3 publishes them.
                RF_STAT_BEGIN();
                float4* dst = reinterpret_cast<float4*>(p.partial) + (size_t)unit * (BM * BN / 4) +
                              ((int)threadIdx.x - 32 * NUM_NON_EPI_WARPS);
#pragma unroll
                for (int q = 0; q < CPT / 4; ++q)
                    __stcg(dst + q * (32 * Cfg::kEpiWarps),
                           make_float4(acc[2 * q].x, acc[2 * q].y, acc[2 * q + 1].x, acc[2 * q + 1].y));
                __syncwarp();
                if (lane == 0) mbar_arrive(sk_stored_bar);
                RF_STAT_END(w_skw);
                advance();
                continue;
            }
            if (CLUSTER_K) {
                // the CTA's only piece: [row][16-byte chunk ^ row % 8] of fp32, read by the whole cluster below
                const uint32_t row_base = smem_base + row_in_tile * (BN * 4) + grp * (CPT * 4);
#pragma unroll
                for (int q = 0; q < CPT / 4; ++q)
                    st_shared_v4(row_base + ((q ^ (row_in_tile & 7)) << 4),
                                 __float_as_uint(acc[2 * q].x), __float_as_uint(acc[2 * q].y),
                                 __float_as_uint(acc[2 * q + 1].x), __float_as_uint(acc[2 * q + 1].y));
                advance();
                continue;
            }
            // Tile store: each warp stages its 32 rows x 128 bytes in its own swizzled shared-memory slab, so
            // that global memory is written in whole 128-byte row segments.
            {
                constexpr int SL = Cfg::kSlabs;
                const TileCoord t = decode_tile(p.splits == 1 ? cur_item : cur_item / p.splits, p.tiles_m, p.tiles_n);
                const int col0 = t.n_blk * BN + grp * CPT;
                const uint32_t slab0 = slab_base + ew * SL * Cfg::kSlabBytes;
                // (128-wide tiles hold 64 accumulators per thread and store one chunk, or two short fp32 ones:
                // measured, drawing the next piece in between makes them slower, so they draw it afterwards)
                constexpr bool kAdvanceMidStore = CPT == 128;
                constexpr bool kClearInStore = CPT == 128 && SL == 1;
                bool advanced = false;
                const int slab_row0 = t.m_blk * BM + quad * 32;
                // One lane hands the slab to the TMA, which clips rows >= m / columns >= n.  Consecutive stores of
                // this warp alternate over its kSlabs slabs (n_stores counts them across tiles, so skipped chunks
                // of a ragged tile cannot break the alternation); before a slab is rewritten, the store that last
                // read it (kSlabs commit groups ago) must have finished reading.  (Reading the slab back and
                // writing C with ordinary vector stores was measured: 20 % slower on the short-K shapes.)
                if (p.splits == 1) {
#pragma unroll
                    for (int ch = 0; ch < CPT / 64; ++ch) {
                        if (col0 + ch * 64 >= p.n) break;
                        const uint32_t slab = slab0 + (n_stores % SL) * Cfg::kSlabBytes;
                        ++n_stores;
                        const uint32_t my_row = slab + lane * 128;
                        if (lane == 0) tma_store_wait_read<SL - 1>();
                        __syncwarp();
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int a0 = ch * 32 + j * 4;
                            st_shared_v4(my_row + ((j ^ (lane & 7)) << 4),
                                         pack_bf16x2(acc[a0 + 0].x, acc[a0 + 0].y), pack_bf16x2(acc[a0 + 1].x, acc[a0 + 1].y),
                                         pack_bf16x2(acc[a0 + 2].x, acc[a0 + 2].y), pack_bf16x2(acc[a0 + 3].x, acc[a0 + 3].y));
                        }
                        // These accumulators are done with: cleared for the next tile here, in the shadow of the
                        // shared-memory stores the fence below waits for.  (Measured: 2 % on the K ~ 2048 shapes
                        // with the four-stage configuration; the two-slab short-K configuration gets 7-10 %
                        // slower with it and keeps clearing at the top of the tile.)
                        if (kClearInStore) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) acc[ch * 32 + j] = make_float2(0.f, 0.f);
                            zeroed = ch + 1 == CPT / 64;      // (every chunk of the thread's columns was stored)
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            if (p.n_dest <= 1) {
                                tma_store_2d(&tma_c, slab, col0 + ch * 64, slab_row0);
                            } else {
                                // N-split GEMM: the slab goes to every GPU's C (own memory and peers over
                                // NVLink), which is the all-gather of C done by the epilogue itself
                                // (own copy first, then rank+1, rank+2, ...: at any moment the ranks store
                                // into different GPUs)
                                for (int dd = 0; dd < p.n_dest; ++dd) {
                                    int dst = p.dest_first + dd;
                                    if (dst >= p.n_dest) dst -= p.n_dest;
                                    tma_store_2d(&dests.m[dst], slab, p.c_col_offset + col0 + ch * 64, slab_row0);
                                }
                            }
                            tma_store_commit();
                        }
                        if (kAdvanceMidStore && ch == 0) {
                            advance();
                            advanced = true;
                        }
                    }
                } else {
                    const int cur_split = cur_item % p.splits;
#pragma unroll
                    for (int ch = 0; ch < CPT / 32; ++ch) {
                        if (col0 + ch * 32 >= p.n) break;
                        const uint32_t slab = slab0 + (n_stores % SL) * Cfg::kSlabBytes;
                        ++n_stores;
                        const uint32_t my_row = slab + lane * 128;
                        if (lane == 0) tma_store_wait_read<SL - 1>();
                        __syncwarp();
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int a0 = ch * 16 + j * 2;
                            st_shared_v4(my_row + ((j ^ (lane & 7)) << 4), __float_as_uint(acc[a0].x),
                                         __float_as_uint(acc[a0].y), __float_as_uint(acc[a0 + 1].x),
                                         __float_as_uint(acc[a0 + 1].y));
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_3d(&tma_p, slab, col0 + ch * 32, slab_row0, cur_split);
                            tma_store_commit();
                        }
                        if (kAdvanceMidStore && ch == 0) {
                            advance();
                            advanced = true;
                        }
                    }
                }
                if (!advanced) advance();
            }
        }
        if (CLUSTER_K) {
            cluster_sync_all();        // every slice of the tile is in its CTA's shared memory
            if (ok) {
                const int n_slices = p.splits;
                const int tile = (int)blockIdx.x / n_slices, slice = (int)blockIdx.x - tile * n_slices;
                const TileCoord t = decode_tile(tile, p.tiles_m, p.tiles_n);
                const int row_end = min(BM * (slice + 1) / n_slices, p.m - t.m_blk * BM);
                // a warp sums one row at a time, 4 columns per lane
                for (int r = BM * slice / n_slices + ew; r < row_end; r += Cfg::kEpiWarps) {
                    const uint32_t src = smem_base + r * (BN * 4) + ((lane ^ (r & 7)) << 4);
                    float4 part[kMaxClusterSlices];
#pragma unroll
                    for (int i = 0; i < kMaxClusterSlices; ++i)
                        if (i < n_slices) part[i] = ld_cluster_f4(mapa_cluster(src, i));
                    float4 sum = part[0];
#pragma unroll
                    for (int i = 1; i < kMaxClusterSlices; ++i)
                        if (i < n_slices) {
                            sum.x += part[i].x; sum.y += part[i].y; sum.z += part[i].z; sum.w += part[i].w;
                        }
                    const int col = t.n_blk * BN + 4 * lane;
                    if (col < p.n)
                        *reinterpret_cast<uint2*>(p.c + (size_t)(t.m_blk * BM + r) * p.n + col) =
                            make_uint2(pack_bf16x2(sum.x, sum.y), pack_bf16x2(sum.z, sum.w));
                }
            }
        }
        // Before exit the warp's slab must have been read by its last store.  Waiting for the writes themselves
        // is left to grid completion (stream order, or the next kernel's griddepcontrol.wait), except when the
        // stores go to other GPUs: the barrier that follows an N-split GEMM is taken after the data has landed.
        if (lane == 0) {
            if (p.n_dest > 1) tma_store_wait_all<0>();
            else tma_store_wait_read<0>();
        }
#ifdef RF_WAIT_STATS
        if (warp == NUM_NON_EPI_WARPS && lane == 0) {
            RF_STAT_FLUSH(3, w_acc);
            RF_STAT_FLUSH(4, clock64() - t_begin);
            RF_STAT_FLUSH(5, w_rel);
            RF_STAT_FLUSH(7, w_skw);
            RF_STAT_FLUSH(8, w_skf);
            RF_STAT_FLUSH(9, w_skr);
        }
#endif
    }

    // ------------------------------------------------------------- tear-down
    tc_fence_before();
    __syncthreads();
    if (CLUSTER_K) cluster_sync_all();     // no other CTA touches this CTA's barriers, smem or TMEM any more
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

// C = bf16( sum_s partial[s] )  -  split-K fix-up (reference: reduce_kernel,
// src/gemm/gemm_kernel.cpp:288-303).  One float4 per thread per slice.
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* partial, __nv_bfloat16* c, size_t mn, int splits) {
    griddep_launch_dependents();
    griddep_wait();     // the slices come from the GEMM launched just before
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= mn) return;
    float4 acc = *reinterpret_cast<const float4*>(partial + i);
    for (int s = 1; s < splits; ++s) {
        const float4 v = *reinterpret_cast<const float4*>(partial + (size_t)s * mn + i);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    uint2 q;
    q.x = pack_bf16x2(acc.x, acc.y);
    q.y = pack_bf16x2(acc.z, acc.w);
    *reinterpret_cast<uint2*>(c + i) = q;
}

// e4m3fnuz -> e4m3fn at equal value, one pass over both operands.
//
// The GEMM reads e4m3fnuz bytes as e4m3fn (twice the value, exactly, folded into the scale product) - except
// that 0x7F / 0xFF (+-240, the largest fnuz magnitudes, present in every block of amax-scaled data) read as
// NaN and 0x80 (the fnuz NaN) reads as -0.  This pass writes, for the whole operand, the e4m3fn byte of the
// SAME value: byte - 8 for exponent fields >= 2; the 15 magnitudes below 2^-6 fall between e4m3fn's
// subnormals and are rounded to nearest-even on that grid (absolute error <= 2^-10); 0x80 becomes the e4m3fn
// NaN.  Every block leaves a word that says in whose share it met one of the three special bytes (1: A, 2: B); the GEMM
// launched next on the stream ORs the words (fnuz_special) and reads a flagged operand from its converted copy, an
// unflagged one, exact, from the original bytes.  (A word per block needs no clearing pass and keeps nothing from one
// call for the next.)  Four bytes are converted at once in ordinary integer arithmetic; bound by the copy through L2.
// 2 + 14 MB ahead of 1024 x 7168 x 2048: the whole call takes 32.0 us (37.0 with a clearing and a table-lookup pass per
// operand).
constexpr int kFnuzThreads = 256;

__device__ __forceinline__ uint32_t fnuz_to_fn_x4(uint32_t w, uint32_t& special) {
    const uint32_t x = w & 0x7F7F7F7Fu;                               // magnitudes
    const uint32_t big = (x + 0x70707070u) & 0x80808080u;             // bit 7 where the magnitude is >= 16
    const uint32_t big_mask = (big >> 7) * 0xFFu;
    const uint32_t t = x & ~big_mask;                                 // the others: x * 2^-10 on the 2^-9 grid
    const uint32_t lo = ((t + ((t >> 1) & 0x01010101u)) >> 1) & 0x0F0F0F0Fu;
    const uint32_t o = (w & 0x80808080u) | ((x - (big >> 4)) & big_mask) | lo;
    const uint32_t is7f = (x + 0x01010101u) & 0x80808080u;            // bit 7 where the magnitude is 0x7F
    const uint32_t zero = ~((x + 0x7F7F7F7Fu) | 0x7F7F7F7Fu);         // bit 7 where the magnitude is 0
    const uint32_t is80 = zero & w & 0x80808080u;
    special |= is7f | is80;
    return o ^ ((is80 >> 7) * 0xFFu);                                 // 0x80 -> 0x7F
}

__global__ void __launch_bounds__(kFnuzThreads)
fnuz_convert_kernel(const uint4* a, uint4* __restrict__ a_dst, size_t a_vec, const uint4* b, uint4* __restrict__ b_dst,
                    size_t b_vec, uint32_t* __restrict__ words, int* __restrict__ status) {
    griddep_launch_dependents();
    griddep_wait();       // the GEMM before this call may still be reading the copies and the words
    constexpr int U = 4;  // loads in flight per thread
    const size_t total = a_vec + b_vec, step = (size_t)gridDim.x * kFnuzThreads;
    uint32_t special_a = 0, special_b = 0;
    for (size_t i0 = (size_t)blockIdx.x * kFnuzThreads + threadIdx.x; i0 < total; i0 += U * step) {
        uint4 q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t i = i0 + u * step;
            if (i < total) q[u] = i < a_vec ? a[i] : b[i - a_vec];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t i = i0 + u * step;
            if (i >= total) break;
            uint32_t special = 0;
            const uint4 o = make_uint4(fnuz_to_fn_x4(q[u].x, special), fnuz_to_fn_x4(q[u].y, special),
                                       fnuz_to_fn_x4(q[u].z, special), fnuz_to_fn_x4(q[u].w, special));
            if (i < a_vec) {
                a_dst[i] = o;
                special_a |= special;
            } else {
                b_dst[i - a_vec] = o;
                special_b |= special;
            }
        }
    }
    const uint32_t any_a = __syncthreads_or(special_a != 0), any_b = __syncthreads_or(special_b != 0);
    if (threadIdx.x == 0) {
        words[blockIdx.x] = (any_a ? 1u : 0u) | (any_b ? 2u : 0u);
        if (any_a || any_b) atomicOr(status + kStatusDiagWord, (int)kDiagFnuzByte);
    }
}

using Cfg128 = GemmCfg<128, 6>;
using Cfg256 = GemmCfg<256, 4>;
using Cfg256ShortK = GemmCfg<256, 3, false, 2>;     // K <= 512: tiles of at most four K blocks
using Cfg128Mn = GemmCfg<128, 6, true>;
using Cfg256Mn = GemmCfg<256, 4, true>;

// Programmatic dependent launch between consecutive GEMM-path kernels of a stream (the launch latency and
// the barrier / TMEM set-up of kernel i+1 overlap the tail of kernel i).  RF_FP8_GEMM_PDL=0 switches it off.
bool overlap_launches() {
    static const bool on = [] {
        const char* e = getenv("RF_FP8_GEMM_PDL");
        return !(e && e[0] == '0');
    }();
    return on;
}

// Tiles of at most four K blocks spend a large share of their time in the tile store: they get the
// two-slab configuration (RF_FP8_GEMM_SHORTK=0 keeps the ordinary one).
bool short_k_config(const GemmParams& p) {
    static const bool on = [] {
        const char* e = getenv("RF_FP8_GEMM_SHORTK");
        return !(e && e[0] == '0');
    }();
    return on && p.splits == 1 && p.k <= 4 * BK;
}

// Clusters of p.splits CTAs that fit the current device together (0 = none, or the query failed).
template <class Cfg>
int resident_clusters(int slices) {
    static std::atomic<int> known[64][kMaxClusterSlices + 1] = {};     // 0 = not asked yet, else the answer + 1
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 0;
    int v = known[dev][slices].load(std::memory_order_relaxed);
    if (v == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(slices, 1, 1);
        cfg.blockDim = dim3(Cfg::kThreads, 1, 1);
        cfg.dynamicSmemBytes = Cfg::kSmemBytes;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = slices;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        auto kernel = fp8_gemm_kernel<Cfg, false, true>;
        int n = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        v = n + 1;
        known[dev][slices].store(v, std::memory_order_relaxed);
    }
    return v - 1;
}

// Split-K inside clusters: every tile's slices resident at once, one piece per CTA.  (More tiles than that would run
// their clusters in waves; they keep the slices in memory and the fix-up kernel.)
template <class Cfg>
bool cluster_split(const GemmParams& p) {
    static_assert(BM * Cfg::kBN * 4 <= Cfg::kStages * Cfg::kStageBytes, "the fp32 tile fits the stage ring");
    return p.splits > 1 && p.splits <= kMaxClusterSlices && p.n_dest <= 1 &&
           p.tiles_m * p.tiles_n <= resident_clusters<Cfg>(p.splits);
}

template <class Cfg>
cudaError_t launch_cluster_split(const CUtensorMap& tma_a, const CUtensorMap& tma_b, const CUtensorMap& tma_c,
                                 const CUtensorMap& tma_p, const GemmDestMaps& dests, const GemmParams& p,
                                 cudaStream_t stream) {
    // (resident_clusters has set the kernel's shared-memory limit on this device)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.tiles_m * p.tiles_n * p.splits, 1, 1);
    cfg.blockDim = dim3(Cfg::kThreads, 1, 1);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap_launches() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, fp8_gemm_kernel<Cfg, false, true>, tma_a, tma_b, tma_c, tma_p, dests, p);
}

template <class Cfg, bool STREAM_K = false>
cudaError_t launch_cfg(const CUtensorMap& tma_a, const CUtensorMap& tma_b, const CUtensorMap& tma_c,
                       const CUtensorMap& tma_p, const GemmDestMaps& dests, const GemmParams& p, int num_sms,
                       cudaStream_t stream) {
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kernel = fp8_gemm_kernel<Cfg, STREAM_K>;
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    const int total = p.tiles_m * p.tiles_n * p.splits;
    // a stream-K launch shares K blocks out over exactly num_sms CTAs, whatever the tile count
    const int grid = (total < num_sms && p.sk_tiles == 0) ? total : num_sms;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(Cfg::kThreads, 1, 1);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap_launches() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, tma_a, tma_b, tma_c, tma_p, dests, p);
}

}  // namespace

namespace {
template <bool STREAM_K>
int walk_pieces(const GemmParams& p, int unit, int n_units, int* out, int max_pieces) {
    const int kb_total = p.k / BK;
    WorkWalker<STREAM_K> walk(p, unit, n_units, kb_total);
    Piece pc;
    int n = 0;
    while (walk.next(pc, p, n_units, kb_total)) {
        if (n < max_pieces) {
            out[4 * n + 0] = pc.item / p.splits;
            out[4 * n + 1] = pc.item % p.splits;
            out[4 * n + 2] = pc.kb0;
            out[4 * n + 3] = pc.kb1;
        }
        ++n;
    }
    return n;
}
}  // namespace

int fp8_gemm_walk_pieces(const GemmParams& p, int unit, int n_units, int* out, int max_pieces) {
    return p.sk_tiles > 0 ? walk_pieces<true>(p, unit, n_units, out, max_pieces)
                          : walk_pieces<false>(p, unit, n_units, out, max_pieces);
}

#ifdef RF_WAIT_STATS
extern "C" void rf_debug_wait_stats(unsigned long long* out8, int reset) {
    cudaDeviceSynchronize();
    cudaMemcpyFromSymbol(out8, g_wait_stats, sizeof(unsigned long long) * 12);
    if (reset) {
        unsigned long long z[12] = {};
        cudaMemcpyToSymbol(g_wait_stats, z, sizeof(z));
    }
}
#endif

cudaError_t fp8_fnuz_convert_launch(const void* a, void* a_dst, size_t a_bytes, const void* b, void* b_dst,
                                    size_t b_bytes, uint32_t* words, int* status, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kFnuzWords, 1, 1);
    cfg.blockDim = dim3(kFnuzThreads, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap_launches() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, fnuz_convert_kernel, static_cast<const uint4*>(a), static_cast<uint4*>(a_dst),
                              a_bytes / 16, static_cast<const uint4*>(b), static_cast<uint4*>(b_dst), b_bytes / 16, words,
                              status);
}

namespace {
template <class Cfg, bool STREAM_K = false>
cudaError_t prepare_cfg() {
    return cudaFuncSetAttribute(fp8_gemm_kernel<Cfg, STREAM_K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                Cfg::kSmemBytes);
}
template <class Cfg>
cudaError_t prepare_cluster_split() {
    for (int s = 2; s <= kMaxClusterSlices; ++s) resident_clusters<Cfg>(s);
    return cudaGetLastError();
}
}  // namespace

cudaError_t fp8_gemm_prepare_device() {
    cudaError_t e;
    if ((e = prepare_cfg<Cfg128>()) != cudaSuccess) return e;
    if ((e = prepare_cfg<Cfg256>()) != cudaSuccess) return e;
    if ((e = prepare_cfg<Cfg128, true>()) != cudaSuccess) return e;
    if ((e = prepare_cfg<Cfg256, true>()) != cudaSuccess) return e;
    if ((e = prepare_cfg<Cfg256ShortK>()) != cudaSuccess) return e;
    if ((e = fp8_gemm_pair_prepare()) != cudaSuccess) return e;
    if ((e = prepare_cfg<Cfg128Mn>()) != cudaSuccess) return e;
    if ((e = prepare_cfg<Cfg256Mn>()) != cudaSuccess) return e;
    if ((e = prepare_cluster_split<Cfg128>()) != cudaSuccess) return e;
    if ((e = prepare_cluster_split<Cfg128Mn>()) != cudaSuccess) return e;
    // the split-K fix-up takes no attribute; querying it loads the function now, not at its first launch
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, splitk_reduce_kernel);
}

bool fp8_gemm_cluster_split(int tiles, int splits) {
    return splits > 1 && splits <= kMaxClusterSlices && tiles <= resident_clusters<Cfg128>(splits);
}

cudaError_t fp8_gemm_launch(const CUtensorMap& tma_a, const CUtensorMap& tma_b, const CUtensorMap& tma_c,
                            const CUtensorMap& tma_p, const GemmDestMaps* dests, const GemmParams& p, int block_n,
                            int num_sms, cudaStream_t stream, bool mn_major) {
    GemmDestMaps local;
    if (!dests) {
        for (int i = 0; i < 8; ++i) local.m[i] = tma_c;
        dests = &local;
    }
    // block_n: 128 / 256 = one-CTA tiles of that width; 512 / 384 = the CTA-pair configurations (256 x 256 and
    // 256 x 128 per pair)
    if (p.sk_tiles > 0) {
        // stream-K: row-major operands, one destination, the one-CTA tiles
        if (mn_major || gemm_is_pair(block_n) || p.splits != 1 || p.n_dest > 1) return cudaErrorInvalidValue;
        return block_n == 256 ? launch_cfg<Cfg256, true>(tma_a, tma_b, tma_c, tma_p, *dests, p, num_sms, stream)
                              : launch_cfg<Cfg128, true>(tma_a, tma_b, tma_c, tma_p, *dests, p, num_sms, stream);
    }
    if (block_n == 128 && p.splits > 1) {
        if (mn_major && cluster_split<Cfg128Mn>(p))
            return launch_cluster_split<Cfg128Mn>(tma_a, tma_b, tma_c, tma_p, *dests, p, stream);
        if (!mn_major && cluster_split<Cfg128>(p))
            return launch_cluster_split<Cfg128>(tma_a, tma_b, tma_c, tma_p, *dests, p, stream);
    }
    cudaError_t e = mn_major
                        ? (block_n == 256 ? launch_cfg<Cfg256Mn>(tma_a, tma_b, tma_c, tma_p, *dests, p, num_sms, stream)
                                          : launch_cfg<Cfg128Mn>(tma_a, tma_b, tma_c, tma_p, *dests, p, num_sms, stream))
                    : gemm_is_pair(block_n)
                        ? fp8_gemm_pair_launch(tma_a, tma_b, tma_c, tma_p, *dests, p, block_n, num_sms, overlap_launches(), stream)
                    : block_n == 256
                        ? (short_k_config(p) ? launch_cfg<Cfg256ShortK>(tma_a, tma_b, tma_c, tma_p, *dests, p, num_sms, stream)
                                             : launch_cfg<Cfg256>(tma_a, tma_b, tma_c, tma_p, *dests, p, num_sms, stream))
                        : launch_cfg<Cfg128>(tma_a, tma_b, tma_c, tma_p, *dests, p, num_sms, stream);
    if (e != cudaSuccess) return e;
    if (p.splits > 1) {
        const size_t mn = (size_t)p.m * p.n;
        const unsigned blocks = (unsigned)((mn / 4 + 255) / 256);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(blocks, 1, 1);
        cfg.blockDim = dim3(256, 1, 1);
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = overlap_launches() ? 1 : 0;
        e = cudaLaunchKernelEx(&cfg, splitk_reduce_kernel, (const float*)p.partial, (__nv_bfloat16*)p.c, mn,
                               (int)p.splits);
    }
    return e;
}

}  // namespace rf
