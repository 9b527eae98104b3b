// C-ABI entry points of the FP8 block-scaled GEMM (declared in include/rf_b200.h).
#include "../../include/rf_b200.h"
#include "fp8_gemm.h"
#include "host_util.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace {

constexpr int kBlockK = 128;
constexpr int kMaxSplits = 64;     // K slices per GEMM (the kernel's 32-bit K-range arithmetic relies on it)

bool shape_ok(int m, int n, int k) { return m > 0 && n > 0 && k > 0 && (n % 64) == 0 && (k % kBlockK) == 0; }

// Tuning knob for experiments: RF_FP8_GEMM_BN=128|256|384|512 forces the tile configuration (512 / 384 = CTA
// pairs with 256 x 256 / 256 x 128 tiles).
int forced_block_n() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("RF_FP8_GEMM_BN");
        v = e ? atoi(e) : 0;
        if (v != 128 && v != 256 && v != 384 && v != 512) v = 0;
    }
    return v;
}

// RF_FP8_GEMM_PAIR=0: the planner never chooses the CTA-pair configuration.
bool pair_config_enabled() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("RF_FP8_GEMM_PAIR");
        v = (e && e[0] == '0') ? 0 : 1;
    }
    return v == 1;
}

// splits: K slices (1 = none), or kStreamK: one pass whose ragged last wave is shared out by K blocks.
constexpr int kStreamK = -1;

struct GemmPlan {
    int block_n;
    int splits;
    double cost;
};

// RF_FP8_GEMM_STREAMK=1 makes every automatic plan whose tiles do not fill whole waves a stream-K plan, =0 never
// uses stream-K; unset, the tuned table and the cost model decide.
int streamk_override() {
    static int v = -2;
    if (v == -2) {
        const char* e = getenv("RF_FP8_GEMM_STREAMK");
        v = e ? (atoi(e) != 0 ? 1 : 0) : -1;
    }
    return v;
}

// Tiles of the stream-K region of this launch, 0 = the plan runs as a plain pass.
int streamk_region(int m, int n, int k, int bn, int num_sms) {
    if (rf::gemm_is_pair(bn)) return 0;
    const int tiles = ((m + 127) / 128) * ((n + bn - 1) / bn);
    const int sk = rf::gemm_streamk_tiles(tiles, num_sms);
    // shares shorter than two K blocks are all fix-up and no work
    if (sk > 0 && (long long)sk * (k / kBlockK) < 2LL * num_sms) return 0;
    return sk;
}

// Whether the planner reckons with the K slices of `tiles` 128 x 128 tiles meeting in clusters: the clusters of 2 .. 8
// CTAs that a B200 answers that it holds at once, one of 3 less (with all 45 in use 50 x 5696 x 2304 takes 9.5 us, one
// pass 7.7).  A table and not a question to the device, so that a plan is the same with and without one; whether a
// launch runs in clusters is asked of its device (fp8_gemm_cluster_split).
bool plan_in_clusters(int tiles, int splits) {
    constexpr int kClusters[9] = {0, 0, 74, 44, 33, 26, 22, 15, 15};
    return splits >= 2 && splits <= 8 && tiles <= kClusters[splits];
}

// Cost model, in units of one 128-deep K block of a 128 x 128 tile (about 0.27 us where one round of tiles fits the
// chip: 64 x 576 x 7168 takes 17.7, 12.8, 8.9, 7.4 us with 56, 28, 14, 7 K blocks per CTA): rounds of tiles over the
// SMs x (K blocks per slice + fixed per-tile cost), plus, for split-K, either the cluster's exchange or the fp32 slices
// (those of one round stay in L2) and the second launch.
struct PlanCosts {
    double wide_block;        // one K block of a 128 x 256 tile with at most one tile per SM, where latency decides
    double exchange;          // of slices that meet in a cluster
    double second_launch;     // 128-wide tiles ...
    double few_rows;          // ... of fewer rows than one 32-row store box
    double wide_launch;       // behind the longer epilogue of a 256-wide tile
    double slice_rate;        // bytes / s
    int short_blocks;         // one tile per SM with at most so many K blocks is not split through memory
};
// Row-major operands: the constants that lose least over 2009 shapes of up to 300 tiles, each timed under every plan in a
// CUDA graph, 1.2 % on the geometric mean against the fastest plan.  (With the row below it was 3.3 %: 4 x 6080 x 2176 was
// split in 3 slices, 9.7 us where one pass takes 7.6, and 50 x 4480 x 4864 in 8 wide ones, 11.7 us where 4 of 128 take
// 9.4.)  A call of two launches keeps the host busy for about 9.4 us, hence short_blocks: called in a loop, one pass
// against 3 slices through memory, 50 x 5888 x 2560 8.4 / 9.5 us, 64 x 5888 x 3072 9.3 / 9.4, 64 x 5888 x 3712 10.6 / 9.4.
constexpr PlanCosts kRowMajorCosts = {1.4, 11.0, 12.0, 21.0, 18.0, 16.0e12, 24};
// The reference's layout: kernels of its own, behind a conversion pass that keeps the GPU busy while the host launches.
// 929 shapes, 1.7 % with these, 1.9 % with the row above (2000 x 704 x 5504 in 3 wide slices 24.3 us, in one
// pass 30.6).
constexpr PlanCosts kRefLayoutCosts = {1.5, 10.0, 9.3, 9.3, 9.3, 12.0e12, 0};

GemmPlan plan_for(int m, int n, int k, int num_sms, int bn, int forced_split, const PlanCosts& c) {
    const int tr = rf::gemm_tile_rows(bn), tc = rf::gemm_tile_cols(bn);
    const int tiles = ((m + tr - 1) / tr) * ((n + tc - 1) / tc);
    const int kb = k / kBlockK;
    if (rf::gemm_is_pair(bn)) num_sms /= 2;     // work items go to CTA pairs
    // relative time of one K block of one work item: 128 x 128 and 128 x 256 from in-kernel cycle counts (~620, ~790).  The
    // pairs' factors choose the slices where RF_FP8_GEMM_BN asks for pairs; whether a call runs on pairs is decided in rounds
    // (choose_plan_inner).  Their 256 x 256 tile takes about 850 cycles, the way to the next tile included.
    const double wide = bn == 512 ? 1.5 : (bn == 256 ? 1.25 : (bn == 384 ? 0.8 : 1.0));
    const bool short_pass = kb <= c.short_blocks && ((m + 127) / 128) * ((n + 127) / 128) <= num_sms;
    GemmPlan best{bn, 1, 1e30};
    for (int s = 1; s <= 8; ++s) {
        if (forced_split > 0 && s != forced_split) continue;
        if (forced_split <= 0 && s > 1 && (kb / s < 4 || tiles >= num_sms)) break;
        if (s > kb) break;
        const int rounds = (tiles * s + num_sms - 1) / num_sms;
        const int kb_per = (kb + s - 1) / s;
        const double tile_w = bn == 256 && rounds == 1 ? c.wide_block : wide;
        double cost = (double)rounds * (kb_per * tile_w + 4.0);
        if (s > 1 && bn == 128 && plan_in_clusters(tiles, s)) {
            cost += c.exchange;
        } else if (s > 1) {
            if (short_pass && forced_split <= 0) continue;
            const double bytes = 8.0 * s * (double)m * n + 2.0 * (double)m * n;
            cost += bytes / c.slice_rate / 0.27e-6 + (bn != 128 ? c.wide_launch : m < 32 ? c.few_rows : c.second_launch);
        }
        if (cost < best.cost) best = GemmPlan{bn, s, cost};
    }
    if (best.cost > 1e29) best = GemmPlan{bn, forced_split > kb ? kb : (forced_split > 0 ? forced_split : 1), 0};
    return best;
}

GemmPlan choose_plan_inner(int m, int n, int k, int num_sms, int forced_split, const PlanCosts& c, bool pairs) {
    const int fb = forced_block_n();
    if (fb) return plan_for(m, n, k, num_sms, fb, forced_split, c);
    // a measured entry for this exact shape beats the model (the caller's explicit split still wins)
    int tbn = 0, tsplits = 0;
    if (forced_split <= 0 && rf::tuned_plan_lookup(m, n, k, &tbn, &tsplits)) return GemmPlan{tbn, tsplits, 0.0};
    GemmPlan p128 = plan_for(m, n, k, num_sms, 128, forced_split, c);
    GemmPlan p256 = plan_for(m, n, k, num_sms, 256, forced_split, c);
    // Wide tiles halve the A traffic and the MMA instruction count per FLOP; prefer them unless
    // they cost noticeably more rounds (ragged N such as 576, or too few tiles).
    GemmPlan best = p256.cost <= p128.cost * 1.02 ? p256 : p128;
    // One pass of 256-wide tiles that takes at least two rounds runs on CTA pairs, unless their 256 x 256 tiles need a round
    // more: over 72 such shapes (m 585 .. 8192, us of the pair / the 128 x 256 tile) between 2 % slower and 16 % faster, the
    // geometric mean 6 %.  In one round the pair's longer hand-offs lose (1337 x 3008 x 1920 11.9 / 11.4; geometric mean of
    // 169 shapes 20 %), and so does a round more (6232 x 2304 x 2432, 225 pair tiles on 74 pairs, 38.8 / 33.0).  Single
    // shapes of one round come out even: 1024 x 3072 x 1536, which the table has on pairs, 10.7 to 12.1 / 10.8 one after the
    // other, 10.5 / 10.6 in a graph.
    const int kb = k / kBlockK;
    const int tiles = ((m + 127) / 128) * ((n + best.block_n - 1) / best.block_n);
    const int rounds = (tiles + num_sms - 1) / num_sms;
    bool pair = false;
    if (pairs && best.block_n == 256 && best.splits == 1 && rounds > 1) {
        const int pair_tiles = ((m + 255) / 256) * ((n + 255) / 256);
        pair = (pair_tiles + num_sms / 2 - 1) / (num_sms / 2) <= rounds;
    }
    // Stream-K instead of a plain single pass, in K blocks of the chosen tile: a plain pass takes
    // rounds x (kb + per-tile cost), 5 % less on pairs, a stream-K pass the even share of all K blocks plus its fixed cost
    // (slot write, slot read, one more piece per CTA).  Behind whole waves that is about 30 K blocks of a 128 x 256 tile
    // (us, stream-K / pairs: 887 x 6272 x 6016 42.4 / 44.6, 736 x 7168 x 4352 33.2 / 33.4, 3655 x 2048 x 6144 50.8 / 46.8),
    // which pays when a long-K shape has just over a whole number of waves (160 tiles of 56 K blocks: 2 x 59 against 66.5 +
    // 30); none of the 18 benchmark shapes is such a shape.  With fewer tiles than SMs every tile has several contributors
    // and a K block takes half the time: about 50 K blocks (256 wide 90; medians of 154 shapes; 300 x 4160 x 7168 takes
    // 26.6 us, a plain pass 18.1).
    if (forced_split == 0 && best.splits == 1 && streamk_region(m, n, k, best.block_n, num_sms) > 0) {
        const double plain = (double)rounds * (kb + 3.0) * (pair ? 0.95 : 1.0);
        const double fixed = rounds > 1 ? 30.0 : (best.block_n == 256 ? 90.0 : 50.0);
        const double shared = (double)tiles * kb / num_sms + 3.0 * (tiles / num_sms + 1) + fixed;
        if (shared < plain) {
            best.splits = kStreamK;
            pair = false;
        }
    }
    if (pair) best.block_n = 512;
    return best;
}

// forced_split: > 0 = that many K slices, kStreamK = stream-K, 0 = the library's choice.
// pairs: whether the planner may choose the CTA-pair configuration (it has no stream-K pass and no column-major kernel).
GemmPlan choose_plan(int m, int n, int k, int num_sms, int forced_split, bool mn_major = false, bool pairs = true) {
    const PlanCosts& costs = mn_major ? kRefLayoutCosts : kRowMajorCosts;
    if (mn_major || forced_split == kStreamK || !pair_config_enabled()) pairs = false;
    GemmPlan plan = choose_plan_inner(m, n, k, num_sms, forced_split == kStreamK ? 1 : forced_split, costs, pairs);
    // a table entry of the pair configuration: column-major operands take the one-CTA tiles of its width
    if (mn_major && plan.block_n == 512 && !forced_block_n()) plan.block_n = 256;
    if (forced_split == kStreamK) plan.splits = kStreamK;
    if (forced_split == 0) {
        const int ov = streamk_override();
        if (ov == 1) {
            if (plan.splits != kStreamK) plan = GemmPlan{forced_block_n() ? plan.block_n : 256, kStreamK, 0.0};
        } else if (ov == 0 && plan.splits == kStreamK) {
            plan.splits = 1;
        }
    }
    // a stream-K plan that has no ragged wave to share out is a plain pass
    if (plan.splits == kStreamK && streamk_region(m, n, k, plan.block_n, num_sms) == 0) plan.splits = 1;
    return plan;
}

// `dest_c` / `n_dest` / `dest_n` / `col_offset`: when n_dest > 1 the [m, n] result is written at column
// `col_offset` of each of the n_dest row-major [m, dest_n] matrices in dest_c (N-split GEMM) and `c` is unused.
int gemm_impl(const void* a, const void* b, const float* as, const float* bs, void* c, int m, int n, int k,
              int split_k, void* workspace, size_t workspace_bytes, bool own_workspace, cudaStream_t stream,
              void* const* dest_c = nullptr, int n_dest = 1, int dest_n = 0, int col_offset = 0,
              bool mn_major = false, bool fnuz = false) {
    if (!shape_ok(m, n, k)) return RF_ERR_BAD_SHAPE;
    if (mn_major && (m % 16) != 0) return RF_ERR_BAD_SHAPE;     // [k][m] rows must be 16-byte multiples for TMA
    if (n_dest > 1) {
        if (!dest_c || n_dest > 8 || dest_n < col_offset + n || dest_n % 8 != 0 || col_offset % 64 != 0)
            return RF_ERR_BAD_SHAPE;
        for (int i = 0; i < n_dest; ++i)
            if (!dest_c[i] || ((uintptr_t)dest_c[i] & 15)) return RF_ERR_NULL_POINTER;
        c = dest_c[0];
        split_k = 1;
    }
    if (!a || !b || !as || !bs || !c) return RF_ERR_NULL_POINTER;
    if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) return RF_ERR_MISALIGNED;
    if (((uintptr_t)as | (uintptr_t)bs) & 3) return RF_ERR_MISALIGNED;
    rf::DeviceState* st = rf::device_state();
    if (!st) return RF_ERR_CUDA;

    const int kb = k / kBlockK;
    if (split_k > kb) split_k = kb;
    if (split_k > kMaxSplits) split_k = kMaxSplits;
    if (split_k < kStreamK) return RF_ERR_BAD_SHAPE;
    // (an N-split GEMM's peer stores were measured from the one-CTA tiles)
    GemmPlan plan = choose_plan(m, n, k, st->num_sms, split_k, mn_major, n_dest == 1);
    if (mn_major && rf::gemm_is_pair(plan.block_n))
        plan = plan_for(m, n, k, st->num_sms, 256, split_k > 0 ? split_k : 0, kRefLayoutCosts);
    // stream-K serves the row-major single-destination GEMM; elsewhere such a plan runs as a plain pass
    if (plan.splits == kStreamK && (mn_major || n_dest > 1 || rf::gemm_is_pair(plan.block_n))) plan.splits = 1;
    const int bn = plan.block_n;
    const int sk_tiles = plan.splits == kStreamK ? streamk_region(m, n, k, bn, st->num_sms) : 0;
    const int splits = plan.splits == kStreamK ? 1 : plan.splits;

    float* partial = nullptr;
    if (splits > 1 || sk_tiles > 0) {
        const size_t need = sk_tiles > 0 ? rf::gemm_streamk_bytes(bn, st->num_sms) : (size_t)splits * m * n * sizeof(float);
        if (own_workspace) {
            partial = static_cast<float*>(rf::device_scratch(need));
            if (!partial) return RF_ERR_CUDA;
        } else {
            if (!workspace || workspace_bytes < need) return RF_ERR_WORKSPACE;
            if ((uintptr_t)workspace & 15) return RF_ERR_MISALIGNED;
            partial = static_cast<float*>(workspace);
        }
    }

    CUtensorMap ta, tb;
    if (mn_major) {
        // a [k][m], b [k][n]: boxes of 128 K-rows x 128 bytes of M / N
        if (!rf::encode_tma_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a, (uint64_t)k, (uint64_t)m, (uint64_t)m, 128,
                               128, true) ||
            !rf::encode_tma_2d(&tb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, b, (uint64_t)k, (uint64_t)n, (uint64_t)n, 128,
                               128, true))
            return RF_ERR_CUDA;
    } else {
        if (!rf::encode_tma_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a, (uint64_t)m, (uint64_t)k, (uint64_t)k, 128,
                               128, true))
            return RF_ERR_CUDA;
        if (!rf::encode_tma_2d(&tb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, b, (uint64_t)n, (uint64_t)k, (uint64_t)k,
                               (uint32_t)rf::gemm_b_box_rows(bn), 128, true))
            return RF_ERR_CUDA;
    }

    CUtensorMap tc, tp;
    if (!rf::encode_tma_2d(&tc, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, c, (uint64_t)m, (uint64_t)n, (uint64_t)n * 2, 32,
                           64, true))
        return RF_ERR_CUDA;
    if (splits > 1) {
        if (!rf::encode_tma_3d(&tp, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, partial, (uint64_t)n, (uint64_t)m,
                               (uint64_t)splits, 32, 32, true))
            return RF_ERR_CUDA;
    } else {
        tp = tc;
    }

    rf::GemmParams p;
    p.a_scale = as;
    p.b_scale = bs;
    p.c = static_cast<__nv_bfloat16*>(c);
    p.partial = partial;
    p.status = st->status;
    p.launch_tag = rf::next_launch_tag();
    p.m = m; p.n = n; p.k = k;
    p.tiles_m = (m + rf::gemm_tile_rows(bn) - 1) / rf::gemm_tile_rows(bn);
    p.tiles_n = (n + rf::gemm_tile_cols(bn) - 1) / rf::gemm_tile_cols(bn);
    p.splits = splits;
    if (mn_major) {
        p.as_row_stride = 1; p.as_k_stride = m;
        p.bs_row_stride = 1; p.bs_k_stride = (n + 127) / 128;
    } else {
        p.as_row_stride = kb; p.as_k_stride = 1;
        p.bs_row_stride = kb; p.bs_k_stride = 1;
    }
    p.n_dest = n_dest;
    p.c_col_offset = col_offset;
    p.dest_first = (n_dest > 1 && dest_n > 0 && n > 0) ? (col_offset / n) % n_dest : 0;   // = rank for an N-split
    if (sk_tiles > 0) {
        p.sk_tiles = sk_tiles;
        p.sk_token = rf::gemm_streamk_token(rf::next_streamk_epoch());
    }
    rf::GemmDestMaps dests;
    bool use_dests = false;
    if (fnuz) {
        // e4m3fnuz operands: one pass over both writes the equal-valued e4m3fn bytes into library-owned
        // scratch and flags operands that hold +-240 or NaN bytes; the kernel reads a flagged operand from
        // its converted copy (maps in dests.m[0] / m[1]) and an unflagged one, exactly, from the caller's bytes.
        const size_t a_bytes = (size_t)m * k, b_bytes = (size_t)n * k;
        if (a_bytes % 16 != 0 || b_bytes % 16 != 0) return RF_ERR_BAD_SHAPE;
        const size_t a_pad = (a_bytes + 255) / 256 * 256, b_pad = (b_bytes + 255) / 256 * 256;
        char* conv = static_cast<char*>(
            rf::device_scratch(a_pad + b_pad + rf::kFnuzWords * sizeof(uint32_t), rf::kScratchFnuz));
        if (!conv) return RF_ERR_CUDA;
        uint32_t* words = reinterpret_cast<uint32_t*>(conv + a_pad + b_pad);
        if (rf::fp8_fnuz_convert_launch(a, conv, a_bytes, b, conv + a_pad, b_bytes, words, st->status, stream) !=
            cudaSuccess)
            return RF_ERR_CUDA;
        if (!rf::encode_tma_2d(&dests.m[0], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, conv, (uint64_t)k, (uint64_t)m,
                               (uint64_t)m, 128, 128, true) ||
            !rf::encode_tma_2d(&dests.m[1], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, conv + a_pad, (uint64_t)k, (uint64_t)n,
                               (uint64_t)n, 128, 128, true))
            return RF_ERR_CUDA;
        for (int i = 2; i < 8; ++i) dests.m[i] = dests.m[0];
        p.fnuz_words = words;
        use_dests = true;
    }
    if (n_dest > 1) {
        for (int i = 0; i < n_dest; ++i) {
            if (!rf::encode_tma_2d(&dests.m[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dest_c[i], (uint64_t)m,
                                   (uint64_t)dest_n, (uint64_t)dest_n * 2, 32, 64, true))
                return RF_ERR_CUDA;
        }
        for (int i = n_dest; i < 8; ++i) dests.m[i] = dests.m[0];
        use_dests = true;
    }
    cudaError_t e = rf::fp8_gemm_launch(ta, tb, tc, tp, use_dests ? &dests : nullptr, p, bn, st->num_sms, stream,
                                        mn_major);
    if (e != cudaSuccess) {
        fprintf(stderr, "rf_b200: fp8 gemm launch failed: %s\n", cudaGetErrorString(e));
        return RF_ERR_CUDA;
    }
    return RF_OK;
}

}  // namespace

namespace rf {
void fp8_gemm_plan(int m, int n, int k, int num_sms, int split_k, int* block_n, int* splits) {
    const int kb = k / kBlockK;
    if (split_k > kb) split_k = kb;
    if (split_k > kMaxSplits) split_k = kMaxSplits;
    const GemmPlan plan = choose_plan(m, n, k, num_sms, split_k);
    *block_n = plan.block_n;
    *splits = plan.splits;
}
}  // namespace rf

extern "C" {

const char* rf_version(void) { return "rf_b200 0.1 sm_100a"; }

int rf_device_status(int* detail) {
    rf::DeviceState* st = rf::device_state();
    if (!st) return RF_ERR_CUDA;
    int v[2] = {0, 0};
    if (cudaDeviceSynchronize() != cudaSuccess) return RF_ERR_CUDA;
    if (cudaMemcpy(v, st->status, sizeof(v), cudaMemcpyDeviceToHost) != cudaSuccess) return RF_ERR_CUDA;
    // word 0: code of an expired wait (1-6); word 1: diagnostic flags (16, 32) that stopped nothing
    if (detail) *detail = v[0] != 0 ? (v[0] & 0xFF) : v[1];
    if (v[0] != 0 || v[1] != 0) {
        cudaMemset(st->status, 0, sizeof(v));
        return RF_ERR_DEVICE_TIMEOUT;
    }
    return RF_OK;
}

int rf_set_wait_limit_ns(unsigned long long limit_ns) {
    rf::DeviceState* st = rf::device_state();
    if (!st) return RF_ERR_CUDA;
    return cudaMemcpy(st->status + rf::kStatusLimitWord, &limit_ns, sizeof(limit_ns), cudaMemcpyHostToDevice) ==
                   cudaSuccess
               ? RF_OK : RF_ERR_CUDA;
}

int rf_fp8_gemm_get_plan(int m, int n, int k, int* block_n, int* split_k) {
    if (!shape_ok(m, n, k)) return RF_ERR_BAD_SHAPE;
    rf::DeviceState* st = rf::device_state();
    const GemmPlan plan = choose_plan(m, n, k, st ? st->num_sms : 148, 0);
    if (block_n) *block_n = plan.block_n;
    if (split_k) *split_k = plan.splits;
    return RF_OK;
}

int rf_fp8_gemm_choose_split(int m, int n, int k) {
    if (!shape_ok(m, n, k)) return 0;
    rf::DeviceState* st = rf::device_state();
    if (!st) return 0;
    return choose_plan(m, n, k, st->num_sms, 0).splits;
}

int rf_fp8_gemm_kernel_launches(int m, int n, int k) {
    if (!shape_ok(m, n, k)) return 0;
    rf::DeviceState* st = rf::device_state();
    if (!st) return 0;
    const GemmPlan plan = choose_plan(m, n, k, st->num_sms, 0);
    const int tiles = ((m + 127) / 128) * ((n + 127) / 128);
    const bool fix_up = plan.splits > 1 && !(plan.block_n == 128 && rf::fp8_gemm_cluster_split(tiles, plan.splits));
    return fix_up ? 2 : 1;
}

int rf_fp8_gemm_work_pieces(int m, int n, int k, int block_n, int split_k, int num_sms, int cta, int* pieces,
                            int max_pieces) {
    if (!shape_ok(m, n, k) || (block_n != 128 && block_n != 256) || num_sms < 1 || cta < 0 || !pieces) return -1;
    const int kb = k / kBlockK;
    if (split_k < kStreamK || split_k == 0 || split_k > kb || split_k > kMaxSplits) return -1;
    rf::GemmParams p;
    p.k = k;
    p.tiles_m = (m + 127) / 128;
    p.tiles_n = (n + block_n - 1) / block_n;
    p.splits = split_k == kStreamK ? 1 : split_k;
    p.sk_tiles = split_k == kStreamK ? rf::gemm_streamk_tiles(p.tiles_m * p.tiles_n, num_sms) : 0;
    const int total = p.tiles_m * p.tiles_n * p.splits;
    const int grid = (total < num_sms && p.sk_tiles == 0) ? total : num_sms;
    if (cta >= grid) return 0;
    return rf::fp8_gemm_walk_pieces(p, cta, grid, pieces, max_pieces);
}

size_t rf_fp8_gemm_workspace_bytes(int m, int n, int k, int split_k) {
    if (!shape_ok(m, n, k) || split_k < kStreamK) return 0;
    rf::DeviceState* st = rf::device_state();
    const int num_sms = st ? st->num_sms : 148;      // (no GPU: the answer for a B200)
    const int kb = k / kBlockK;
    if (split_k > kb) split_k = kb;
    if (split_k > kMaxSplits) split_k = kMaxSplits;
    // (the reference's layout may have another plan, and runs a stream-K one as a plain pass)
    size_t bytes = 0;
    for (bool mn_major : {false, true}) {
        const GemmPlan plan = choose_plan(m, n, k, num_sms, split_k, mn_major);
        size_t need = plan.splits > 1 ? (size_t)plan.splits * m * n * sizeof(float) : 0;
        if (plan.splits == kStreamK && !mn_major) need = rf::gemm_streamk_bytes(plan.block_n, num_sms);
        if (need > bytes) bytes = need;
    }
    return bytes;
}

int rf_fp8_gemm(const void* a, const void* b, const float* as, const float* bs, void* c, int m, int n, int k,
                int split_k, void* workspace, size_t workspace_bytes, rf_stream_t stream) {
    return gemm_impl(a, b, as, bs, c, m, n, k, split_k, workspace, workspace_bytes, false,
                     reinterpret_cast<cudaStream_t>(stream));
}

int rf_fp8_gemm_nsplit(const void* a, const void* b_shard, const float* as, const float* bs_shard,
                       void* const* c_all, int m, int n_total, int k, int rank, int world, rf_stream_t stream) {
    if (world < 1 || world > 8 || rank < 0 || rank >= world || n_total % world != 0) return RF_ERR_BAD_SHAPE;
    const int n_loc = n_total / world;
    if (n_loc % 128 != 0) return RF_ERR_BAD_SHAPE;     // shards must keep whole 128-wide scale blocks
    if (!c_all) return RF_ERR_NULL_POINTER;
    if (world == 1)
        return gemm_impl(a, b_shard, as, bs_shard, c_all[0], m, n_total, k, 1, nullptr, 0, true,
                         reinterpret_cast<cudaStream_t>(stream));
    return gemm_impl(a, b_shard, as, bs_shard, nullptr, m, n_loc, k, 1, nullptr, 0, true,
                     reinterpret_cast<cudaStream_t>(stream), c_all, world, n_total, rank * n_loc);
}

int rf_fp8_gemm_colmajor(const void* a, const void* b, const float* as, const float* bs, void* c, int m, int n,
                         int k, void* workspace, size_t workspace_bytes, rf_stream_t stream) {
    return gemm_impl(a, b, as, bs, c, m, n, k, 0, workspace, workspace_bytes, workspace == nullptr,
                     reinterpret_cast<cudaStream_t>(stream), nullptr, 1, 0, 0, true);
}

int rf_fp8_gemm_colmajor_fnuz(const void* a, const void* b, const float* as, const float* bs, void* c, int m, int n,
                              int k, void* workspace, size_t workspace_bytes, rf_stream_t stream) {
    return gemm_impl(a, b, as, bs, c, m, n, k, 0, workspace, workspace_bytes, workspace == nullptr,
                     reinterpret_cast<cudaStream_t>(stream), nullptr, 1, 0, 0, true, true);
}

void run(void* a, void* b, void* as, void* bs, void* c, int m, int n, int k, PerfMetrics* metrics,
         rf_stream_t stream) {
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (metrics) {
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        cudaEventRecord(e0, s);
    }
    int rc = gemm_impl(a, b, static_cast<const float*>(as), static_cast<const float*>(bs), c, m, n, k, 0, nullptr, 0,
                       true, s);
    if (rc != RF_OK) {
        fprintf(stderr, "Error: fp8 gemm failed (status %d) for M=%d, K=%d, N=%d\n", rc, m, k, n);
        abort();
    }
    if (metrics) {
        cudaEventRecord(e1, s);
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (metrics->count < 1) metrics->count = 1;
        strncpy(metrics->entries[0].name, "gemm", sizeof(metrics->entries[0].name) - 1);
        metrics->entries[0].time = ms;
        metrics->entries[0].gflops = ms > 0.f ? (float)(2.0 * m * n * k / (ms * 1e-3) / 1e9) : 0.f;
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }
}

}  // extern "C"
