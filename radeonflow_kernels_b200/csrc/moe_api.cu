// C-ABI entry points of the MoE layer (declared in include/rf_b200.h): stage sequencing, workspace
// carving, per-expert tensor-map cache, per-stage timing.  Host code only; kernels live in
// moe_route.cu, moe_router.cu and moe_gemm.cu.
#include "../../include/rf_b200.h"
#include "host_util.h"
#include "moe_kernels.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

namespace {

using rf::DeviceState;

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

bool is_pow2(int v) { return v > 0 && (v & (v - 1)) == 0; }

int validate_params(const InputParams& q) {
    const long long t = (long long)q.batch_size * q.seq_len;
    if (t <= 0 || t > (1 << 24)) return RF_ERR_BAD_SHAPE;
    if (q.d_hidden <= 0 || q.d_hidden % 64 != 0 || q.d_expert <= 0 || q.d_expert % 64 != 0) return RF_ERR_BAD_SHAPE;
    if (!is_pow2(q.n_routed_experts) || q.n_routed_experts > 256) return RF_ERR_UNSUPPORTED;
    if (q.n_experts_per_token < 1 || q.n_experts_per_token > 8 || q.n_experts_per_token > q.n_routed_experts)
        return RF_ERR_UNSUPPORTED;
    if (q.n_shared_experts < 1) return RF_ERR_UNSUPPORTED;
    return RF_OK;
}

// ---------------------------------------------------------------- per-expert tensor-map cache --
// Weights are static across calls, so the device array of tensor maps built for a set of weight
// pointers is kept and found again by (device, pointers, shape).  The cache holds 2048 sets by default (a
// model of 100 MoE layers uses about 300) and evicts the least recently used one; a set used by the
// grouped GEMM that is being enqueued is never evicted, and an evicted array is freed only after an event
// recorded on the calling stream has completed, so a kernel that was enqueued with it can still read it.
// (That, like the shared tile-list scratch, assumes what the reference also assumes: the MoE entry points
// of one device are issued on one stream at a time.)  A miss costs one cudaMalloc and one blocking copy;
// it happens at a layer's first call only.
struct MapSet {
    int device;
    int rows, cols, box_rows, box_cols;
    std::vector<const void*> ptrs;
    CUtensorMap* dev_maps;
    unsigned long long last_call;
};
struct RetiredMaps {
    int device;
    CUtensorMap* dev_maps;
    cudaEvent_t done;
};
size_t g_max_map_sets = 2048;
std::mutex g_map_mu;
std::vector<MapSet> g_map_sets;
std::vector<RetiredMaps> g_retired;
unsigned long long g_map_call = 0;      // one number per grouped GEMM being enqueued

void begin_map_call() {
    std::lock_guard<std::mutex> lock(g_map_mu);
    ++g_map_call;
}

// Frees retired arrays whose event has completed (never blocks).
void reap_retired_locked(int dev) {
    for (size_t i = 0; i < g_retired.size();) {
        RetiredMaps& r = g_retired[i];
        if (r.device == dev && cudaEventQuery(r.done) == cudaSuccess) {
            cudaFree(r.dev_maps);
            cudaEventDestroy(r.done);
            g_retired.erase(g_retired.begin() + i);
        } else {
            ++i;
        }
    }
    cudaGetLastError();     // cudaErrorNotReady from the queries is not an error
}

// Row-major fp16 matrices [rows, cols]; one map per pointer; returns a device array.
const CUtensorMap* weight_maps(const void* const* ptrs, int count, int rows, int cols, int box_rows, int box_cols,
                               cudaStream_t stream) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(g_map_mu);
    for (MapSet& m : g_map_sets) {
        if (m.device == dev && m.rows == rows && m.cols == cols && m.box_rows == box_rows && m.box_cols == box_cols &&
            (int)m.ptrs.size() == count && memcmp(m.ptrs.data(), ptrs, sizeof(void*) * count) == 0) {
            m.last_call = g_map_call;
            return m.dev_maps;
        }
    }
    std::vector<CUtensorMap> host(count);
    for (int i = 0; i < count; ++i) {
        if (!ptrs[i] || ((uintptr_t)ptrs[i] & 15)) return nullptr;
        if (!rf::encode_tma_2d(&host[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, ptrs[i], (uint64_t)rows, (uint64_t)cols,
                               (uint64_t)cols * 2, (uint32_t)box_rows, (uint32_t)box_cols, true))
            return nullptr;
    }
    reap_retired_locked(dev);
    MapSet m;
    m.device = dev;
    m.rows = rows; m.cols = cols; m.box_rows = box_rows; m.box_cols = box_cols;
    m.ptrs.assign(ptrs, ptrs + count);
    m.dev_maps = nullptr;
    m.last_call = g_map_call;
    if (cudaMalloc(&m.dev_maps, sizeof(CUtensorMap) * count) != cudaSuccess) return nullptr;
    if (cudaMemcpy(m.dev_maps, host.data(), sizeof(CUtensorMap) * count, cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaFree(m.dev_maps);
        return nullptr;
    }
    if (g_map_sets.size() >= g_max_map_sets) {
        // least recently used set that the call in progress does not use
        size_t victim = g_map_sets.size();
        for (size_t i = 0; i < g_map_sets.size(); ++i)
            if (g_map_sets[i].last_call != g_map_call &&
                (victim == g_map_sets.size() || g_map_sets[i].last_call < g_map_sets[victim].last_call))
                victim = i;
        if (victim < g_map_sets.size()) {
            RetiredMaps r{g_map_sets[victim].device, g_map_sets[victim].dev_maps, nullptr};
            // kernels already enqueued on this stream may still read the array: free it after they are done
            if (cudaEventCreateWithFlags(&r.done, cudaEventDisableTiming) == cudaSuccess &&
                cudaEventRecord(r.done, stream) == cudaSuccess)
                g_retired.push_back(r);
            // (if the event could not be made the array is leaked rather than freed under a running kernel)
            g_map_sets.erase(g_map_sets.begin() + victim);
        }
    }
    g_map_sets.push_back(m);
    return m.dev_maps;
}

// Grid cap of the grouped GEMMs enqueued by this host thread (0 = one CTA per SM): the expert-parallel layer
// lowers it while its dispatch kernel owns a few SMs.
thread_local int g_grid_limit = 0;

// ------------------------------------------------------------------------------ aux scratch --
struct Aux {
    rf::MoeTile* tiles;
    int* counters;         // moe_tile_list_launch
    int* sort_scratch;
};

// row tiles of `rows` expanded rows in n_groups groups and of n_alt rows of the alt group
size_t max_tiles(int rows, int n_groups, int n_alt) {
    return (size_t)rows / rf::kMoeTileRows + n_groups + (size_t)n_alt / rf::kMoeTileRows + 2;
}

// n_tokens: of a layer, whose tiles may include the shared expert's and whose pairs are sorted; 0 elsewhere
bool carve_aux(Aux* a, int rows, int n_groups, int n_tokens) {
    const size_t tile_bytes = align_up(max_tiles(rows, n_groups, n_tokens) * sizeof(rf::MoeTile), 256);
    const size_t sort_bytes = n_tokens > 0 ? align_up(rf::moe_topk_counts_bytes(n_tokens, n_groups), 256) : 0;
    char* base = static_cast<char*>(rf::device_scratch(tile_bytes + 256 + sort_bytes, rf::kScratchMoeAux));
    if (!base) return false;
    a->tiles = reinterpret_cast<rf::MoeTile*>(base);
    a->counters = reinterpret_cast<int*>(base + tile_bytes);
    a->sort_scratch = reinterpret_cast<int*>(base + tile_bytes + 256);
    return true;
}

// ------------------------------------------------------------------------------ stage timer --
struct StageTimer {
    PerfMetrics* pm;
    cudaStream_t stream;
    cudaEvent_t ev[26];
    int used = 0;
    struct Span { int idx, a, b; double flops; };
    std::vector<Span> spans;
    StageTimer(PerfMetrics* m, cudaStream_t s) : pm(m), stream(s) {}
    int mark() {
        if (!pm || used >= 26) return -1;
        cudaEventCreate(&ev[used]);
        cudaEventRecord(ev[used], stream);
        return used++;
    }
    void span(int idx, int a, int b, double flops) {
        if (pm && a >= 0 && b >= 0) spans.push_back({idx, a, b, flops});
    }
    void finish() {
        if (!pm) return;
        static const char* names[12] = {"overall", "moe_misc", "transpose", "routed_fc1", "routed_fc2", "shared_fc1",
                                        "shared_fc2", "routed_fc1_reduce", "routed_fc2_reduce", "shared_fc1_reduce",
                                        "shared_fc2_reduce", "reduce_output"};
        pm->count = 12;
        for (int i = 0; i < 12; ++i) {
            memset(pm->entries[i].name, 0, sizeof(pm->entries[i].name));
            strncpy(pm->entries[i].name, names[i], sizeof(pm->entries[i].name) - 1);
            pm->entries[i].time = 0.f;
            pm->entries[i].gflops = 0.f;
        }
        if (used > 0) cudaEventSynchronize(ev[used - 1]);
        for (const Span& s : spans) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ev[s.a], ev[s.b]);
            pm->entries[s.idx].time += ms;
            if (ms > 0.f) pm->entries[s.idx].gflops = (float)(s.flops / (ms * 1e-3) / 1e9);
        }
        for (int i = 0; i < used; ++i) cudaEventDestroy(ev[i]);
    }
};

// Rows of the alt group of a grouped GEMM (the shared expert): `rows` rows of x [rows, k], results in out.
struct AltGroup {
    const void* x = nullptr;
    int rows = 0;
    void* out = nullptr;
};

// Result rows stored through a table of return addresses instead of in order.
struct RowScatter {
    const int* meta = nullptr;
    const rf::PeerPtrs* dst = nullptr;
};

bool encode_row_maps(rf::MoeRowMaps* m, const void* x, int rows, int k) {
    uint32_t box_rows = 16;
    for (CUtensorMap& map : m->box) {
        if (!rf::encode_tma_2d(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, (uint64_t)rows, (uint64_t)k,
                               (uint64_t)k * 2, box_rows, 64, true))
            return false;
        box_rows += 16;
    }
    return true;
}

int build_tiles(const int* offsets_dev, int n_groups, int alt_rows, const Aux& aux, cudaStream_t stream) {
    return rf::moe_tile_list_launch(offsets_dev, n_groups, alt_rows, aux.tiles, aux.counters, stream) == cudaSuccess
               ? RF_OK : RF_ERR_CUDA;
}

// The `nth` grouped GEMM (< kMoeItemCounters) over the row tiles built last in `aux`: rows of `x` [n_rows, k] by
// per-group weights (w2_host: SwiGLU of the two products).  With alt.rows > 0 the weight lists hold one entry more, the
// alt group's, behind the n_groups others.
int grouped_gemm(int nth, const void* x, int n_rows, const void* const* w_host, const void* const* w2_host, int n_groups,
                 int n_out, int k, void* out, const Aux& aux, DeviceState* st, cudaStream_t stream,
                 const AltGroup& alt = {}, const RowScatter& scatter = {}, bool overlap = false) {
    if (n_rows <= 0 && alt.rows <= 0) return RF_OK;
    // result rows leave as 16-byte stores
    if (((uintptr_t)out | (uintptr_t)alt.out) & 15) return RF_ERR_CUDA;
    const int n_sets = n_groups + (alt.rows > 0 ? 1 : 0);
    begin_map_call();
    // [K, N] row-major, box 64 K-rows x 64 N
    const CUtensorMap* maps = weight_maps(w_host, n_sets, k, n_out, 64, 64, stream);
    const CUtensorMap* maps2 = w2_host ? weight_maps(w2_host, n_sets, k, n_out, 64, 64, stream) : nullptr;
    if (!maps || (w2_host && !maps2)) return RF_ERR_CUDA;
    rf::MoeRowMaps mx, ma;
    if (n_rows > 0 && !encode_row_maps(&mx, x, n_rows, k)) return RF_ERR_CUDA;
    if (alt.rows > 0 && !encode_row_maps(&ma, alt.x, alt.rows, k)) return RF_ERR_CUDA;
    if (alt.rows <= 0) ma = mx;
    if (n_rows <= 0) mx = ma;
    rf::MoeGemmParams p;
    p.tiles = aux.tiles;
    p.tile_count = aux.counters;
    p.next_item = aux.counters + 1 + nth;
    p.w_maps = maps;
    p.w2_maps = maps2;
    p.out = out;
    p.alt_group = alt.rows > 0 ? n_groups : -1;
    p.alt_out = alt.out;
    p.n_out = n_out;
    p.k = k;
    p.scatter_meta = scatter.meta;
    if (scatter.dst) p.scatter_dst = *scatter.dst;
    else memset(&p.scatter_dst, 0, sizeof p.scatter_dst);
    p.status = st->status;
    p.launch_tag = rf::next_launch_tag();
    const int ctas = g_grid_limit > 0 && g_grid_limit < st->num_sms ? g_grid_limit : st->num_sms;
    return rf::moe_gemm_launch(w2_host != nullptr, mx, ma, p, ctas, overlap, stream) == cudaSuccess ? RF_OK : RF_ERR_CUDA;
}

// logits [n_rows, n_out] = x [n_rows, k] . w [n_out, k]^T + bias
int router_gemm(const void* x, const void* w, const float* bias, int n_rows, int n_out, int k, void* out,
                DeviceState* st, cudaStream_t stream, bool overlap = false) {
    CUtensorMap tx, tw, to;
    if (((uintptr_t)w & 15) ||
        !rf::encode_tma_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, (uint64_t)n_rows, (uint64_t)k, (uint64_t)k * 2,
                           128, 64, true) ||
        !rf::encode_tma_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, w, (uint64_t)n_out, (uint64_t)k, (uint64_t)k * 2,
                           (uint32_t)(n_out + 15) / 16 * 16, 64, true))
        return RF_ERR_CUDA;
    rf::MoeRouterParams p;
    p.tma_store = n_out % 64 == 0;
    if (p.tma_store) {
        if (!rf::encode_tma_2d(&to, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, out, (uint64_t)n_rows, (uint64_t)n_out,
                               (uint64_t)n_out * 2, 32, 64, true))
            return RF_ERR_CUDA;
    } else {
        to = tx;
    }
    p.bias = bias;
    p.out = out;
    p.n_rows = n_rows;
    p.n_out = n_out;
    p.k = k;
    p.status = st->status;
    p.launch_tag = rf::next_launch_tag();
    const int ctas = g_grid_limit > 0 && g_grid_limit < st->num_sms ? g_grid_limit : st->num_sms;
    return rf::moe_router_launch(tx, tw, to, p, ctas, overlap, stream) == cudaSuccess ? RF_OK : RF_ERR_CUDA;
}

// `fill_expanded`: the gathered token rows go to expanded_seq_input (the reference's expand_input output, a stage
// tensor its checker compares); false: that buffer is left untouched and the rows pass through expanded_fc2_output,
// which has their size and is first written by fc2.
int moe_layer(MoEInputRaw* in, bool compute_router, const float* router_bias, cudaStream_t stream,
              PerfMetrics* metrics, bool fill_expanded) {
    if (!in) return RF_ERR_NULL_POINTER;
    const InputParams& q = in->params;
    int rc = validate_params(q);
    if (rc != RF_OK) return rc;
    const int T = q.batch_size * q.seq_len;
    const int d = q.d_hidden, f = q.d_expert, E = q.n_routed_experts, K = q.n_experts_per_token;
    const int fs = f * q.n_shared_experts;
    const int TK = T * K;
    const void* need[] = {in->expert_weight_gate, in->expert_weight_up, in->expert_weight_down, in->input_seq,
                          in->shared_expert_weight_gate, in->shared_expert_weight_up, in->shared_expert_weight_down,
                          in->expert_scores, in->seq_experts_index, in->seq_experts_softmax, in->source_rows,
                          in->permuted_experts, in->permuted_rows, in->first_token_offset, in->expanded_seq_input,
                          in->expanded_seq_softmax, in->rev_permuted_rows, in->expanded_fc1_output,
                          in->expanded_fc2_output, in->shared_fc1_output, in->shared_fc2_output, in->final_output};
    for (const void* ptr : need)
        if (!ptr) return RF_ERR_NULL_POINTER;
    if (compute_router && !in->router_weight) return RF_ERR_NULL_POINTER;
    // Before anything is enqueued: what is moved 16 bytes at a time (the logits by the top-k of 256 experts and by the router's
    // tile stores, the weights and rows by the TMA and the row kernels), and the rest by its element.
    const bool scores16 = compute_router ? E % 64 == 0 : E == 256;
    if (rf::misaligned({in->input_seq, in->shared_expert_weight_gate, in->shared_expert_weight_up,
                        in->shared_expert_weight_down, compute_router ? in->router_weight : nullptr,
                        scores16 ? in->expert_scores : nullptr, fill_expanded ? in->expanded_seq_input : nullptr,
                        in->expanded_fc1_output, in->expanded_fc2_output, in->shared_fc1_output, in->shared_fc2_output,
                        in->final_output}, 16) ||
        rf::misaligned({in->seq_experts_index, in->source_rows, in->permuted_experts, in->permuted_rows,
                        in->first_token_offset, in->rev_permuted_rows, compute_router ? router_bias : nullptr}, 4) ||
        rf::misaligned({in->expert_scores, in->seq_experts_softmax, in->expanded_seq_softmax}, 2))
        return RF_ERR_MISALIGNED;
    for (int e = 0; e < E; ++e)
        if (rf::misaligned({in->expert_weight_gate[e], in->expert_weight_up[e], in->expert_weight_down[e]}, 16))
            return RF_ERR_MISALIGNED;
    DeviceState* st = rf::device_state();
    if (!st) return RF_ERR_CUDA;
    Aux aux;
    if (!carve_aux(&aux, TK, E, T)) return RF_ERR_CUDA;

    StageTimer tm(metrics, stream);
    const int t_begin = tm.mark();

    // Each kernel of the layer is a programmatic dependent of the one before it (not with stage times, whose events lie in
    // between): 128 tokens, 32 experts spent 28 us on the starts of ten kernels.
    const bool overlap = !metrics;
    // A shared expert as wide as the routed ones joins their launches as one more group: alone, its 16 and 28 column blocks
    // (d 7168, f 2048) would occupy 22 and 38 % of the 74 CTA pairs while a small batch streams its weights.  With stage
    // times asked for it runs by itself, so that each of the reference's stages keeps a time of its own; the arithmetic is
    // the same.
    const bool merged = fs == f && !metrics;

    // ---- router GEMM (optional), softmax + top-k, counting sort with the row tiles, row gather  -> "moe_misc"
    if (compute_router) {
        rc = router_gemm(in->input_seq, in->router_weight, router_bias, T, E, d, in->expert_scores, st, stream, overlap);
        if (rc != RF_OK) return rc;
    }
    if (rf::moe_topk_launch(in->expert_scores, T, E, K, in->seq_experts_index, in->seq_experts_softmax,
                            in->source_rows, aux.sort_scratch, overlap, stream) != cudaSuccess)
        return RF_ERR_CUDA;
    if (rf::moe_permute_launch(in->seq_experts_index, in->source_rows, in->seq_experts_softmax, T, K, E,
                               in->permuted_experts, in->permuted_rows, in->first_token_offset, in->rev_permuted_rows,
                               in->expanded_seq_softmax, aux.sort_scratch, true, merged ? T : 0, aux.tiles, aux.counters,
                               overlap, stream) != cudaSuccess)
        return RF_ERR_CUDA;
    void* rows = fill_expanded ? in->expanded_seq_input : in->expanded_fc2_output;
    if (rf::moe_gather_rows_launch(in->input_seq, static_cast<const int*>(in->permuted_rows), T, TK, d * 2, rows,
                                   st->num_sms, overlap, stream) != cudaSuccess)
        return RF_ERR_CUDA;
    const int t_misc = tm.mark();
    tm.span(1, t_begin, t_misc, 0.0);

    // ---- experts: fc1 (gate and up in one pass, SwiGLU in the epilogue), fc2
    std::vector<const void*> wg(in->expert_weight_gate, in->expert_weight_gate + E),
        wu(in->expert_weight_up, in->expert_weight_up + E), wd(in->expert_weight_down, in->expert_weight_down + E);
    wg.push_back(in->shared_expert_weight_gate);
    wu.push_back(in->shared_expert_weight_up);
    wd.push_back(in->shared_expert_weight_down);
    AltGroup s1{in->input_seq, T, in->shared_fc1_output}, s2{in->shared_fc1_output, T, in->shared_fc2_output};
    rc = grouped_gemm(0, rows, TK, wg.data(), wu.data(), E, f, d, in->expanded_fc1_output, aux, st, stream,
                      merged ? s1 : AltGroup{}, RowScatter{}, overlap);
    if (rc != RF_OK) return rc;
    const int t_fc1 = tm.mark();
    tm.span(3, t_misc, t_fc1, 2.0 * TK * (double)f * d * 2);
    rc = grouped_gemm(1, in->expanded_fc1_output, TK, wd.data(), nullptr, E, d, f, in->expanded_fc2_output, aux, st, stream,
                      merged ? s2 : AltGroup{}, RowScatter{}, overlap);
    if (rc != RF_OK) return rc;
    const int t_fc2 = tm.mark();
    tm.span(4, t_fc1, t_fc2, 2.0 * TK * (double)f * d);

    // ---- shared expert over all tokens, unless it ran above
    int t_s2 = t_fc2;
    if (!merged) {
        if ((rc = build_tiles(nullptr, 0, T, aux, stream)) != RF_OK) return rc;
        rc = grouped_gemm(0, nullptr, 0, &wg[E], &wu[E], 0, fs, d, nullptr, aux, st, stream, s1);
        if (rc != RF_OK) return rc;
        const int t_s1 = tm.mark();
        tm.span(5, t_fc2, t_s1, 2.0 * T * (double)fs * d * 2);
        rc = grouped_gemm(1, nullptr, 0, &wd[E], nullptr, 0, d, fs, nullptr, aux, st, stream, s2);
        if (rc != RF_OK) return rc;
        t_s2 = tm.mark();
        tm.span(6, t_s1, t_s2, 2.0 * T * (double)fs * d);
    }

    // ---- weighted combine + shared add
    if (rf::moe_combine_launch(in->expanded_fc2_output, in->shared_fc2_output,
                               static_cast<const int*>(in->rev_permuted_rows), in->expanded_seq_softmax, T, K, d * 2,
                               in->final_output, overlap, stream) != cudaSuccess)
        return RF_ERR_CUDA;
    const int t_end = tm.mark();
    tm.span(11, t_s2, t_end, 0.0);
    tm.span(0, t_begin, t_end, 2.0 * (double)d * f * 3.0 * ((double)TK + (double)T * q.n_shared_experts));
    tm.finish();
    return RF_OK;
}

// rf_moe_set_fused_gather, or RF_MOE_FUSED_GATHER=1 at first use: rf_moe_forward and rf_run_from_python leave
// expanded_seq_input unwritten.  (Gathering inside the first expert GEMM's loader is slower than a pass of its own: with
// 16-byte cp.async copies a layer of 8192 tokens, 32 experts takes 6.07 ms, with TMA row gathers 5.65, with the pass
// 3.52.)
int g_fused_gather = -1;
bool fill_expanded_default() {
    if (g_fused_gather < 0) {
        const char* e = getenv("RF_MOE_FUSED_GATHER");
        g_fused_gather = (e && e[0] == '1') ? 1 : 0;
    }
    return g_fused_gather == 0;
}

}  // namespace

extern "C" {

int rf_moe_set_fused_gather(int on) {
    g_fused_gather = on ? 1 : 0;
    return RF_OK;
}

int rf_moe_set_grid_limit(int max_ctas) {
    if (max_ctas < 0) return RF_ERR_BAD_SHAPE;
    g_grid_limit = max_ctas;
    return RF_OK;
}

int rf_moe_set_map_cache_sets(int max_sets) {
    if (max_sets < 4) return RF_ERR_BAD_SHAPE;      // one grouped GEMM pins up to two sets
    std::lock_guard<std::mutex> lock(g_map_mu);
    g_max_map_sets = (size_t)max_sets;
    return RF_OK;
}

int run_topk(MoEInputRaw* input, rf_stream_t stream, PerfMetrics* metrics) {
    return moe_layer(input, false, nullptr, reinterpret_cast<cudaStream_t>(stream), metrics, true);
}

int rf_moe_forward(MoEInputRaw* input, const float* router_bias, rf_stream_t stream, PerfMetrics* metrics) {
    return moe_layer(input, true, router_bias, reinterpret_cast<cudaStream_t>(stream), metrics, fill_expanded_default());
}

size_t rf_moe_workspace_bytes(const InputParams* q) {
    if (!q || validate_params(*q) != RF_OK) return 0;
    const size_t T = (size_t)q->batch_size * q->seq_len, K = q->n_experts_per_token, E = q->n_routed_experts;
    const size_t d = q->d_hidden, f = q->d_expert, fs = f * q->n_shared_experts, TK = T * K;
    size_t b = 0;
    auto add = [&](size_t n) { b += align_up(n, 256); };
    add(T * E * 2);            // expert_scores
    add(TK * 4); add(TK * 2); add(TK * 4);           // seq_experts_index, seq_experts_softmax, source_rows
    add(TK * 4); add(TK * 4); add((E + 1) * 4);      // permuted_experts, permuted_rows, first_token_offset
    add(TK * d * 2); add(TK * 2); add(TK * 4);       // expanded_seq_input, expanded_seq_softmax, rev_permuted_rows
    add(TK * f * 2); add(TK * d * 2);                // expanded_fc1_output, expanded_fc2_output
    add(T * fs * 2); add(T * d * 2);                 // shared_fc1_output, shared_fc2_output
    return b;
}

int rf_moe_bind_workspace(MoEInputRaw* in, void* workspace, size_t workspace_bytes) {
    if (!in || !workspace) return RF_ERR_NULL_POINTER;
    const size_t need = rf_moe_workspace_bytes(&in->params);
    if (need == 0) return RF_ERR_BAD_SHAPE;
    if (workspace_bytes < need) return RF_ERR_WORKSPACE;
    if ((uintptr_t)workspace & 255) return RF_ERR_MISALIGNED;
    const InputParams* q = &in->params;
    const size_t T = (size_t)q->batch_size * q->seq_len, K = q->n_experts_per_token, E = q->n_routed_experts;
    const size_t d = q->d_hidden, f = q->d_expert, fs = f * q->n_shared_experts, TK = T * K;
    char* pcur = static_cast<char*>(workspace);
    auto take = [&](size_t n) { void* r = pcur; pcur += align_up(n, 256); return r; };
    if (!in->expert_scores) in->expert_scores = take(T * E * 2); else take(T * E * 2);
    in->seq_experts_index = take(TK * 4);
    in->seq_experts_softmax = take(TK * 2);
    in->source_rows = take(TK * 4);
    in->permuted_experts = take(TK * 4);
    in->permuted_rows = take(TK * 4);
    in->first_token_offset = take((E + 1) * 4);
    in->expanded_seq_input = take(TK * d * 2);
    in->expanded_seq_softmax = take(TK * 2);
    in->rev_permuted_rows = take(TK * 4);
    in->expanded_fc1_output = take(TK * f * 2);
    in->expanded_fc2_output = take(TK * d * 2);
    in->shared_fc1_output = take(T * fs * 2);
    in->shared_fc2_output = take(T * d * 2);
    return RF_OK;
}

void initialize_workspace(void** workspace) {
    // src/moe/moe.cpp:36-40: MAX_SEQ_LEN 8192, MAX_N_EXPERT_PER_TOKEN 4, 7168 / 2048, 32 experts
    InputParams q = {1, 8192, 7168, 2048, 32, 4, 1, 0};
    void* p = rf::device_scratch(rf_moe_workspace_bytes(&q), rf::kScratchMoeWork);
    if (workspace) *workspace = p;
}

int rf_run_from_python(int seq_len, int batch_size, int d_hidden, int d_expert, int n_routed_experts,
                       int n_experts_per_token, int n_shared_experts, unsigned long long input_seq,
                       unsigned long long expert_scores, const unsigned long long* expert_weight_gate_p,
                       const unsigned long long* expert_weight_up_p, const unsigned long long* expert_weight_down_p,
                       unsigned long long shared_expert_weight_gate, unsigned long long shared_expert_weight_up,
                       unsigned long long shared_expert_weight_down, unsigned long long router_weight,
                       unsigned long long final_output, rf_stream_t stream) {
    if (!expert_weight_gate_p || !expert_weight_up_p || !expert_weight_down_p) return RF_ERR_NULL_POINTER;
    MoEInputRaw in;
    memset(&in, 0, sizeof(in));
    in.params = InputParams{batch_size, seq_len, d_hidden, d_expert, n_routed_experts, n_experts_per_token,
                            n_shared_experts, 0};
    int rc = validate_params(in.params);
    if (rc != RF_OK) return rc;
    std::vector<void*> g(n_routed_experts), u(n_routed_experts), dn(n_routed_experts);
    for (int i = 0; i < n_routed_experts; ++i) {
        g[i] = reinterpret_cast<void*>(expert_weight_gate_p[i]);
        u[i] = reinterpret_cast<void*>(expert_weight_up_p[i]);
        dn[i] = reinterpret_cast<void*>(expert_weight_down_p[i]);
    }
    in.expert_weight_gate = g.data();
    in.expert_weight_up = u.data();
    in.expert_weight_down = dn.data();
    in.input_seq = reinterpret_cast<void*>(input_seq);
    in.shared_expert_weight_gate = reinterpret_cast<void*>(shared_expert_weight_gate);
    in.shared_expert_weight_up = reinterpret_cast<void*>(shared_expert_weight_up);
    in.shared_expert_weight_down = reinterpret_cast<void*>(shared_expert_weight_down);
    in.router_weight = reinterpret_cast<void*>(router_weight);
    in.expert_scores = reinterpret_cast<void*>(expert_scores);
    in.final_output = reinterpret_cast<void*>(final_output);
    const size_t need = rf_moe_workspace_bytes(&in.params);
    void* ws = rf::device_scratch(need, rf::kScratchMoeWork);
    if (!ws) return RF_ERR_CUDA;
    rc = rf_moe_bind_workspace(&in, ws, need);
    if (rc != RF_OK) return rc;
    return moe_layer(&in, expert_scores == 0, nullptr, reinterpret_cast<cudaStream_t>(stream), nullptr,
                     fill_expanded_default());
}

int rf_moe_topk(const void* expert_scores, int n_tokens, int n_experts, int top_k, void* seq_experts_index,
                void* seq_experts_softmax, void* source_rows, rf_stream_t stream) {
    if (!expert_scores || !seq_experts_index || !seq_experts_softmax || !source_rows) return RF_ERR_NULL_POINTER;
    if (n_tokens < 0 || !is_pow2(n_experts) || n_experts > 256 || top_k < 1 || top_k > 8 || top_k > n_experts)
        return RF_ERR_UNSUPPORTED;
    if (n_tokens == 0) return RF_OK;
    if (rf::misaligned({expert_scores}, n_experts == 256 ? 16 : 2) || rf::misaligned({seq_experts_softmax}, 2) ||
        rf::misaligned({seq_experts_index, source_rows}, 4))
        return RF_ERR_MISALIGNED;
    return rf::moe_topk_launch(expert_scores, n_tokens, n_experts, top_k, seq_experts_index, seq_experts_softmax,
                               source_rows, nullptr, false, reinterpret_cast<cudaStream_t>(stream)) == cudaSuccess
               ? RF_OK : RF_ERR_CUDA;
}

size_t rf_moe_permute_scratch_bytes(int n_items, int n_experts) {
    return rf::moe_permute_scratch_bytes(n_items, n_experts);
}

int rf_moe_permute(const void* seq_experts_index, const void* source_rows, const void* seq_experts_softmax,
                   int n_tokens, int n_experts, int top_k, void* permuted_experts, void* permuted_rows,
                   void* first_token_offset, void* rev_permuted_rows, void* expanded_seq_softmax, void* scratch,
                   rf_stream_t stream) {
    if (!seq_experts_index || !source_rows || !seq_experts_softmax || !permuted_experts || !permuted_rows ||
        !first_token_offset || !rev_permuted_rows || !expanded_seq_softmax || !scratch)
        return RF_ERR_NULL_POINTER;
    if (n_tokens < 0 || n_experts < 1 || n_experts > 1024 || top_k < 1) return RF_ERR_UNSUPPORTED;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n_tokens == 0)
        return cudaMemsetAsync(first_token_offset, 0, (n_experts + 1) * sizeof(int), s) == cudaSuccess ? RF_OK
                                                                                                        : RF_ERR_CUDA;
    if (rf::misaligned({seq_experts_index, source_rows, permuted_experts, permuted_rows, first_token_offset,
                        rev_permuted_rows, scratch}, 4) ||
        rf::misaligned({seq_experts_softmax, expanded_seq_softmax}, 2))
        return RF_ERR_MISALIGNED;
    return rf::moe_permute_launch(seq_experts_index, source_rows, seq_experts_softmax, n_tokens, top_k, n_experts,
                                  permuted_experts, permuted_rows, first_token_offset, rev_permuted_rows,
                                  expanded_seq_softmax, scratch, false, 0, nullptr, nullptr, false, s) == cudaSuccess
               ? RF_OK : RF_ERR_CUDA;
}

int rf_moe_gather_rows(const void* input_seq, const void* permuted_rows, int n_tokens, int n_rows, int d_hidden,
                       void* expanded_seq_input, rf_stream_t stream) {
    if (!input_seq || !permuted_rows || !expanded_seq_input) return RF_ERR_NULL_POINTER;
    if (d_hidden <= 0 || d_hidden % 8 != 0 || n_tokens <= 0 || n_rows < 0) return RF_ERR_BAD_SHAPE;
    if (n_rows > 0 && (rf::misaligned({input_seq, expanded_seq_input}, 16) || rf::misaligned({permuted_rows}, 4)))
        return RF_ERR_MISALIGNED;
    DeviceState* st = rf::device_state();
    if (!st) return RF_ERR_CUDA;
    return rf::moe_gather_rows_launch(input_seq, static_cast<const int*>(permuted_rows), n_tokens, n_rows,
                                      d_hidden * 2, expanded_seq_input, st->num_sms, false,
                                      reinterpret_cast<cudaStream_t>(stream)) == cudaSuccess
               ? RF_OK : RF_ERR_CUDA;
}

int rf_moe_grouped_gemm(const void* x, int n_rows, const void* const* w_ptrs_host, const void* const* w2_ptrs_host,
                        const int* group_offsets_dev, int n_groups, int n_dim, int k_dim, void* out,
                        rf_stream_t stream) {
    if (!x || !w_ptrs_host || !group_offsets_dev || !out) return RF_ERR_NULL_POINTER;
    if (n_rows < 0 || n_groups < 1 || n_groups > 1024 || n_dim <= 0 || n_dim % 64 != 0 || k_dim <= 0 ||
        k_dim % 64 != 0)
        return RF_ERR_BAD_SHAPE;
    DeviceState* st = rf::device_state();
    if (!st) return RF_ERR_CUDA;
    if (n_rows == 0) return RF_OK;
    Aux aux;
    if (!carve_aux(&aux, n_rows, n_groups, 0)) return RF_ERR_CUDA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int rc = build_tiles(group_offsets_dev, n_groups, 0, aux, s);
    if (rc != RF_OK) return rc;
    return grouped_gemm(0, x, n_rows, w_ptrs_host, w2_ptrs_host, n_groups, n_dim, k_dim, out, aux, st, s);
}

int rf_moe_grouped_gemm_scatter(const void* x, int n_rows, const void* const* w_ptrs_host,
                                const int* group_offsets_dev, int n_groups, int n_dim, int k_dim,
                                const int* row_dest_dev, void* const* dest_all, int world, rf_stream_t stream) {
    if (!x || !w_ptrs_host || !group_offsets_dev || !row_dest_dev || !dest_all) return RF_ERR_NULL_POINTER;
    if (n_rows < 0 || n_groups < 1 || n_groups > 1024 || n_dim <= 0 || n_dim % 64 != 0 || k_dim <= 0 ||
        k_dim % 64 != 0 || world < 1 || world > 8)
        return RF_ERR_BAD_SHAPE;
    rf::PeerPtrs pp;
    for (int i = 0; i < 8; ++i) pp.p[i] = dest_all[i < world ? i : 0];
    for (int i = 0; i < world; ++i)
        if (!pp.p[i] || ((uintptr_t)pp.p[i] & 15)) return RF_ERR_NULL_POINTER;
    DeviceState* st = rf::device_state();
    if (!st) return RF_ERR_CUDA;
    if (n_rows == 0) return RF_OK;
    Aux aux;
    if (!carve_aux(&aux, n_rows, n_groups, 0)) return RF_ERR_CUDA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int rc = build_tiles(group_offsets_dev, n_groups, 0, aux, s);
    if (rc != RF_OK) return rc;
    return grouped_gemm(0, x, n_rows, w_ptrs_host, nullptr, n_groups, n_dim, k_dim, nullptr, aux, st, s, {},
                        RowScatter{row_dest_dev, &pp});
}

int rf_moe_router_gemm(const void* x, const void* router_weight, const float* router_bias, int n_tokens,
                       int n_experts, int d_hidden, void* expert_scores, rf_stream_t stream) {
    if (!x || !router_weight || !expert_scores) return RF_ERR_NULL_POINTER;
    if (n_tokens < 0 || n_experts < 1 || n_experts > 256 || d_hidden <= 0 || d_hidden % 64 != 0)
        return RF_ERR_BAD_SHAPE;
    // (whole 64-column pieces of a row leave as 16-byte stores where every row starts at a multiple of 16 bytes)
    if (n_tokens > 0 &&
        (rf::misaligned({x, router_weight}, 16) ||
         rf::misaligned({expert_scores}, n_experts >= 64 && n_experts % 8 == 0 ? 16 : 2) || rf::misaligned({router_bias}, 4)))
        return RF_ERR_MISALIGNED;
    DeviceState* st = rf::device_state();
    if (!st) return RF_ERR_CUDA;
    if (n_tokens == 0) return RF_OK;
    return router_gemm(x, router_weight, router_bias, n_tokens, n_experts, d_hidden, expert_scores, st,
                       reinterpret_cast<cudaStream_t>(stream));
}

int rf_moe_combine(const void* expanded_fc2_output, const void* shared_fc2_output, const void* rev_permuted_rows,
                   const void* expanded_seq_softmax, int n_tokens, int top_k, int d_hidden, void* final_output,
                   rf_stream_t stream) {
    if (!expanded_fc2_output || !shared_fc2_output || !rev_permuted_rows || !expanded_seq_softmax || !final_output)
        return RF_ERR_NULL_POINTER;
    if (n_tokens < 0 || top_k < 1 || top_k > 8 || d_hidden <= 0 || d_hidden % 8 != 0) return RF_ERR_BAD_SHAPE;
    if (n_tokens > 0 &&
        (rf::misaligned({expanded_fc2_output, shared_fc2_output, final_output}, 16) ||
         rf::misaligned({rev_permuted_rows}, 4) || rf::misaligned({expanded_seq_softmax}, 2)))
        return RF_ERR_MISALIGNED;
    return rf::moe_combine_launch(expanded_fc2_output, shared_fc2_output, static_cast<const int*>(rev_permuted_rows),
                                  expanded_seq_softmax, n_tokens, top_k, d_hidden * 2, final_output, false,
                                  reinterpret_cast<cudaStream_t>(stream)) == cudaSuccess
               ? RF_OK : RF_ERR_CUDA;
}

}  // extern "C"
