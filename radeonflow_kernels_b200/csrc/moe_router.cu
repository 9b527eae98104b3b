// Router GEMM of the MoE layer on sm_100a: logits[t, e] = fp16(X[t,:] . W[e,:] + bias[e]).
//
// Replaces the PyTorch router matmul (scripts/gen_submission.py:400).  One CTA per 128-row tile, warp-specialised:
//   warp 0     TMA producer: A tile [128 x 64] fp16 and one box of the weight's rows x 64, both K-major, 128-byte swizzle
//   warp 1     MMA issuer: 4 x tcgen05.mma.kind::f16 (128 x N x 16) per stage, whole K accumulated in TMEM
//   warps 4-11 epilogue of the previous tile while the next tile's MMAs run
//
// What bounds it: one tile's K loop.  Producer and issuer run on one lane each: 128 tokens, K = 7168, operands in L2, us as
// whole warps that vote and elect at every step / now: 4 experts 28.5 / 19.0, 32 experts 31.3 / 21.9, 256 experts 36.7 /
// 35.7 (there four MMAs of 128 cycles are the step); 8192 tokens 33.0 / 27.2.  Two K steps per stage change nothing (21.5).
// N is the experts rounded up to 16, and the stages are as small as that allows and as many as fit: with boxes and MMAs of
// 256 rows for 32 experts 128 tokens took 42.1 us (32.0 with 20 KB stages).  (K is not split over CTAs: sums in another order
// round single logits the other way, and a token then chooses another expert.)
#include "ptx.cuh"
#include "moe_kernels.h"

namespace rf {

namespace {

constexpr int BM = 128;
constexpr int BN = 256;          // largest MMA N, TMEM columns per accumulator buffer
constexpr int BK = 64;           // 128 bytes of fp16: one swizzle row
constexpr int UMMA_K = 16;
constexpr int MAX_STAGES = 9;
constexpr int RING_BYTES = 192 * 1024;
constexpr int A_BYTES = BM * BK * 2;        // 16 KB; B: 128 bytes for each of the MMA's N rows
constexpr int NUM_NON_EPI_WARPS = 4;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 32 * (NUM_NON_EPI_WARPS + EPI_WARPS);
constexpr int SLAB_BYTES = 32 * 128;
constexpr int NBUF = 2;
constexpr int TMEM_COLS = NBUF * BN;
constexpr int BAR_BYTES = (2 * MAX_STAGES + 2 * NBUF) * 8 + 16;
constexpr int SMEM_BYTES = RING_BYTES + EPI_WARPS * SLAB_BYTES + BAR_BYTES + 1024;

__global__ void __launch_bounds__(THREADS, 1)
moe_router_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                  const __grid_constant__ CUtensorMap tma_out, const MoeRouterParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t slab_base = smem_base + RING_BYTES;
    const uint32_t bar_base = slab_base + EPI_WARPS * SLAB_BYTES;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (MAX_STAGES + s); };
    auto tmem_full_bar = [&](int b) { return bar_base + 8u * (2 * MAX_STAGES + b); };
    auto tmem_empty_bar = [&](int b) { return bar_base + 8u * (2 * MAX_STAGES + NBUF + b); };
    const uint32_t tmem_slot = bar_base + 8u * (2 * MAX_STAGES + 2 * NBUF);
    uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    griddep_launch_dependents();

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tma_a);
        for (int s = 0; s < MAX_STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < NBUF; ++b) {
            mbar_init(tmem_full_bar(b), 1);
            mbar_init(tmem_empty_bar(b), EPI_WARPS);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot_ptr);

    griddep_wait();

    const int total_work = (p.n_rows + BM - 1) / BM;
    const int k_steps = p.k / BK;
    const int n_mma = (p.n_out + 15) & ~15;
    const uint32_t stage_bytes = A_BYTES + n_mma * (BK * 2);
    const uint32_t n_stages = min((uint32_t)MAX_STAGES, RING_BYTES / stage_bytes);

    if (warp == 0) {
        // ------------------------------------------------------ TMA producer (one lane, like the issuer)
        if (elect_one()) {
            uint32_t it = 0, s = 0, ph = 0;       // loads so far; stage, parity of its use
            bool ok = true;
            for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x) {
                const int row0 = w * BM;
                for (int ks = 0; ks < k_steps; ++ks, ++it) {
                    ok = mbar_wait(empty_bar(s), ph ^ 1, p.status, kErrProducerWait, p.launch_tag);
                    if (!ok) break;
                    mbar_expect_tx(full_bar(s), stage_bytes);
                    const uint32_t sa = smem_base + s * stage_bytes;
                    tma_load_2d(sa, &tma_a, full_bar(s), ks * BK, row0);
                    tma_load_2d(sa + A_BYTES, &tma_b, full_bar(s), ks * BK, 0);
                    if (++s == n_stages) { s = 0; ph ^= 1; }
                }
            }
            finish_producer(ok, it, n_stages, empty_bar(0), p.status, kErrProducerWait, p.launch_tag);
        }
        __syncwarp();
    } else if (warp == 1) {
        // -------------------------------------------------------- MMA issuer
        if (elect_one()) {
            const uint32_t idesc = make_idesc(BM, n_mma, /*f16*/ 0, /*f16*/ 0, 0, 0);
            uint32_t s = 0, ph = 0, tcount = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++tcount) {
                const int buf = tcount & 1;
                const uint32_t bph = (tcount >> 1) & 1;
                ok = mbar_wait(tmem_empty_bar(buf), bph ^ 1, p.status, kErrMmaWaitTmem, p.launch_tag);
                if (!ok) break;
                const uint32_t d = tmem_base + buf * BN;
                for (int ks = 0; ks < k_steps; ++ks) {
                    ok = mbar_wait(full_bar(s), ph, p.status, kErrMmaWaitFull, p.launch_tag);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t sa = smem_base + s * stage_bytes;
                    const uint64_t adesc = smem_desc_kmajor_sw128(sa);
                    const uint64_t bdesc = smem_desc_kmajor_sw128(sa + A_BYTES);
#pragma unroll
                    for (int j = 0; j < BK / UMMA_K; ++j)
                        umma_f16(d, adesc + 2 * j, bdesc + 2 * j, idesc, (ks > 0 || j > 0) ? 1u : 0u);
                    umma_commit(empty_bar(s));
                    if (ks == k_steps - 1) umma_commit(tmem_full_bar(buf));
                    if (++s == n_stages) { s = 0; ph ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp >= NUM_NON_EPI_WARPS) {
        // ---------------------------------------------------------- epilogue
        const int ew = warp - NUM_NON_EPI_WARPS;
        const int quad = warp & 3;
        const int grp_c = ew >> 2;                         // column group 0/1
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
        const uint32_t slab = slab_base + ew * SLAB_BYTES;
        const uint32_t my_row = slab + lane * 128;
        __half* out = static_cast<__half*>(p.out);
        uint32_t tcount = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++tcount) {
            const int buf = tcount & 1;
            const uint32_t bph = (tcount >> 1) & 1;
            if (!mbar_wait(tmem_full_bar(buf), bph, p.status, kErrEpilogueWait, p.launch_tag)) { ok = false; break; }
            tc_fence_after();

            const int slab_row0 = w * BM + quad * 32;
            const int rows_valid = p.n_rows - slab_row0;         // <= 0: nothing to store
            const bool full_slab = rows_valid >= 32;
            const bool my_row_ok = lane < rows_valid;
            const uint32_t tbase = lane_addr + buf * BN;
            // 64 output columns (one 128-byte slab row) per iteration
            constexpr int OUT_COLS = BN / 2;                     // per epilogue warp
#pragma unroll 1
            for (int c64 = 0; c64 < OUT_COLS; c64 += 64) {
                const int out_col = grp_c * OUT_COLS + c64;
                uint32_t packed[32];                              // 64 fp16 values of this thread's row
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float v[32];
                    tmem_ld32_async(tbase + grp_c * 128 + c64 + h * 32, v);
                    tmem_ld_fence(v);
                    if (p.bias != nullptr) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const int col = out_col + h * 32 + j;
                            v[j] += col < p.n_out ? p.bias[col] : 0.f;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) packed[h * 16 + j] = pack_f16x2(v[2 * j], v[2 * j + 1]);
                }
                if (out_col >= p.n_out || rows_valid <= 0) continue;
                if (p.tma_store && full_slab) {
                    if (lane == 0) tma_store_wait_read<0>();
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        st_shared_v4(my_row + ((j ^ (lane & 7)) << 4), packed[4 * j], packed[4 * j + 1],
                                     packed[4 * j + 2], packed[4 * j + 3]);
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_2d(&tma_out, slab, out_col, slab_row0);
                        tma_store_commit();
                    }
                } else if (my_row_ok) {
                    __half* orow = out + (size_t)(slab_row0 + lane) * p.n_out + out_col;
                    if (out_col + 64 <= p.n_out && (p.n_out % 8) == 0) {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            *reinterpret_cast<uint4*>(orow + 8 * j) =
                                make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
                    } else {
                        // ragged column tail (router with few experts): element stores, fully unrolled
                        // so `packed` stays in registers
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const __half2 hv = *reinterpret_cast<const __half2*>(&packed[j]);
                            if (out_col + 2 * j < p.n_out) orow[2 * j] = __low2half(hv);
                            if (out_col + 2 * j + 1 < p.n_out) orow[2 * j + 1] = __high2half(hv);
                        }
                    }
                }
            }
            // every TMEM read of this buffer by this warp has completed (loads are fenced above)
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tmem_empty_bar(buf));
        }
        if (lane == 0) tma_store_wait_read<0>();   // the slab has been read; the writes complete with the grid
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

}  // namespace

cudaError_t moe_router_launch(const CUtensorMap& tma_x, const CUtensorMap& tma_w, const CUtensorMap& tma_out,
                              const MoeRouterParams& p, int num_sms, bool overlap, cudaStream_t stream) {
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e =
            cudaFuncSetAttribute(moe_router_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    const int tiles = (p.n_rows + BM - 1) / BM;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles < num_sms ? tiles : num_sms, 1, 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, moe_router_kernel, tma_x, tma_w, tma_out, p);
}

}  // namespace rf
