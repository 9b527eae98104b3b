// Work items of the FP8 GEMM kernels: tile numbering and the sequence of pieces a CTA (or CTA pair) works through.
#pragma once
#include "fp8_gemm.h"

namespace rf {

struct TileCoord {
    int m_blk, n_blk;
};

// Tile number -> tile.  Consecutive tiles walk down M inside a band of GROUP_M row blocks before moving to
// the next column block, so the CTAs that run concurrently share B tiles (and A bands) in L2.
__device__ __forceinline__ TileCoord decode_tile(int tile, int tiles_m, int tiles_n) {
    // (This runs once per tile in every role, on the epilogue's critical path between two tiles: one integer
    // division, and shifts for the full bands.  Measured: the earlier form with five divisions, together with two
    // 64-bit divisions for the K range, cost the epilogue about 1400 cycles per tile, the present one 600.)
    constexpr int GROUP_M = 8;
    TileCoord t;
    const int group = GROUP_M * tiles_n;
    const int band = tile / group;
    const int first_m = band * GROUP_M;
    const int band_rows = min(GROUP_M, tiles_m - first_m);
    const int in_band = tile - band * group;
    if (band_rows == GROUP_M) {
        t.m_blk = first_m + (in_band & (GROUP_M - 1));
        t.n_blk = in_band >> 3;
    } else {
        t.n_blk = in_band / band_rows;
        t.m_blk = first_m + in_band - t.n_blk * band_rows;
    }
    return t;
}

// One stretch of work of a CTA: K blocks [kb0, kb1) of work item `item` = tile * splits + K-slice number.
struct Piece {
    int item, kb0, kb1;
};

// The sequence of pieces a CTA (or pair) works through in a plain launch: work items unit, unit + n_units, ... (a work
// item is a tile, or one K slice of a tile; the K slices of one tile are adjacent).  Producer, MMA issuers and epilogue
// each walk their own copy.  (One register of state: the epilogue's register budget is tight and its allocation fragile.)
struct PlainWalker {
    int w;                     // the work item drawn last
    __host__ __device__ __forceinline__ PlainWalker(const GemmParams&, int unit, int n_units, int) { w = unit - n_units; }
    __host__ __device__ __forceinline__ bool next(Piece& pc, const GemmParams& p, int n_units, int kb_total) {
        w += n_units;
        if (w >= p.tiles_m * p.tiles_n * p.splits) return false;
        pc.item = w;
        if (p.splits == 1) {
            pc.kb0 = 0;
            pc.kb1 = kb_total;
        } else {
            // (k / 128 < 2^24 and splits <= 64: the products fit 32 bits)
            const int split = w % p.splits;
            pc.kb0 = kb_total * split / p.splits;
            pc.kb1 = kb_total * (split + 1) / p.splits;
        }
        return true;
    }
};

}  // namespace rf
