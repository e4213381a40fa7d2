// tile_rows.cuh -- the row of every edge of a tile of consecutive edges.
#pragma once

#include "common.cuh"

namespace mg {

// A block of kExpandThreads takes a tile of kExpandTile consecutive edges.
// The non-empty rows that start inside the tile are marked at their first edge,
// a prefix maximum over the tile then gives every edge its row.  Tile position
// q lives at q + q/32 (one padding word per 32: the per-thread runs of 16
// positions then fall on distinct banks).
constexpr int kExpandThreads = 256;
constexpr int kExpandPer = 16;
constexpr uint32_t kExpandTile = kExpandThreads * kExpandPer;

struct TileRows {
    uint32_t rowat[kExpandTile + kExpandTile / 32];
    uint32_t part[kExpandThreads];
    uint32_t r0, r1;
    __device__ __forceinline__ uint32_t row(uint32_t q) const { return rowat[q + (q >> 5)]; }
};

// last row in [0, n) with off[row] <= e (off[0] = 0 <= e)
__device__ __forceinline__ uint32_t last_row_at(const uint32_t *off, uint32_t n, uint64_t e) {
    uint32_t lo = 0, hi = n - 1;
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo + 1) >> 1);
        if (off[mid] <= e) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Rows of the edges [E0, E1) into s (all threads of the block; s is ready
// when it returns, and may be filled again after a barrier).  The tile's first
// and last row are found by two binary searches side by side, so the rows
// between them -- millions of empty ones between two communities of a
// coarsened graph with isolated vertices -- are read without a barrier per 256
// of them (R-MAT-21's levels of 853,000 mostly isolated vertices: expansion
// 1.57 ms with the barriers).
__device__ __forceinline__ void tile_rows(const uint32_t *off, uint32_t n, uint64_t E0, uint64_t E1, TileRows &s) {
    const uint32_t t = threadIdx.x;
    if (t == 0) s.r0 = last_row_at(off, n, E0);
    if (t == 32) s.r1 = last_row_at(off, n, E1 - 1);
    for (uint32_t q = t; q < kExpandTile + kExpandTile / 32; q += kExpandThreads) s.rowat[q] = 0;
    __syncthreads();
    const uint32_t r0 = s.r0, r1 = s.r1;
    if (t == 0) s.rowat[0] = r0;
#pragma unroll 4
    for (uint64_t j = (uint64_t)r0 + 1 + t; j <= r1; j += kExpandThreads) {
        const uint32_t st = off[j];
        if (st < off[j + 1]) {  // (one non-empty row per position: no conflict)
            const uint32_t q = (uint32_t)(st - E0);
            s.rowat[q + (q >> 5)] = (uint32_t)j;
        }
    }
    __syncthreads();
    // prefix maximum: 16 positions per thread, then across the threads
    uint32_t run = 0;
#pragma unroll
    for (int k = 0; k < kExpandPer; k++) {
        const uint32_t q = t * kExpandPer + k;
        run = max(run, s.rowat[q + (q >> 5)]);
        s.rowat[q + (q >> 5)] = run;
    }
    s.part[t] = run;
    __syncthreads();
    if (t < 32) {
        // exclusive prefix maximum of the 256 thread maxima: 8 per lane
        constexpr int L = kExpandThreads / 32;
        uint32_t loc[L], v = 0;
#pragma unroll
        for (int k = 0; k < L; k++) {
            v = max(v, s.part[t * L + k]);
            loc[k] = v;
        }
        uint32_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if ((int)t >= o) inc = max(inc, y);
        }
        uint32_t ex = __shfl_up_sync(0xffffffffu, inc, 1);
        if (t == 0) ex = 0;
#pragma unroll
        for (int k = 0; k < L; k++) s.part[t * L + k] = k ? max(ex, loc[k - 1]) : ex;
    }
    __syncthreads();
    const uint32_t pre = s.part[t];
#pragma unroll
    for (int k = 0; k < kExpandPer; k++) {
        const uint32_t q = t * kExpandPer + k;
        s.rowat[q + (q >> 5)] = max(s.rowat[q + (q >> 5)], pre);
    }
    __syncthreads();
}

}  // namespace mg
