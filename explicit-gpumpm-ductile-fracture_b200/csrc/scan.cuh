// Device-wide exclusive prefix sums of the binning: page ranks and cell starts.
// Replaces the reference's recursive block scan and Thrust scans
// (cuda_kernal_tools.cu:15-203, Transformer_kernal.cu:142-207).
//
// One pass ("decoupled look-back", Merrill and Garland, "Single-pass Parallel
// Prefix Scan with Decoupled Look-back", 2016): a CTA takes the next tile from
// a ticket, sums it, and gets the sum of the tiles before it from their status
// words.  Tiles are taken in order, so every tile waited for is held by a CTA
// that already runs.  A batch, whose launches serve all its scenes, scans in
// three passes (tile sums, their scan, apply: the bodies at the end).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "launch.cuh"

namespace gmpm {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;

inline int64_t scan_tiles(int64_t n) { return (n + kScanTile - 1) / kScanTile; }

// Working words of the binning's three scans (page flags, grid flags, cell
// counts), one after the other: a status word per tile and the ticket.  The
// last word is set when a wait of any of them gave up.  They are zero between
// binnings (the last kernel of a binning clears them).
struct ScanScratch {
    uint32_t* words;
    int32_t count;
    int32_t grid, cells;  // first word of the second and the third scan
    int32_t* tile_sums;   // the batched scans' tile sums: one per tile of the longer of the key space and the cells, + 1
};
inline int64_t scan_scratch_words(int64_t key_space, int64_t ncell) {
    return 2 * (scan_tiles(key_space) + 1) + scan_tiles(ncell) + 1 + 1;
}
inline ScanScratch scan_scratch(uint32_t* words, int64_t key_space, int64_t ncell, int32_t* tile_sums = nullptr) {
    const int32_t k = (int32_t)scan_tiles(key_space) + 1;
    return ScanScratch{words, (int32_t)scan_scratch_words(key_space, ncell), k, 2 * k, tile_sums};
}

__device__ __forceinline__ int32_t block_exclusive_sum(int32_t x, int32_t* total) {
    __shared__ int32_t warp_sums[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int32_t w = (lane < kScanThreads / 32) ? warp_sums[lane] : 0;
        int32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        if (lane < kScanThreads / 32) warp_sums[lane] = wi - w;
        if (lane == kScanThreads / 32 - 1) *total = wi;
    }
    __syncthreads();
    const int32_t r = warp_sums[warp] + incl - x;
    __syncthreads();
    return r;
}

// Status word of a tile: its own sum, or the sum up to and with it; both bits:
// a wait gave up.  Sums stay below 2^28 (the particle limit).
enum : uint32_t { kScanSum = 1u << 30, kScanPrefix = 2u << 30, kScanBad = 3u << 30, kScanValue = (1u << 30) - 1 };
constexpr int kScanSpinLimit = 1 << 22;

// The CTA's next tile.
__device__ __forceinline__ int scan_take_tile(uint32_t* ticket) {
    __shared__ int s_tile;
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(ticket, 1u);
    __syncthreads();
    return s_tile;
}

// Sum of the tiles before `tile`, whose own sum is `total`; every thread of the
// CTA calls it.  `bad`: a wait gave up here or before (the sum is then 0).  A
// tile after a bad one may still get its sum (it read the bad tile's own sum
// and waited longer), so every bad tile reports, not only the last.
__device__ __forceinline__ int32_t scan_look_back(uint32_t* status, int tile, int32_t total, bool& bad) {
    __shared__ int32_t s_prefix;
    __shared__ int s_bad;
    volatile uint32_t* st = status;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int32_t prefix = 0;
        bool gave_up = false;
        if (tile > 0) {
            if (lane == 0) st[tile] = kScanSum | (uint32_t)total;
            for (int end = tile - 1;; end -= 32) {
                const int i = end - lane;
                uint32_t s = i >= 0 ? st[i] : kScanPrefix;
                for (int spin = 0; __any_sync(0xffffffffu, s == 0); ++spin) {
                    if (spin >= kScanSpinLimit) {
                        if (s == 0) s = kScanBad;
                        break;
                    }
                    if (s == 0) s = st[i];
                }
                const unsigned ends = __ballot_sync(0xffffffffu, (s & kScanPrefix) != 0);
                const int last = ends ? __ffs(ends) - 1 : 31;
                if (__any_sync(0xffffffffu, lane <= last && s >= kScanBad)) {
                    gave_up = true;
                    break;
                }
                prefix += (int32_t)__reduce_add_sync(0xffffffffu, lane <= last ? (s & kScanValue) : 0u);
                if (ends) break;
            }
        }
        if (lane == 0) {
            st[tile] = gave_up ? kScanBad : kScanPrefix | (uint32_t)(prefix + total);
            s_prefix = gave_up ? 0 : prefix;
            s_bad = gave_up;
        }
    }
    __syncthreads();
    bad = s_bad != 0;
    return s_prefix;
}

// ---- three-pass scan of a batch (vb: the CTA's tile within its scene's scan) ---

template <typename TIn>
__device__ __forceinline__ void scan_load(const TIn* in, int64_t n, int64_t base, int32_t v[kScanItems]) {
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const int64_t idx = base + q;
        v[q] = (idx < n) ? (int32_t)in[idx] : 0;
    }
}

// Entries scanned: all n, or with `live` (a device count of live blocks of 64
// entries, the active pages of a cell scan, whose capacity is larger) only the
// live entries.  The scan then writes the live entries and the one after them,
// which receives the total; the entries beyond are left as they are, and no
// reader looks past the live pages.
__device__ __forceinline__ int64_t scan_live_len(int64_t n, const int32_t* live) {
    return live ? min(n, (int64_t)max(*live, 0) * 64) : n;
}

template <typename TIn>
__device__ __forceinline__ void scan_reduce_body(VB vb, const TIn* __restrict__ in, int64_t n,
                                                 int32_t* __restrict__ tile_sums, const int32_t* live = nullptr) {
    const int64_t m = scan_live_len(n, live);
    if ((int64_t)vb.b * kScanTile >= m) {  // a tile past the live entries (whole CTA)
        if (threadIdx.x == 0) tile_sums[vb.b] = 0;
        return;
    }
    const int64_t base = (int64_t)vb.b * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    scan_load(in, m, base, v);
    int32_t s = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) s += v[q];
    __shared__ int32_t tot;
    block_exclusive_sum(s, &tot);
    if (threadIdx.x == 0) tile_sums[vb.b] = tot;
}

// Single CTA: exclusive scan of the tile sums in place, total to *total.
__device__ __forceinline__ void scan_tiles_body(int32_t* __restrict__ tile_sums, int64_t ntiles,
                                                int32_t* __restrict__ total) {
    __shared__ int32_t chunk_total;
    int32_t carry = 0;
    for (int64_t base = 0; base < ntiles; base += kScanTile) {
        const int64_t b = base + (int64_t)threadIdx.x * kScanItems;
        int32_t v[kScanItems];
        scan_load(tile_sums, ntiles, b, v);
        int32_t s = 0;
#pragma unroll
        for (int q = 0; q < kScanItems; ++q) s += v[q];
        int32_t run = block_exclusive_sum(s, &chunk_total) + carry;
#pragma unroll
        for (int q = 0; q < kScanItems; ++q) {
            if (b + q < ntiles) tile_sums[b + q] = run;
            run += v[q];
        }
        carry += chunk_total;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

template <typename TIn>
__device__ __forceinline__ void scan_apply_body(VB vb, const TIn* __restrict__ in, int64_t n,
                                                const int32_t* __restrict__ tile_offsets, int32_t* __restrict__ out,
                                                const int32_t* live = nullptr) {
    const int64_t m = scan_live_len(n, live);
    const int64_t w = min(n, m + 1);  // entries written: the live ones and the total after them
    if ((int64_t)vb.b * kScanTile >= w) return;  // whole CTA
    const int64_t base = (int64_t)vb.b * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    scan_load(in, m, base, v);
    int32_t s = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) s += v[q];
    __shared__ int32_t tot;
    int32_t run = block_exclusive_sum(s, &tot) + tile_offsets[vb.b];
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        if (base + q < w) out[base + q] = run;
        run += v[q];
    }
}

}  // namespace gmpm
