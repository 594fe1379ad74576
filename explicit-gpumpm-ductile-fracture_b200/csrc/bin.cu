// Particle binning by SPGrid page/cell key, replacing the reference's hash +
// counting sort (Particles::sort_by_offsets, Particle_kernal.cu:158-249,484-542)
// and DomainTransformer::rebuild (Transformer_kernal.cu:15-209).
//
// Instead of an open-addressing page hash with unbounded probes and host
// syncs, pages are marked in a dense page-key table (the key space of the
// scene's grid), ranked by an exclusive scan (ascending page key = canonical
// page ids), and the +x/+y/+z neighbour pages are found by the same table.
// Particles are counting-sorted by (page rank, cell); the in-cell order is
// then made canonical (ascending previous slot), so the result equals a
// stable sort by (key, previous slot) bit for bit.  No host synchronisation.
#include <algorithm>
#include <cstdint>

#include "kernels.h"
#include "scan.cuh"

namespace gmpm {

// Particles per thread of the streaming binning kernels: each thread takes
// kBinILP particles one CTA width apart (coalesced per round) and issues all
// their loads before using any, so more requests are in flight per SM.
constexpr int kBinThreads = 256;
constexpr int kBinILP = 8;
// Scenes that would leave SMs without a CTA take two particles per thread: the
// scatter's chain of loads and atomics is then latency, not throughput (131k
// particles: histogram and scatter 5 and 10 us at eight per thread).
constexpr int kBinSmallILP = 2;
constexpr int64_t kBinSmall = (int64_t)2 * 148 * kBinThreads * kBinILP;
__host__ __device__ inline int bin_ilp(int64_t n) { return n < kBinSmall ? kBinSmallILP : kBinILP; }

// The kernels' bodies take the CTA's index within its scene's share of the
// launch (VB, common.cuh); the __global__ wrappers below each body serve a
// one-scene launch, the batched launches at the end of this file many scenes.

// The key pass: cell keys and page flags of positions that no G2P wrote
// (creation, restore, rebin).  A substep's binning starts from the keys its
// previous G2P formed for the positions it wrote.
template <typename R>
__device__ __forceinline__ void bin_keys_body(VB vb, int64_t n, const R* __restrict__ x0, const R* __restrict__ x1,
                                              const R* __restrict__ x2, const SceneDev<R>* __restrict__ sc,
                                              uint32_t* __restrict__ keys, uint8_t* __restrict__ page_flag,
                                              Counters* cnt) {
    const int64_t i0 = (int64_t)vb.b * kBinThreads * kBinILP + threadIdx.x;
    const double inv_dx = sc->inv_dx_d;
    const int res[3] = {sc->res[0], sc->res[1], sc->res[2]};
    R xs[kBinILP][3];
#pragma unroll
    for (int u = 0; u < kBinILP; ++u) {
        const int64_t i = i0 + (int64_t)u * kBinThreads;
        if (i < n) {
            xs[u][0] = x0[i];
            xs[u][1] = x1[i];
            xs[u][2] = x2[i];
        }
    }
    bool bad = false;
#pragma unroll
    for (int u = 0; u < kBinILP; ++u) {
        const int64_t i = i0 + (int64_t)u * kBinThreads;
        if (i >= n) continue;
        const uint32_t key = cell_key(xs[u], inv_dx, res, bad);
        keys[i] = key;
        page_flag[key >> 6] = 1;
    }
    if (bad) raise_flag(cnt, GMPM_FLAG_OUT_OF_DOMAIN);
}

template <typename R>
__global__ void __launch_bounds__(kBinThreads) k_bin_keys(int64_t n, const R* __restrict__ x0,
                                                          const R* __restrict__ x1, const R* __restrict__ x2,
                                                          const SceneDev<R>* __restrict__ sc,
                                                          uint32_t* __restrict__ keys,
                                                          uint8_t* __restrict__ page_flag, Counters* cnt) {
    bin_keys_body<R>(own_blocks(), n, x0, x1, x2, sc, keys, page_flag, cnt);
}

// A wait of a scan gave up: ranks, counts or starts are not to be used.  The
// rest of the binning then does nothing but restore its working words, and
// without pages the substep's other kernels do nothing.
__device__ __forceinline__ void scan_gave_up(uint32_t* failed, Counters* cnt) {
    *failed = 1u;
    raise_flag(cnt, GMPM_FLAG_COPY_TIMEOUT);
}
// The page scan found pages and no wait gave up (n >= 1, so there are pages).
__device__ __forceinline__ bool scans_done(const ScanScratch& scan, const Counters* cnt) {
    return (scan.words[scan.count - 1] == 0u) & (cnt->n_blocks > 0);  // both loads at once
}

// Ranks of the flagged keys in ascending order, with their list and count:
// page ids (the first scan) or grid page ids (the second).  The first also
// marks every active page and its 7 "+" neighbours as grid pages
// (supplementAdjacentPages, Transformer_kernal.cu:70-96).  words: the scan's
// status words and, after them, its ticket.  Ranks of keys without a flag are
// left as they are; no reader looks at them.  failed: set where a wait gave up.
__device__ __forceinline__ void page_scan_body(uint32_t key_space, const uint8_t* flag,
                                               int32_t* rank, uint32_t* list, int cap,
                                               int32_t* total, uint8_t* grid_flag,
                                               uint32_t* words, uint32_t* failed, Counters* cnt) {
    const int ntiles = (int)((key_space + kScanTile - 1) / kScanTile);
    const int tile = scan_take_tile(words + ntiles);
    if (tile >= ntiles) return;
    static_assert(kScanItems == 16, "one 16-byte load per thread");
    const uint32_t k0 = (uint32_t)tile * kScanTile + threadIdx.x * kScanItems;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (k0 < key_space) v = *reinterpret_cast<const uint4*>(flag + k0);  // the key space is a multiple of 64
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t bits = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) bits |= ((w[q] | w[q] >> 7 | w[q] >> 14 | w[q] >> 21) & 15u) << (4 * q);
    __shared__ int32_t tot;
    int32_t run = block_exclusive_sum(__popc(bits), &tot);
    bool bad;
    const int32_t before = scan_look_back(words, tile, tot, bad);
    run += before;
    bool over = false;
    while (bits) {
        const uint32_t k = k0 + (uint32_t)__ffs((int)bits) - 1;
        bits &= bits - 1;
        rank[k] = run;
        if (run < cap)
            list[run] = k;
        else
            over = true;
        ++run;
        if (grid_flag) {
            // the next coordinate along an axis is an increment of the key's interleaved bits of that axis
            // (decoding the key and interleaving eight took most of the scan's time)
            constexpr uint32_t kAxis[3] = {0x24924924u, 0x12492492u, 0x09249249u};
            uint32_t c[3][2];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                c[a][0] = k & kAxis[a];
                c[a][1] = ((k | ~kAxis[a]) + 1) & kAxis[a];
            }
#pragma unroll
            for (int d = 0; d < 8; ++d) grid_flag[c[0][d >> 2] | c[1][(d >> 1) & 1] | c[2][d & 1]] = 1;
        }
    }
    if (over) raise_flag(cnt, GMPM_FLAG_TABLE_OVERFLOW);
    if (threadIdx.x == 0) {
        if (tile == ntiles - 1) *total = before + tot;
        if (bad) scan_gave_up(failed, cnt);
    }
}

__global__ void __launch_bounds__(kScanThreads)
    k_page_scan(uint32_t key_space, const uint8_t* flag, int32_t* rank,
                uint32_t* list, int cap, int32_t* total, uint8_t* grid_flag,
                uint32_t* words, uint32_t* failed, Counters* cnt) {
    depend_on_previous();
    page_scan_body(key_space, flag, rank, list, cap, total, grid_flag, words, failed, cnt);
}

// Zero `bytes` (a multiple of 16, from a 16-byte boundary) in 4 KiB pieces: pieces vb.b, vb.b + vb.g, ...
__device__ __forceinline__ void zero_bytes_body(VB vb, void* p, int64_t bytes) {
    char* c = static_cast<char*>(p);
    for (int64_t off = (int64_t)vb.b * 4096 + (int64_t)threadIdx.x * 16; off < bytes; off += (int64_t)vb.g * 4096)
        *reinterpret_cast<uint4*>(c + off) = make_uint4(0u, 0u, 0u, 0u);
}

// Cell starts of the active pages (live cells; the capacity is larger) and the
// total after them.  The starts also replace the counts, as the scatter's fill
// pointers.  clear: flags whose last use in the binning was the page links,
// cleared here for the next one (or null).
__device__ __forceinline__ void cell_scan_body(VB vb, int64_t ncell, int32_t* count,
                                               int32_t* start, const ScanScratch& scan,
                                               uint8_t* clear0, uint8_t* clear1, uint32_t key_space, Counters* cnt) {
    if (clear0) zero_bytes_body(vb, clear0, key_space);
    if (clear1) zero_bytes_body(vb, clear1, key_space);
    uint32_t* words = scan.words + scan.cells;
    // read once per CTA (a peer that gives up may set the failure word meanwhile), beside thread 0's ticket
    __shared__ int64_t live;
    if (threadIdx.x == 32) live = scans_done(scan, cnt) ? min(ncell, (int64_t)cnt->n_blocks * 64) : 0;
    const int tile = scan_take_tile(words + (ncell + kScanTile - 1) / kScanTile);  // with a barrier
    const int64_t m = live;
    const int64_t base = (int64_t)tile * kScanTile + (int64_t)threadIdx.x * kScanItems;
    if ((int64_t)tile * kScanTile >= max(m, (int64_t)1)) return;  // whole CTA; tile 0 writes the total of no cells
    int4 v[kScanItems / 4];
    int32_t s = 0;
#pragma unroll
    for (int q = 0; q < kScanItems / 4; ++q) {
        // live cells come in pages of 64
        v[q] = base + 4 * q < m ? *reinterpret_cast<const int4*>(count + base + 4 * q) : make_int4(0, 0, 0, 0);
        s += v[q].x + v[q].y + v[q].z + v[q].w;
    }
    __shared__ int32_t tot;
    int32_t run = block_exclusive_sum(s, &tot);
    bool bad;
    const int32_t before = scan_look_back(words, tile, tot, bad);
    run += before;
#pragma unroll
    for (int q = 0; q < kScanItems / 4; ++q) {
        const int4 o = make_int4(run, run + v[q].x, run + v[q].x + v[q].y, run + v[q].x + v[q].y + v[q].z);
        if (base + 4 * q < m) {
            *reinterpret_cast<int4*>(start + base + 4 * q) = o;
            *reinterpret_cast<int4*>(count + base + 4 * q) = o;
        }
        run = o.w + v[q].w;
    }
    if (threadIdx.x == 0) {
        if (m <= (int64_t)(tile + 1) * kScanTile) start[m] = before + tot;  // the tile of the last live cell
        if (bad) scan_gave_up(scan.words + scan.count - 1, cnt);
    }
}

__global__ void __launch_bounds__(kScanThreads)
    k_cell_scan(int64_t ncell, int32_t* count, int32_t* start, ScanScratch scan,
                uint8_t* clear0, uint8_t* clear1, uint32_t key_space, Counters* cnt) {
    depend_on_previous();
    cell_scan_body(own_blocks(), ncell, count, start, scan, clear0, clear1, key_space, cnt);
}

// Page topology: adj (establishPageTopology, Transformer_kernal.cu:98-114) and
// its inverse grid_src used by the fixed-order grid gather.
__device__ __forceinline__ void page_links_body(VB vb, const BinDev& bin, const Counters* cnt) {
    const int nb = min(cnt->n_blocks, bin.nb_cap);
    const int ng = min(cnt->n_grid_blocks, bin.ng_cap);
    const int t = vb.b * blockDim.x + threadIdx.x;
    const int slot = t & 7;
    const int idx = t >> 3;
    const int di = slot >> 2, dj = (slot >> 1) & 1, dk = slot & 1;
    if (idx < nb) {
        int bx, by, bz;
        page_coords(bin.block_keys[idx], bx, by, bz);
        const int r = bin.grid_rank[page_key(bx + di, by + dj, bz + dk)];
        bin.adj[idx * 8 + slot] = (r < bin.ng_cap) ? r : -1;  // overflow is flagged by the page scan
    }
    if (idx < ng) {
        int gx, gy, gz;
        page_coords(bin.grid_keys[idx], gx, gy, gz);
        int src = -1;
        if (gx - di >= 0 && gy - dj >= 0 && gz - dk >= 0) {
            const uint32_t k = page_key(gx - di, gy - dj, gz - dk);
            if (k < bin.key_space && bin.page_flag[k]) {
                const int r = bin.page_rank[k];
                src = (r < bin.nb_cap) ? r : -1;
            }
        }
        bin.grid_src[idx * 8 + slot] = src;
    }
}

// Histogram of (page rank, cell) buckets with warp-aggregated atomics.  done: the ranks are there (if not, nothing is
// counted); used late, so that its loads travel beside the keys'.
template <int kILP>
__device__ __forceinline__ void bin_hist_body(VB vb, int64_t n, const uint32_t* keys,
                                              const int32_t* page_rank, int32_t* cell_count,
                                              int nb_cap, bool done) {
    const int64_t i0 = (int64_t)vb.b * kBinThreads * kILP + threadIdx.x;
    uint32_t key[kILP];
    int rank[kILP];
#pragma unroll
    for (int u = 0; u < kILP; ++u) key[u] = i0 + (int64_t)u * kBinThreads < n ? keys[i0 + (int64_t)u * kBinThreads] : 0u;
#pragma unroll
    for (int u = 0; u < kILP; ++u)
        rank[u] = i0 + (int64_t)u * kBinThreads < n ? page_rank[key[u] >> 6] : nb_cap;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int u = 0; u < kILP; ++u) {
        const int bucket = done && rank[u] < nb_cap ? rank[u] * 64 + (int)(key[u] & 63) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, bucket);
        if (bucket >= 0 && lane == __ffs(peers) - 1) atomicAdd(&cell_count[bucket], __popc(peers));
    }
}

__host__ __device__ inline int bin_ctas(int64_t n, int ilp) {
    const int64_t c = (n + (int64_t)kBinThreads * ilp - 1) / ((int64_t)kBinThreads * ilp);
    return c < 1 ? 1 : (int)c;
}

// The histogram's CTAs and, after them, the page links' (both need the ranks only).
template <int kILP>
__global__ void __launch_bounds__(kBinThreads) k_bin_hist_links(BinDev bin, ScanScratch scan, const Counters* cnt) {
    depend_on_previous();
    const bool done = scans_done(scan, cnt);
    const VB vb = own_blocks();
    const int hist = bin_ctas(bin.n, kILP);
    if (vb.b < hist)
        bin_hist_body<kILP>(vb, bin.n, bin.keys, bin.page_rank, bin.cell_count, bin.nb_cap, done);
    else if (done)
        page_links_body(VB{vb.b - hist, vb.g - hist}, bin, cnt);
}

// Scatter slots; lanes of one warp with the same bucket keep their order.  fill: the cells' fill pointers, or
// (kOffsets) fill counts beside the cells' starts.
template <int kILP, bool kOffsets>
__device__ __forceinline__ void bin_scatter_body(VB vb, int64_t n, const uint32_t* keys,
                                                 const int32_t* page_rank,
                                                 const int32_t* cell_start, int32_t* fill,
                                                 int32_t* perm, uint32_t* keys_sorted,
                                                 int nb_cap, bool done) {
    const int64_t i0 = (int64_t)vb.b * kBinThreads * kILP + threadIdx.x;
    uint32_t key[kILP];
    int bucket[kILP], start[kILP];
#pragma unroll
    for (int u = 0; u < kILP; ++u) key[u] = i0 + (int64_t)u * kBinThreads < n ? keys[i0 + (int64_t)u * kBinThreads] : 0u;
#pragma unroll
    for (int u = 0; u < kILP; ++u) {
        const int r = i0 + (int64_t)u * kBinThreads < n ? page_rank[key[u] >> 6] : nb_cap;
        bucket[u] = done && r < nb_cap ? r * 64 + (int)(key[u] & 63) : -1;
    }
#pragma unroll
    for (int u = 0; u < kILP; ++u) start[u] = kOffsets && bucket[u] >= 0 ? cell_start[bucket[u]] : 0;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int u = 0; u < kILP; ++u) {
        const unsigned peers = __match_any_sync(0xffffffffu, bucket[u]);
        const int leader = __ffs(peers) - 1;
        int base = 0;
        if (bucket[u] >= 0 && lane == leader) base = atomicAdd(&fill[bucket[u]], __popc(peers));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (bucket[u] >= 0) {
            const int slot = start[u] + base + __popc(peers & ((1u << lane) - 1u));
            perm[slot] = (int32_t)(i0 + (int64_t)u * kBinThreads);
            keys_sorted[slot] = key[u];
        }
    }
}

template <int kILP>
__global__ void __launch_bounds__(kBinThreads) k_bin_scatter(BinDev bin, ScanScratch scan, Counters* cnt) {
    depend_on_previous();
    const bool done = scans_done(scan, cnt);  // if not, the counts are no fill pointers: nothing is scattered
    bin_scatter_body<kILP, false>(own_blocks(), bin.n, bin.keys, bin.page_rank, nullptr, bin.cell_count, bin.perm,
                                  bin.keys_sorted, bin.nb_cap, done);
    if (!done && blockIdx.x == 0 && threadIdx.x == 0) cnt->n_blocks = cnt->n_grid_blocks = 0;  // for the kernels after
}

// Canonical in-cell order: ascending previous slot.  Each warp takes one page
// (up to 8 pages per CTA in flight, so the page's few dependent global round
// trips overlap across pages) and ranks every slot within its cell in shared memory
// (cells hold few particles).  A page above the warp's buffer is left to the
// whole CTA, which ranks it in windows of whole cells after the warps'
// pages; a single cell above the CTA buffer (thousands of particles in one
// cell, which only a failed state with clamped positions produces) keeps its
// scatter order and raises GMPM_FLAG_TABLE_OVERFLOW instead of being ranked
// in quadratic time.
constexpr int kCanonWarps = 8;
constexpr int kCanonWarpBuf = 768;
constexpr int kCanonBuf = kCanonWarps * kCanonWarpBuf;

// Rank slots [lo, hi) of a page (whole cells) by previous slot within their
// cells; buf holds perm[lo, hi).  Threads tid, tid + step, ... of the caller.
__device__ __forceinline__ void canon_rank(const BinDev& bin, const int32_t* cs, const int32_t* buf, int lo, int hi,
                                           int tid, int step) {
    for (int s = lo + tid; s < hi; s += step) {
        const int cell = (int)(bin.keys_sorted[s] & 63);
        const int a = cs[cell] - lo, e = cs[cell + 1] - lo;
        const int32_t v = buf[s - lo];
        int r = 0;
        for (int u = a; u < e; ++u) r += buf[u] < v;
        bin.perm[lo + a + r] = v;
    }
}

// The cell of slot s (cs: the page's 65 cell starts).
__device__ __forceinline__ int cell_of_slot(const int32_t* cs, int s) {
    int c = 0;  // the last cell that starts at or before s and is not empty there
#pragma unroll
    for (int step = 32; step > 0; step >>= 1)
        if (cs[c + step] <= s) c += step;
    return c;
}

// Warp path: the scatter keeps the order of the lanes of one warp, so most
// cells already ascend by previous slot; an ascending cell is its own canonical
// order.  desc: a bit per slot that descends from the one before, less the
// first slots of cells.  Only where one is left are the cells looked up and
// the descending ones ranked: a few of them one after the other, a lane per
// particle, many (positions in no order) a lane per slot of the page (1M
// shuffled positions: 164 us of binning against 177; sorted ones, 8.4M
// particles: 150 against 140).
constexpr int kCanonFewCells = 24;
__device__ __forceinline__ void canon_rank_warp(const BinDev& bin, const int32_t* cs, const int32_t* buf,
                                                uint32_t* desc, uint8_t* bad, int lo, int hi, int lane) {
    const int n = hi - lo, words = (n + 31) >> 5;
    for (int w = 0; w < words; ++w) {
        const int s = 32 * w + lane;
        const unsigned d = __ballot_sync(0xffffffffu, s > 0 && s < n && buf[s - 1] > buf[s]);
        if (lane == 0) desc[w] = d;
    }
    __syncwarp();
    for (int c = lane; c < 64; c += 32) {
        const int s = cs[c] - lo;
        if (s < n) atomicAnd(&desc[s >> 5], ~(1u << (s & 31)));
        bad[c] = 0;
    }
    __syncwarp();
    const uint32_t mine = lane < words ? desc[lane] : 0u;
    if (!__any_sync(0xffffffffu, mine != 0u)) return;
    for (uint32_t d = mine; d; d &= d - 1) bad[cell_of_slot(cs, lo + 32 * lane + __ffs((int)d) - 1)] = 1;
    __syncwarp();
    const unsigned b0 = __ballot_sync(0xffffffffu, bad[lane] != 0), b1 = __ballot_sync(0xffffffffu, bad[32 + lane] != 0);
    if (__popc(b0) + __popc(b1) > kCanonFewCells) {
        for (int s = lo + lane; s < hi; s += 32) {
            const int cell = cell_of_slot(cs, s);
            if (!bad[cell]) continue;
            const int a = cs[cell] - lo, e = cs[cell + 1] - lo;
            const int32_t v = buf[s - lo];
            int r = 0;
            for (int u = a; u < e; ++u) r += buf[u] < v;
            bin.perm[lo + a + r] = v;
        }
        return;
    }
#pragma unroll
    for (int h = 0; h < 64; h += 32)
        for (unsigned cells = h ? b1 : b0; cells; cells &= cells - 1) {
            const int cell = h + __ffs((int)cells) - 1;
            const int a = cs[cell] - lo, e = cs[cell + 1] - lo;
            for (int s = a + lane; s < e; s += 32) {
                const int32_t v = buf[s];
                int r = 0;
                for (int u = a; u < e; ++u) r += buf[u] < v;
                bin.perm[lo + a + r] = v;
            }
        }
}

// Also clears, for the next binning, the fill pointers of the pages' cells
// (without pages, after a scan that gave up, those of every cell: the
// histogram may have run) and the scans' words.
__device__ __forceinline__ void bin_canon_body(VB vb, const BinDev& bin, const ScanScratch& scan, Counters* cnt) {
    __shared__ int32_t buf[kCanonBuf];
    __shared__ int32_t cs[kCanonWarps][68];
    __shared__ uint8_t bad[kCanonWarps][64];
    __shared__ uint32_t desc[kCanonWarps][kCanonWarpBuf / 32];
    static_assert(kCanonWarpBuf / 32 <= 32, "one word of slots per lane");
    __shared__ int big[kCanonWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nb = min(cnt->n_blocks, bin.nb_cap);
    int32_t* wbuf = buf + warp * kCanonWarpBuf;
    if (vb.b == 0)
        for (int q = threadIdx.x; q < scan.count; q += blockDim.x) scan.words[q] = 0u;
    if (nb <= 0) zero_bytes_body(vb, bin.cell_count, (int64_t)bin.nb_cap * 64 * 4);
    for (int g = vb.b; g < nb; g += vb.g * kCanonWarps) {
        const int b = g + warp * vb.g;
        int is_big = 0;
        if (b < nb) {
            for (int q = lane; q < 65; q += 32) cs[warp][q] = bin.cell_start[(int64_t)b * 64 + q];
            for (int q = lane; q < 64; q += 32) bin.cell_count[(int64_t)b * 64 + q] = 0;
            __syncwarp();
            const int lo = cs[warp][0], hi = cs[warp][64];
            if (hi - lo <= kCanonWarpBuf) {
                // eight loads in flight per lane: one at a time, a page was a chain of 12 round trips
                for (int s0 = lo + lane; s0 < hi; s0 += 32 * 8) {
                    int32_t v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u] = s0 + 32 * u < hi ? bin.perm[s0 + 32 * u] : 0;
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (s0 + 32 * u < hi) wbuf[s0 + 32 * u - lo] = v[u];
                }
                __syncwarp();
                canon_rank_warp(bin, cs[warp], wbuf, desc[warp], bad[warp], lo, hi, lane);
            } else {
                is_big = 1;
            }
        }
        if (lane == 0) big[warp] = is_big;
        __syncthreads();
        // pages above a warp's buffer: the whole CTA, one at a time
        for (int w = 0; w < kCanonWarps; ++w) {
            if (!big[w]) continue;
            const int32_t* pcs = cs[w];
            int c0 = 0;
            while (c0 < 64) {
                int c1 = c0;
                while (c1 < 64 && pcs[c1 + 1] - pcs[c0] <= kCanonBuf) ++c1;
                if (c1 == c0) {
                    if (threadIdx.x == 0) raise_flag(cnt, GMPM_FLAG_TABLE_OVERFLOW);
                    c0 = c0 + 1;
                    continue;
                }
                const int lo = pcs[c0], hi = pcs[c1];
                for (int s = lo + (int)threadIdx.x; s < hi; s += blockDim.x) buf[s - lo] = bin.perm[s];
                __syncthreads();
                canon_rank(bin, pcs, buf, lo, hi, threadIdx.x, blockDim.x);
                __syncthreads();
                c0 = c1;
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(32 * kCanonWarps) k_bin_canon(BinDev bin, ScanScratch scan, Counters* cnt) {
    depend_on_previous();
    bin_canon_body(own_blocks(), bin, scan, cnt);
}

// About a CTA for each live page (the capacity is twice their number at creation), as far as they are resident at once,
// and pages dealt out one per CTA before a second: pages above a warp's buffer take a whole CTA each.  (Eight neighbouring
// pages per CTA left the work of dense scenes to a few CTAs, which a dependent launch also packs onto few SMs: binning of
// 1M particles, 27 per cell 197 -> 56 us, 64 per cell 453 -> 100; 8 per cell 51 -> 46.)
static int canon_ctas(int nb_cap, int sms) { return std::max(1, std::min((nb_cap + 1) / 2, sms * 8)); }

// ---------------------------------------------------------------------------

static int links_ctas(const BinDev& bin) { return (int)(((int64_t)std::max(bin.nb_cap, bin.ng_cap) * 8 + 255) / 256); }

static cudaError_t launch_page_scan(const BinDev& bin, const ScanScratch& scan, Counters* cnt, bool mark, cudaStream_t s) {
    return launch_dependent(k_page_scan, dim3((unsigned)scan_tiles(bin.key_space)), dim3(kScanThreads), 0, s, bin.key_space,
                         (const uint8_t*)bin.page_flag, bin.page_rank, bin.block_keys, (int)bin.nb_cap, &cnt->n_blocks,
                         mark ? bin.grid_flag : nullptr, scan.words, scan.words + scan.count - 1, cnt);
}
static cudaError_t launch_grid_scan(const BinDev& bin, const ScanScratch& scan, Counters* cnt, cudaStream_t s) {
    return launch_dependent(k_page_scan, dim3((unsigned)scan_tiles(bin.key_space)), dim3(kScanThreads), 0, s, bin.key_space,
                         (const uint8_t*)bin.grid_flag, bin.grid_rank, bin.grid_keys, (int)bin.ng_cap,
                         &cnt->n_grid_blocks, (uint8_t*)nullptr, scan.words + scan.grid, scan.words + scan.count - 1, cnt);
}

cudaError_t launch_page_scans(BinDev bin, ScanScratch scan, Counters* cnt, cudaStream_t s) {
    const cudaError_t e = launch_page_scan(bin, scan, cnt, true, s);
    return e == cudaSuccess ? launch_grid_scan(bin, scan, cnt, s) : e;
}

// Histogram (with the page links where the binning has grid pages), cell scan, scatter, canonical order.
static cudaError_t launch_bin_sort(const BinDev& bin, const ScanScratch& scan, Counters* cnt, int num_sms, bool clear_pages,
                                   cudaStream_t s) {
    const int64_t ncell = (int64_t)bin.nb_cap * 64;
    const int ilp = bin_ilp(bin.n), ctas = bin_ctas(bin.n, ilp);
    const unsigned hist = (unsigned)(ctas + (bin.grid_flag ? links_ctas(bin) : 0));
    cudaError_t e = launch_dependent(ilp == kBinILP ? k_bin_hist_links<kBinILP> : k_bin_hist_links<kBinSmallILP>, dim3(hist), dim3(kBinThreads), 0, s, bin, scan, (const Counters*)cnt);
    if (e == cudaSuccess)
        e = launch_dependent(k_cell_scan, dim3((unsigned)scan_tiles(ncell)), dim3(kScanThreads), 0, s, ncell, bin.cell_count,
                          bin.cell_start, scan, clear_pages ? bin.page_flag : nullptr, bin.grid_flag,
                          bin.key_space, cnt);
    if (e == cudaSuccess)
        e = launch_dependent(ilp == kBinILP ? k_bin_scatter<kBinILP> : k_bin_scatter<kBinSmallILP>, dim3((unsigned)ctas), dim3(kBinThreads), 0, s, bin, scan, cnt);
    if (e == cudaSuccess)
        e = launch_dependent(k_bin_canon, dim3((unsigned)canon_ctas(bin.nb_cap, num_sms)), dim3(32 * kCanonWarps), 0, s, bin,
                          scan, cnt);
    return e;
}

cudaError_t launch_bin_no_grid(BinDev bin, ScanScratch scan, Counters* cnt, int num_sms, cudaStream_t s) {
    const cudaError_t e = launch_page_scan(bin, scan, cnt, false, s);
    return e == cudaSuccess ? launch_bin_sort(bin, scan, cnt, num_sms, true, s) : e;
}

template <typename R>
cudaError_t launch_binning(const SceneDev<R>* sc, const PState<R>& st, BinDev bin, ScanScratch scan, Counters* cnt,
                           int num_sms, cudaStream_t stream, bool keys_ready, bool reset) {
    if (reset) {
        cudaMemsetAsync(bin.grid_flag, 0, bin.key_space, stream);
        cudaMemsetAsync(bin.cell_count, 0, (size_t)bin.nb_cap * 64 * sizeof(int32_t), stream);
        cudaMemsetAsync(scan.words, 0, (size_t)scan.count * sizeof(uint32_t), stream);
    }
    if (!keys_ready) {
        cudaMemsetAsync(bin.page_flag, 0, bin.key_space, stream);
        k_bin_keys<R><<<bin_ctas(bin.n, kBinILP), kBinThreads, 0, stream>>>(bin.n, st.x[0], st.x[1], st.x[2], sc, bin.keys,
                                                                   bin.page_flag, cnt);
    }
    cudaError_t e = launch_page_scans(bin, scan, cnt, stream);
    // with keys_ready the page flags are cleared after their last use, for the G2P that keys the next positions
    if (e == cudaSuccess) e = launch_bin_sort(bin, scan, cnt, num_sms, keys_ready, stream);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

template <typename R>
cudaError_t launch_keys(const SceneDev<R>* sc, const PState<R>& st, BinDev bin, Counters* cnt, cudaStream_t s) {
    k_bin_keys<R><<<bin_ctas(bin.n, kBinILP), kBinThreads, 0, s>>>(bin.n, st.x[0], st.x[1], st.x[2], sc, bin.keys,
                                                                 bin.page_flag, cnt);
    return cudaGetLastError();
}
template cudaError_t launch_keys<float>(const SceneDev<float>*, const PState<float>&, BinDev, Counters*,
                                        cudaStream_t);
template cudaError_t launch_keys<double>(const SceneDev<double>*, const PState<double>&, BinDev, Counters*,
                                         cudaStream_t);

// ---- batched binning over many scenes ------------------------------------------

void batch_scene_ctas(int64_t n, uint32_t key_space, int nb_cap, int ng_cap, int sms, int real_bytes,
                      int ctas[kBatchMaps]) {
    auto cdiv = [](int64_t a, int64_t b) { return (int)std::max<int64_t>(1, (a + b - 1) / b); };
    const int64_t ncell = (int64_t)nb_cap * 64;
    ctas[BM_ZERO_FLAGS] = cdiv(key_space, 4096);
    ctas[BM_PARTICLES] = bin_ctas(n, kBinILP);
    ctas[BM_KEYSPACE] = cdiv(key_space, 256);
    ctas[BM_KEY_TILES] = (int)scan_tiles(key_space);
    ctas[BM_LINKS] = cdiv((int64_t)std::max(nb_cap, ng_cap) * 8, 256);
    ctas[BM_ZERO_CELLS] = cdiv(ncell * 4, 4096);
    ctas[BM_CELL_TILES] = (int)scan_tiles(ncell);
    // a page for each warp of the live half of the capacity: beside many scenes, CTAs of few pages cost more than they
    // give (64 bars: 67 us with twice as many, 44 with these)
    ctas[BM_CANON] = std::min(cdiv(nb_cap, 2 * kCanonWarps), sms * 8);
    ctas[BM_P2G] = real_bytes == 4 ? p2g_ctas<float>(nb_cap, sms) : p2g_ctas<double>(nb_cap, sms);
    ctas[BM_GRID] = std::max(1, std::min(ng_cap / 4 + 1, sms * 8));
    const int per_sm = real_bytes == 4 ? 2 : 1;  // G2P's resident CTAs per SM
    ctas[BM_G2P] = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)sms * per_sm));
    ctas[BM_ONE] = 1;
}

// Mark every active page and its 7 "+" neighbours as grid pages
// (supplementAdjacentPages, Transformer_kernal.cu:70-96).
__device__ __forceinline__ void mark_grid_body(VB vb, uint32_t key_space, const uint8_t* __restrict__ page_flag,
                                               uint8_t* __restrict__ grid_flag) {
    const uint32_t k = vb.b * blockDim.x + threadIdx.x;
    if (k >= key_space || !page_flag[k]) return;
    int bx, by, bz;
    page_coords(k, bx, by, bz);
#pragma unroll
    for (int d = 0; d < 8; ++d) grid_flag[page_key(bx + (d >> 2), by + ((d >> 1) & 1), bz + (d & 1))] = 1;
}

// Compact flagged keys into ascending order.
__device__ __forceinline__ void compact_keys_body(VB vb, uint32_t key_space, const uint8_t* __restrict__ flag,
                                                  const int32_t* __restrict__ rank, uint32_t* __restrict__ out,
                                                  int cap, Counters* cnt) {
    const uint32_t k = vb.b * blockDim.x + threadIdx.x;
    if (k >= key_space || !flag[k]) return;
    const int r = rank[k];
    if (r < cap)
        out[r] = k;
    else
        raise_flag(cnt, GMPM_FLAG_TABLE_OVERFLOW);
}

// which: 1 grid flags; 2 cell counters; 3 cell counters and the flags (after
// their last use in the binning: the page flags for the G2P that sets them, the
// grid flags for a binning of the scene by itself, which expects them zero).
template <typename R>
__global__ void __launch_bounds__(256) k_batch_zero(const SceneArgs<R>* __restrict__ A, const int32_t* __restrict__ start,
                                                    int ns, int which) {
    VB vb;
    const BinDev& bin = A[scene_of_block(start, ns, vb)].bin;
    if (which != 2) zero_bytes_body(vb, bin.grid_flag, bin.key_space);
    if (which >= 2) zero_bytes_body(vb, bin.cell_count, (int64_t)bin.nb_cap * 64 * 4);
    if (which == 3) zero_bytes_body(vb, bin.page_flag, bin.key_space);
}

// The three scans of the binning: 0 page flags -> page ranks, 1 grid flags ->
// grid ranks, 2 cell counts -> cell starts.
template <int kWhich>
struct ScanSel;
template <>
struct ScanSel<0> {
    using T = uint8_t;
    static __device__ const T* in(const BinDev& b) { return b.page_flag; }
    static __device__ int64_t n(const BinDev& b) { return b.key_space; }
    static __device__ int32_t* out(const BinDev& b) { return b.page_rank; }
    static __device__ int32_t* total(const BinDev& b, Counters* c) { return &c->n_blocks; }
    static __device__ const int32_t* live(Counters*) { return nullptr; }
};
template <>
struct ScanSel<1> {
    using T = uint8_t;
    static __device__ const T* in(const BinDev& b) { return b.grid_flag; }
    static __device__ int64_t n(const BinDev& b) { return b.key_space; }
    static __device__ int32_t* out(const BinDev& b) { return b.grid_rank; }
    static __device__ int32_t* total(const BinDev& b, Counters* c) { return &c->n_grid_blocks; }
    static __device__ const int32_t* live(Counters*) { return nullptr; }
};
template <>
struct ScanSel<2> {
    using T = int32_t;
    static __device__ const T* in(const BinDev& b) { return b.cell_count; }
    static __device__ int64_t n(const BinDev& b) { return (int64_t)b.nb_cap * 64; }
    static __device__ int32_t* out(const BinDev& b) { return b.cell_start; }
    static __device__ int32_t* total(const BinDev& b, Counters*) { return b.cell_start + (int64_t)b.nb_cap * 64; }
    static __device__ const int32_t* live(Counters* c) { return &c->n_blocks; }  // the active pages' cells
};

template <typename R, int kWhich>
__global__ void __launch_bounds__(kScanThreads) k_batch_scan_reduce(const SceneArgs<R>* __restrict__ A,
                                                                    const int32_t* __restrict__ start, int ns) {
    VB vb;
    const SceneArgs<R>& a = A[scene_of_block(start, ns, vb)];
    using S = ScanSel<kWhich>;
    scan_reduce_body(vb, S::in(a.bin), S::n(a.bin), a.scan.tile_sums, S::live(a.cnt));
}

template <typename R, int kWhich>
__global__ void __launch_bounds__(kScanThreads) k_batch_scan_tiles(const SceneArgs<R>* __restrict__ A,
                                                                   const int32_t* __restrict__ start, int ns) {
    VB vb;
    const SceneArgs<R>& a = A[scene_of_block(start, ns, vb)];
    using S = ScanSel<kWhich>;
    const int64_t ntiles = (S::n(a.bin) + kScanTile - 1) / kScanTile;
    scan_tiles_body(a.scan.tile_sums, ntiles, S::total(a.bin, a.cnt));
}

template <typename R, int kWhich>
__global__ void __launch_bounds__(kScanThreads) k_batch_scan_apply(const SceneArgs<R>* __restrict__ A,
                                                                   const int32_t* __restrict__ start, int ns) {
    VB vb;
    const SceneArgs<R>& a = A[scene_of_block(start, ns, vb)];
    using S = ScanSel<kWhich>;
    scan_apply_body(vb, S::in(a.bin), S::n(a.bin), a.scan.tile_sums, S::out(a.bin), S::live(a.cnt));
}

template <typename R>
__global__ void __launch_bounds__(256) k_batch_mark(const SceneArgs<R>* __restrict__ A,
                                                    const int32_t* __restrict__ start, int ns) {
    VB vb;
    const BinDev& bin = A[scene_of_block(start, ns, vb)].bin;
    mark_grid_body(vb, bin.key_space, bin.page_flag, bin.grid_flag);
}

template <typename R>
__global__ void __launch_bounds__(256) k_batch_compact(const SceneArgs<R>* __restrict__ A,
                                                       const int32_t* __restrict__ start, int ns) {
    VB vb;
    const SceneArgs<R>& a = A[scene_of_block(start, ns, vb)];
    compact_keys_body(vb, a.bin.key_space, a.bin.page_flag, a.bin.page_rank, a.bin.block_keys, a.bin.nb_cap, a.cnt);
    compact_keys_body(vb, a.bin.key_space, a.bin.grid_flag, a.bin.grid_rank, a.bin.grid_keys, a.bin.ng_cap, a.cnt);
}

template <typename R>
__global__ void __launch_bounds__(256) k_batch_links(const SceneArgs<R>* __restrict__ A,
                                                     const int32_t* __restrict__ start, int ns) {
    VB vb;
    const SceneArgs<R>& a = A[scene_of_block(start, ns, vb)];
    page_links_body(vb, a.bin, a.cnt);
}

template <typename R>
__global__ void __launch_bounds__(kBinThreads) k_batch_hist(const SceneArgs<R>* __restrict__ A,
                                                            const int32_t* __restrict__ start, int ns) {
    VB vb;
    const SceneArgs<R>& a = A[scene_of_block(start, ns, vb)];
    const bool done = a.cnt->n_blocks > 0;  // else no page has a flag (a binning before gave up): ranks and starts are old
    const BinDev& bin = a.bin;
    bin_hist_body<kBinILP>(vb, bin.n, bin.keys, bin.page_rank, bin.cell_count, bin.nb_cap, done);
}

template <typename R>
__global__ void __launch_bounds__(kBinThreads) k_batch_scatter(const SceneArgs<R>* __restrict__ A,
                                                               const int32_t* __restrict__ start, int ns) {
    VB vb;
    const SceneArgs<R>& a = A[scene_of_block(start, ns, vb)];
    const bool done = a.cnt->n_blocks > 0;
    const BinDev& bin = a.bin;
    bin_scatter_body<kBinILP, true>(vb, bin.n, bin.keys, bin.page_rank, bin.cell_start, bin.cell_count, bin.perm, bin.keys_sorted,
                     bin.nb_cap, done);
}

template <typename R>
__global__ void __launch_bounds__(32 * kCanonWarps) k_batch_canon(const SceneArgs<R>* __restrict__ A,
                                                                  const int32_t* __restrict__ start, int ns) {
    VB vb;
    const SceneArgs<R>& a = A[scene_of_block(start, ns, vb)];
    bin_canon_body(vb, a.bin, a.scan, a.cnt);
}

// The binning of every scene of a batch: the same steps as launch_binning with
// keys_ready, each one launch over all scenes, with the scans in three passes.
template <typename R>
cudaError_t launch_batch_binning(const SceneArgs<R>* A, const BatchPlan& P, cudaStream_t s) {
    const int ns = P.n_scenes;
    auto T = [&](int m) { return dim3((unsigned)P.total[m]); };
    auto S = [&](int m) { return P.start[m]; };
    cudaError_t e = launch_kernel(k_batch_zero<R>, T(BM_ZERO_FLAGS), dim3(256), 0, s, A, S(BM_ZERO_FLAGS), ns, 1);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scan_reduce<R, 0>, T(BM_KEY_TILES), dim3(kScanThreads), 0, s, A, S(BM_KEY_TILES), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scan_tiles<R, 0>, T(BM_ONE), dim3(kScanThreads), 0, s, A, S(BM_ONE), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scan_apply<R, 0>, T(BM_KEY_TILES), dim3(kScanThreads), 0, s, A, S(BM_KEY_TILES), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_mark<R>, T(BM_KEYSPACE), dim3(256), 0, s, A, S(BM_KEYSPACE), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scan_reduce<R, 1>, T(BM_KEY_TILES), dim3(kScanThreads), 0, s, A, S(BM_KEY_TILES), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scan_tiles<R, 1>, T(BM_ONE), dim3(kScanThreads), 0, s, A, S(BM_ONE), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scan_apply<R, 1>, T(BM_KEY_TILES), dim3(kScanThreads), 0, s, A, S(BM_KEY_TILES), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_compact<R>, T(BM_KEYSPACE), dim3(256), 0, s, A, S(BM_KEYSPACE), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_links<R>, T(BM_LINKS), dim3(256), 0, s, A, S(BM_LINKS), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_zero<R>, T(BM_ZERO_CELLS), dim3(256), 0, s, A, S(BM_ZERO_CELLS), ns, 3);
    if (e == cudaSuccess) e = launch_kernel(k_batch_hist<R>, T(BM_PARTICLES), dim3(kBinThreads), 0, s, A, S(BM_PARTICLES), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scan_reduce<R, 2>, T(BM_CELL_TILES), dim3(kScanThreads), 0, s, A, S(BM_CELL_TILES), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scan_tiles<R, 2>, T(BM_ONE), dim3(kScanThreads), 0, s, A, S(BM_ONE), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scan_apply<R, 2>, T(BM_CELL_TILES), dim3(kScanThreads), 0, s, A, S(BM_CELL_TILES), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_zero<R>, T(BM_ZERO_CELLS), dim3(256), 0, s, A, S(BM_ZERO_CELLS), ns, 2);
    if (e == cudaSuccess) e = launch_kernel(k_batch_scatter<R>, T(BM_PARTICLES), dim3(kBinThreads), 0, s, A, S(BM_PARTICLES), ns);
    if (e == cudaSuccess) e = launch_kernel(k_batch_canon<R>, T(BM_CANON), dim3(32 * kCanonWarps), 0, s, A, S(BM_CANON), ns);
    return e;
}
template cudaError_t launch_batch_binning<float>(const SceneArgs<float>*, const BatchPlan&, cudaStream_t);
template cudaError_t launch_batch_binning<double>(const SceneArgs<double>*, const BatchPlan&, cudaStream_t);

template cudaError_t launch_binning<float>(const SceneDev<float>*, const PState<float>&, BinDev, ScanScratch,
                                           Counters*, int, cudaStream_t, bool, bool);
template cudaError_t launch_binning<double>(const SceneDev<double>*, const PState<double>&, BinDev, ScanScratch,
                                            Counters*, int, cudaStream_t, bool, bool);

}  // namespace gmpm
