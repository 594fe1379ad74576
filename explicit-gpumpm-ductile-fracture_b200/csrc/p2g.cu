// P2G: APIC particle-to-grid transfer on SPGrid pages (P2G_APIC,
// P2GKernal.cu:512-702) plus the phase-field channels (volP2G_APIC,
// preConditionP2G_APIC, AxP2G_APIC: P2GKernal.cu:897-1326).
//
// Each CTA walks its particle pages (grid-stride) in chunks of up to kP2GChunk
// sorted slots (a whole page of 8 particles per cell; denser pages are cut into
// runs of cells, CellChunkIter).  A page's particles
// share the page's 6x6x6 node window and, within a cell, the same 3x3x3
// stencil.  Between substeps the particle planes are in the previous sorted
// order and perm is close to the identity, so the 28 raw input planes of a
// chunk are fetched as contiguous windows of previous slots with bulk copies
// (one lane of every warp issues a few planes; the tensor memory accelerator
// moves the data) and read where they land, through the slot's place in the
// window.  A chunk with a particle whose previous slot falls outside the window
// (it changed page) is first gathered into sorted order in shared memory: nearly
// every chunk of a scene's first substep, whose previous order is the caller's,
// and 3 to 9% of the chunks of 8.4M-particle plates 100 to 300 substeps on.
//
// Work split: one lane per cell and channel group (in dense pages several lanes
// share a cell and add their sums by shuffles).  A lane walks its cell's
// particles and keeps the cell's 27 node sums of its channels in registers, so
// a particle costs each lane its weights once and 27 fused multiply-adds per
// term and channel, with no shuffles and no atomics.  The groups, one per pair
// of warps, hold two channels per packed FP32 instruction (fma.rn.f32x2):
//   0: momentum x, y        1: momentum z, grad w . q
//   2: mass, damage weight  3: weight, V w, V w FP
// With w = X_i Y_j Z_k, the momentum of node (i, j, k) is
//   P_i (Y_j Z_k) + X_i (Y_j U_k + Q_j Z_k),
// where P, Q and U hold the APIC and stress terms of one axis each:
//   P_i = b_x (i - d_x) X_i + s_x X'_i, Q likewise, U_k with the velocity term.
// Lane l of a group's first warp takes the fuller of cells l and l + 32, and of
// its second warp the other, so that a warp's lanes hold cells of similar
// counts (its loop runs as long as its fullest cell).
//
// The page's cell sums then go to shared memory (over the staged planes) and
// are gathered per window node in a fixed order (gather_item) into the page's
// tile, which one bulk copy writes to HBM.  Results are bitwise reproducible
// in both modes of the scene.  The grid kernel sums the eight page tiles
// overlapping each grid page in fixed slot order.
//
// Bound: neither HBM (19% of its peak) nor one pipe, but the chain of a page's
// phases (copy 2,000 cycles, sweep 9,000, gather 3,000), which the two CTAs of an
// SM overlap in part: 54% of the issue slots, FMA pipe 48%, shared memory 47%.
// Measured on FP32 plates: 0.73 ms at 8.4M particles and 2.78 ms at 33.5M, where
// one lane per stencil column, all lanes on the same particle, took 1.209 and
// 4.67 (88 warp instructions a particle against 52: every particle's words were
// read, and its weights formed, by 27 lanes).
#include <cstdint>

#include "launch.cuh"
#include "p2g_common.cuh"

namespace gmpm {
namespace {

using R = float;

constexpr int kP2GGroups = 4;
constexpr int kP2GThreads = 64 * kP2GGroups;  // two warps (64 cells) per channel group
constexpr int kP2GChunk = 576;
constexpr int kCtasPerSm = 2;  // by registers and shared memory

// Staging window of previous slots: the chunk's slots plus kMargin on either
// side; planes padded in shared memory to spread banks.
struct Staging {
    static constexpr int W = kP2GChunk + 2 * kMargin;      // longest window (elements)
    static constexpr int WS = W + (int)(16 / sizeof(R));   // plane stride in shared memory
    static_assert(W <= kPlanePad, "window fits the plane padding");
    static_assert((W * sizeof(R)) % 16 == 0 && (WS * sizeof(R)) % 16 == 0, "bulk copy granularity");
};
__device__ __forceinline__ int window_length(int n) { return (n + 2 * kMargin + 3) & ~3; }

// Two channels of one value, for Blackwell's packed FP32 instructions.
using P2 = float2;
__device__ __forceinline__ P2 pk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ P2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ P2 fma2(P2 a, P2 b, P2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ P2 mul2(P2 a, P2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ P2 add2(P2 a, P2 b) { return __fadd2_rn(a, b); }

// quadratic B-spline weights on nodes base+0..2 and their gradients times dx,
// d = (x - x_base) / dx (P2GKernal.cu:590-611)
__device__ __forceinline__ void bspline1d(R d, R* w, R* h) {
    const R z0 = R(1.5) - d, z1 = d - R(1), z2 = d - R(0.5);
    w[0] = R(0.5) * z0 * z0;
    w[1] = R(0.75) - z1 * z1;
    w[2] = R(0.5) * z2 * z2;
    h[0] = -z0;
    h[1] = R(-2) * z1;
    h[2] = z2;
}

__device__ __forceinline__ void kahan_add2(P2& s, P2& c, P2 v) {
    const P2 minus = dup(R(-1));
    const P2 y = fma2(c, minus, v);
    const P2 t = add2(s, y);
    c = fma2(y, minus, fma2(s, minus, t));
    s = t;
}
// The CTA's barrier at points where warps of different groups arrive from
// different code (barrier 1; __syncthreads uses barrier 0).
__device__ __forceinline__ void p2g_barrier() {
    asm volatile("bar.sync 1, %0;\n" ::"n"(kP2GThreads) : "memory");
}

// Chunk sequence of one CTA: its pages b + k g (b, g: the CTA's index and the
// CTA count of its scene's share of the launch).  A page of up to kP2GChunk
// slots is one chunk.  A fuller page is cut into aligned runs of 32, 16, 8, ...
// cells, each the largest that fits, whose particles several lanes share; a
// single cell above kP2GChunk is cut by slots.  P2G of 1M particles with a lane
// per cell of runs of kP2GChunk slots, and so: 16 per cell 167 -> 146 us, 32 per
// cell 250 -> 169, 64 per cell 469 -> 221; 5,000 particles of 105k in one cell
// 803 -> 187.  Every thread runs the same iterator.
struct CellChunkIter {
    int page, next, end;  // current page, next slot, page end
    int cell;             // cell of the next slot (or an empty one before it)
    int nbs, nbe;         // slot range of the following page (loaded one page ahead)
    int stride;           // CTAs of the scene's share of the launch
    __device__ void init(const BinDev& bin, int nb, VB vb) {
        page = vb.b;
        stride = vb.g;
        next = end = cell = 0;
        if (page < nb) {
            next = bin.cell_start[(int64_t)page * 64];
            end = bin.cell_start[(int64_t)page * 64 + 64];
        }
        preload(bin, nb);
    }
    __device__ void preload(const BinDev& bin, int nb) {
        const int q = page + stride;
        nbs = nbe = 0;
        if (q < nb) {
            nbs = bin.cell_start[(int64_t)q * 64];
            nbe = bin.cell_start[(int64_t)q * 64 + 64];
        }
    }
    // The next chunk of a page (start: its cells' starts) that is cut: its first slot, count and cells (as in step),
    // and the cell after it.  Out of line, with few registers, for the sake of the pages that are not.
    static __device__ __noinline__ int4 cut(const int32_t* start, int cell, int next) {
        int n, cells;
        do {
            int stop[6];  // ends of the runs of 1, 2, 4, ... cells
#pragma unroll
            for (int q = 0; q < 6; ++q) stop[q] = start[min(cell + (1 << q), 64)];
            int size = 1, e = min(stop[0], next + kP2GChunk);
#pragma unroll
            for (int q = 1; q < 6; ++q)
                if ((cell & ((1 << q) - 1)) == 0 && stop[q] - next <= kP2GChunk) {
                    size = 1 << q;
                    e = stop[q];
                }
            n = e - next;
            cells = size | cell << 8;
            if (size > 1 || e == stop[0]) cell += size;
        } while (n == 0);
        return make_int4(next, n, cells, cell);
    }
    // Next chunk (page, first slot, count; 0 when done) and its cells: their number (a power of two), << 8 the
    // first, kLastChunk: the last chunk of its page.
    __device__ void step(const BinDev& bin, int nb, int& b, int& s0, int& n, int& cells) {
        while (page < nb && next >= end) {
            page += stride;
            next = nbs;
            end = nbe;
            cell = 0;
            if (page < nb) preload(bin, nb);
        }
        b = -1;
        s0 = n = cells = 0;
        if (page >= nb) return;
        b = page;
        s0 = next;
        if (cell == 0 && end - next <= kP2GChunk) {
            n = end - next;
            cells = 64;
        } else {
            const int4 r = cut(bin.cell_start + (int64_t)page * 64, cell, next);
            n = r.y;
            cells = r.z;
            cell = r.w;
        }
        next = s0 + n;
        if (next >= end) cells |= kLastChunk;
    }
    static constexpr int kLastChunk = 1 << 16;
};

// What a lane keeps about its cell and the scene.
struct LaneCell {
    R b[3];           // base node coordinates
    R dx, inv_dx, kD, kS;  // kD = dx D^-1, kS = -dt / dx
};

// Staged words of a group's particle, x y z first.
__device__ constexpr int kWordsXY[17] = {RW_X,     RW_X + 1, RW_X + 2, RW_M,       RW_V,       RW_V + 1,
                                         RW_B,     RW_B + 1, RW_B + 3, RW_B + 4,   RW_B + 6,   RW_B + 7,
                                         RW_SIG,   RW_SIG + 1, RW_SIG + 3, RW_SIG + 4, RW_SIG + 5};
__device__ constexpr int kWordsZQ[14] = {RW_X,     RW_X + 1, RW_X + 2,   RW_M,       RW_V + 2,   RW_B + 2, RW_B + 5,
                                         RW_B + 8, RW_SIG + 4, RW_SIG + 5, RW_SIG + 2, RW_Q,     RW_Q + 1, RW_Q + 2};
__device__ constexpr int kWordsMC[5] = {RW_X, RW_X + 1, RW_X + 2, RW_M, RW_C};
__device__ constexpr int kWordsV[5] = {RW_X, RW_X + 1, RW_X + 2, RW_VOL, RW_FP};

__device__ __forceinline__ void particle_weights(const R* x, const LaneCell& L, R d[3], R w[3][3], R h[3][3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        d[a] = (x[a] - L.b[a] * L.dx) * L.inv_dx;
        bspline1d(d[a], w[a], h[a]);
    }
}

// acc += P_i (Y_j Z_k) + X_i (Y_j U_k + Q_j Z_k)
__device__ __forceinline__ void add_terms(const P2 P[3], const P2 Q[3], const P2 U[3],
                                          const R w[3][3], P2 acc[27]) {
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const P2 yz = dup(w[1][j] * w[2][k]);
            const P2 g = fma2(dup(w[1][j]), U[k], mul2(Q[j], dup(w[2][k])));
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                P2& A = acc[i * 9 + j * 3 + k];
                A = fma2(dup(w[0][i]), g, fma2(P[i], yz, A));
            }
        }
}

// A lane's particles lo, lo + step, ... below hi: o holds their previous slots, w0 the first one staged.  Loading the
// next particle's words ahead was slower (730 against 715 us at 8.4M particles): the moves it takes cost more than the
// latency.
template <bool kStep, int N, typename F>
__device__ __forceinline__ void sweep(const R* stage, const int32_t* o, int w0, int lo, int hi, int step,
                                      const int (&plane)[N], F add) {
#pragma unroll 1
    for (int p = lo; p < hi; p += kStep ? step : 1) {
        const R* s = stage + (o[p] - w0);
        R v[N];
#pragma unroll
        for (int q = 0; q < N; ++q) v[q] = s[plane[q] * Staging::WS];
        add(v);
    }
}

// Group 0: momentum x and y.
__device__ __forceinline__ void add_momentum_xy(const R (&v)[17], const LaneCell& L, P2 acc[27]) {
    R d[3], w[3][3], h[3][3];
    particle_weights(v, L, d, w, h);
    const R m = v[3];
    const P2 mD = dup(m * L.kD);
    // sigma rows x, y; stored xx yy zz xy xz yz.  B planes are column-major (r + 3c).
    const R xx = L.kS * v[12], yy = L.kS * v[13], xy = L.kS * v[14], xz = L.kS * v[15], yz = L.kS * v[16];
    const P2 sg[3] = {pk(xx, xy), pk(xy, yy), pk(xz, yz)};
    P2 T[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const P2 b = mul2(mD, pk(v[6 + 2 * a], v[7 + 2 * a]));
        P2 t = mul2(b, dup(-d[a]));
        if (a == 2) t = fma2(dup(m), pk(v[4], v[5]), t);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            T[a][i] = fma2(t, dup(w[a][i]), mul2(sg[a], dup(h[a][i])));
            if (i < 2) t = add2(t, b);
        }
    }
    add_terms(T[0], T[1], T[2], w, acc);
}

// Group 1: momentum z and the phase-field flux grad w . q.
__device__ __forceinline__ void add_momentum_z_flux(const R (&v)[14], const LaneCell& L, P2 acc[27]) {
    R d[3], w[3][3], h[3][3];
    particle_weights(v, L, d, w, h);
    const R m = v[3];
    const R mD = m * L.kD;
    const P2 kk = pk(L.kS, L.inv_dx);
    P2 T[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const P2 sg = mul2(kk, pk(v[8 + a], v[11 + a]));
        const R b = mD * v[5 + a];
        R t = -(b * d[a]);
        if (a == 2) t += m * v[4];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            T[a][i] = mul2(sg, dup(h[a][i]));
            T[a][i].x += t * w[a][i];
            if (i < 2) t += b;
        }
    }
    add_terms(T[0], T[1], T[2], w, acc);
}

// Group 2: mass and damage weight.
__device__ __forceinline__ void add_mass_damage(const R (&v)[5], const LaneCell& L, P2 acc[27]) {
    R d[3], w[3][3], h[3][3];
    particle_weights(v, L, d, w, h);
    P2 X[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) X[i] = mul2(pk(v[3], v[4]), dup(w[0][i]));
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const P2 yz = dup(w[1][j] * w[2][k]);
#pragma unroll
            for (int i = 0; i < 3; ++i) acc[i * 9 + j * 3 + k] = fma2(X[i], yz, acc[i * 9 + j * 3 + k]);
        }
}

// Group 3: weight and V w (pairs), V w FP.
__device__ __forceinline__ void add_weights(const R (&v)[5], const LaneCell& L, P2 acc[27], R one[27]) {
    R d[3], w[3][3], h[3][3];
    particle_weights(v, L, d, w, h);
    const R V = v[3], VF = v[3] * v[4];
    P2 X[3];
    R X1[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        X[i] = pk(w[0][i], V * w[0][i]);
        X1[i] = VF * w[0][i];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const R yz = w[1][j] * w[2][k];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const int q = i * 9 + j * 3 + k;
                acc[q] = fma2(X[i], dup(yz), acc[q]);
                one[q] += X1[i] * yz;
            }
        }
}

// Sums of `step` neighbouring lanes that share a cell (a power of two), in the
// lane that writes them; the others write zeros, to cells without particles.
template <typename T>
__device__ __forceinline__ void share_sums(T acc[27], int step, bool writes);
template <>
__device__ __forceinline__ void share_sums(R acc[27], int step, bool writes) {
#pragma unroll 1
    for (int o = 1; o < step; o <<= 1)
#pragma unroll
        for (int q = 0; q < 27; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
#pragma unroll
    for (int q = 0; q < 27; ++q) acc[q] = writes ? acc[q] : R(0);
}
template <>
__device__ __forceinline__ void share_sums(P2 acc[27], int step, bool writes) {
#pragma unroll 1
    for (int o = 1; o < step; o <<= 1)
#pragma unroll
        for (int q = 0; q < 27; ++q)
            acc[q] = add2(acc[q], pk(__shfl_xor_sync(0xffffffffu, acc[q].x, o), __shfl_xor_sync(0xffffffffu, acc[q].y, o)));
#pragma unroll
    for (int q = 0; q < 27; ++q) acc[q] = writes ? acc[q] : pk(R(0), R(0));
}

// Cell sums of a page, [slot][stencil node][cell] pairs: slots 0..2 are groups
// 0..2, slot 3 (W, V w), slot 4 (V w FP, 0).  The slot stride is padded so that
// the five slots of a gathered column fall in different banks.
constexpr int kSlots = 5;
constexpr int kSlotStride = 27 * 64 + 2;
constexpr int kItems = 36 * kSlots * 2;  // of the page gather
// Tile channels of a slot's pair (-1: none).
__device__ __forceinline__ int slot_channel(int slot, int half) {
    const int c0 = slot == 0 ? CH_P0 : slot == 1 ? CH_P2 : slot == 2 ? CH_M : slot == 3 ? CH_W : CH_VWFP;
    const int c1 = slot == 0 ? CH_P1 : slot == 1 ? CH_KC : slot == 2 ? CH_CW : slot == 3 ? CH_VW : -1;
    return half == 0 ? c0 : c1;
}
// Window columns (a, b) as 6 a + b, by the number of cell columns that reach
// them (9 6 4 3 2 1), so that a warp of the gather runs a similar number of terms.
__constant__ unsigned char kColumnOrder[36] = {14, 15, 20, 21, 8,  9,  26, 27, 13, 16, 19, 22, 7,  10, 25, 28, 12, 17,
                                               18, 23, 2,  3,  32, 33, 6,  11, 24, 29, 1,  4,  31, 34, 0,  5,  30, 35};

__device__ __forceinline__ void set_lane_cell(LaneCell& L, uint32_t page, int cell) {
    int bx, by, bz;
    page_coords(page, bx, by, bz);
    L.b[0] = R(4 * bx + (cell >> 4));
    L.b[1] = R(4 * by + ((cell >> 2) & 3));
    L.b[2] = R(4 * bz + (cell & 3));
}

// Sums of a gather item (see make_item): three nodes of a window column, over
// the cell columns that reach it, x-major.  A cell column's cells are added
// first, then the up to nine columns, compensated.  (Compensating along x only
// took 1% off the kernel and lost what the sums of one cell column had over
// those of a lane per stencil column.)  The upper half is the
// mirror image: node 5 - z takes cell 3 - cz at stencil node 2 - k.
constexpr int kNextY = 4 - 3 * 64, kNextX = 16 - 9 * 64;  // a node's sum in the next cell column along y, x
__device__ __forceinline__ void gather_item(const P2* __restrict__ sums, uint32_t w, P2 sum[3]) {
    const int ni = (w >> 15) & 3, nj = (w >> 17) & 3;
    const bool up = (w >> 19) & 1;
    const int sk = up ? -64 : 64, sc = up ? -1 : 1;
    const P2* src = sums + (w & 0x7fff);
    P2 comp[3];
#pragma unroll
    for (int z = 0; z < 3; ++z) sum[z].x = sum[z].y = comp[z].x = comp[z].y = 0;
#pragma unroll 1
    for (int i = 0; i < ni; ++i) {
        const P2* col = src;
#pragma unroll 1
        for (int j = 0; j < nj; ++j) {
            kahan_add2(sum[0], comp[0], col[0]);
            kahan_add2(sum[1], comp[1], add2(col[sk], col[sc]));
            kahan_add2(sum[2], comp[2], add2(add2(col[2 * sk], col[sk + sc]), col[2 * sc]));
            col += kNextY;
        }
        src += kNextX;
    }
}

struct P2GMeta {
    R tile[kP2GChannels * kWindowNodes];  // the page's gathered tile
    int32_t o[2][kP2GChunk];              // previous slot per chunk slot; 2 buffers
    int32_t cs[2][68];                    // cell starts of the chunk's page (65 used)
    uint32_t bkey[2];
    uint64_t bar;                         // completion of the staging bulk copies
    const R* plane[kRawWords];            // raw planes in HBM
    uint32_t item[kItems][2];             // gather items, built once per CTA (make_item)
    int abort;                            // a bounded wait gave up
};

// A gather item: window column (a, b), slot and half of the column's six nodes.
//   word 0: the first column's cell sum (bits 0-14), columns along x and y (15-16, 17-18), half (19)
//   word 1: the item's first node in the tile, of the slot's first and second channel (bits 0-10, 16-26; 0xffff: none)
__device__ __forceinline__ void make_item(int q, uint32_t w[2]) {
    const int rank = q / (2 * kSlots), r = q - rank * 2 * kSlots;
    const int slot = r >> 1, up = r & 1, col = kColumnOrder[rank];
    const int a = col / 6, b = col - 6 * a;
    // cell columns cx0 .. cx0 + ni - 1, cy0 .. cy0 + nj - 1, at stencil nodes (a - cx, b - cy)
    const int cx0 = max(0, a - 2), ni = min(3, a) - cx0 + 1, cy0 = max(0, b - 2), nj = min(3, b) - cy0 + 1;
    const int src = slot * kSlotStride + ((a - cx0) * 9 + (b - cy0) * 3) * 64 + cx0 * 16 + cy0 * 4;
    w[0] = (uint32_t)(src + (up ? 2 * 64 + 3 : 0)) | (uint32_t)ni << 15 | (uint32_t)nj << 17 | (uint32_t)up << 19;
    const int ch0 = slot_channel(slot, 0), ch1 = slot_channel(slot, 1), z = col * 6 + (up ? 5 : 0);
    w[1] = (uint32_t)(ch0 * kWindowNodes + z) | ((uint32_t)(ch1 < 0 ? 0xffff : ch1 * kWindowNodes + z) << 16);
}

// Bulk copies of the raw planes over the chunk's window, a few planes per warp.
// Called by one lane of every warp.
__device__ __forceinline__ void issue_staging(const R* const* plane, uint64_t* bar, R* stage, int64_t w0, int len, int warp) {
    constexpr int WS = Staging::WS, kWarps = kP2GThreads / 32;
    fence_proxy_async_shared();
    const int planes = (kRawWords - warp + kWarps - 1) / kWarps;
    mbar_arrive_expect_tx(bar, (unsigned)(planes * len * sizeof(R)));
    for (int q = warp; q < kRawWords; q += kWarps)
        bulk_copy_g2s(stage + (size_t)q * WS, plane[q] + w0, (unsigned)(len * sizeof(R)), bar);
}

// Slots, cell starts and key of a chunk.
__device__ __forceinline__ void issue_p2g_meta(int32_t* o, int32_t* cs, uint32_t* bkey, int t, int b, int s0, int n,
                                               const BinDev& bin) {
    if (n <= 0) return;
    for (int p = t; p < n; p += kP2GThreads) cp_async_elem(&o[p], &bin.perm[s0 + p]);
    if (t < 65) cp_async_elem(&cs[t], &bin.cell_start[(int64_t)b * 64 + t]);
    if (t == 65) cp_async_elem(bkey, &bin.block_keys[b]);
}

// Particles outside the window: gather the whole chunk into sorted order, in
// place (a batch of planes is read by every thread before any is written), and
// set the slots o to their new places.
__device__ __forceinline__ void sort_staged(const R* const* plane, int32_t* o, R* stage, int n, int64_t w0, int len) {
    const int t = threadIdx.x;
    constexpr int kThreads = kP2GThreads;
    constexpr int WS = Staging::WS, kBatch = 4, kPer = (kP2GChunk + kThreads - 1) / kThreads;
    static_assert(kRawWords % kBatch == 0, "whole batches");
#pragma unroll 1
    for (int qb = 0; qb < kRawWords; qb += kBatch) {
        R v[kPer][kBatch];
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int p = t + i * kThreads;
            if (p >= n) continue;
            const int64_t r = (int64_t)o[p] - w0;
            if (r >= 0 && r < len) {
#pragma unroll
                for (int q = 0; q < kBatch; ++q) v[i][q] = stage[(size_t)(qb + q) * WS + r];
            } else {
#pragma unroll
                for (int q = 0; q < kBatch; ++q) v[i][q] = plane[qb + q][o[p]];
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int p = t + i * kThreads;
            if (p >= n) continue;
#pragma unroll
            for (int q = 0; q < kBatch; ++q) stage[(size_t)(qb + q) * WS + p] = v[i][q];
        }
    }
    for (int p = t; p < n; p += kThreads) o[p] = (int32_t)(w0 + p);
    __syncthreads();
}

constexpr size_t p2g_stage_bytes() {
    return sizeof(R) * (size_t)kRawWords * Staging::WS;
}
static_assert(2 * sizeof(float) * kSlots * kSlotStride <= p2g_stage_bytes(), "cell sums fit the staged planes");

// Cell sums of a chunk: this lane's particles lo, lo + step, ... below hi of its cell (L), summed into column `cell`.
// Each group's sums stay in its own registers over the CTA's barrier, after which they overwrite the staged planes.
// kShared: `step` neighbouring lanes share the cell, and one of them writes.
template <bool kShared>
__device__ __forceinline__ void cell_sums(const R* stage, P2* sums, const int32_t* o, int win, int group, int cell, int lo,
                                          int hi, int step, bool writes, const LaneCell& L) {
    P2 acc[27];
#pragma unroll
    for (int q = 0; q < 27; ++q) acc[q] = pk(R(0), R(0));
    P2* out = sums + group * kSlotStride + cell;
    if (group == 0)
        sweep<kShared>(stage, o, win, lo, hi, step, kWordsXY, [&](auto& v) { add_momentum_xy(v, L, acc); });
    else if (group == 1)
        sweep<kShared>(stage, o, win, lo, hi, step, kWordsZQ, [&](auto& v) { add_momentum_z_flux(v, L, acc); });
    else if (group == 2)
        sweep<kShared>(stage, o, win, lo, hi, step, kWordsMC, [&](auto& v) { add_mass_damage(v, L, acc); });
    if (group < 3) {
        if (kShared) share_sums(acc, step, writes);
        if (threadIdx.x == 0) bulk_store_wait_read();  // the previous tile has left shared memory
        p2g_barrier();
#pragma unroll
        for (int q = 0; q < 27; ++q) out[q * 64] = acc[q];
    } else {
        R one[27];
#pragma unroll
        for (int q = 0; q < 27; ++q) one[q] = R(0);
        sweep<kShared>(stage, o, win, lo, hi, step, kWordsV, [&](auto& v) { add_weights(v, L, acc, one); });
        if (kShared) {
            share_sums(acc, step, writes);
            share_sums(one, step, writes);
        }
        p2g_barrier();
#pragma unroll
        for (int q = 0; q < 27; ++q) {
            out[q * 64] = acc[q];
            out[kSlotStride + q * 64] = pk(one[q], R(0));
        }
    }
}

// Cell sums of a chunk of part of a page's cells: a group's 64 lanes share them, up to 32 lanes (of one warp) each.  Out
// of line and with loops of its own, for the sake of whole pages (P2G of 1M particles, 8 per cell: 131.6 us; 132.5 with
// this inlined, 142 with one loop for both forms).
__device__ __noinline__ void shared_cell_sums(const R* stage, P2* sums, const int32_t* o, const int32_t* cs, uint32_t page,
                                              int win, int c0, int n0, int cells, int group, bool lighter, R dx, R inv_dx,
                                              R kD, R kS) {
    const int nc = cells & 127, ca = (cells >> 8) & 63, vl = (threadIdx.x & 31) + (lighter ? 32 : 0);
    const int step = min(64 / nc, 32), c = vl / step, sub = vl & (step - 1);
    int cell = min(ca + c, ca + nc - 1);
    LaneCell L;
    L.dx = dx;
    L.inv_dx = inv_dx;
    L.kD = kD;
    L.kS = kS;
    set_lane_cell(L, page, cell);
    const int hi = min(cs[cell + 1], c0 + n0) - c0;
    const int lo = c < nc ? max(cs[cell], c0) - c0 + sub : hi;
    const bool writes = c < nc && sub == 0;
    if (!writes) {  // the cell it writes zeros to: as many are without particles as lanes do not write
        const int j = c < nc ? vl - c - 1 : vl - nc;
        cell = j < ca ? j : j + nc;
    }
    cell_sums<true>(stage, sums, o, win, group, cell, lo, hi, step, writes, L);
}

__device__ __forceinline__ void p2g_body(VB vb, const SceneDev<R>* sc, const PState<R>& st,
                                         const PAux<R>& aux, const BinDev& bin, R* tile,
                                         Counters* cnt) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* stage = reinterpret_cast<R*>(smem_raw);   // [kRawWords][WS] raw planes
    P2* sums = reinterpret_cast<P2*>(smem_raw);  // the page's cell sums, once the planes are read
    P2GMeta& S = *reinterpret_cast<P2GMeta*>(smem_raw + p2g_stage_bytes());

    const int t = threadIdx.x;
    const int warp = t >> 5, lane = t & 31;
    // Two warps per group.  A scheduler (warp mod 4) holds one with the fuller and one with the lighter
    // cells, of a momentum group and of a weight group.
    const int group = (warp & 1) | ((warp >> 2) << 1);
    const bool lighter = ((warp >> 1) & 1) != (warp >> 2);
    const int nb = min(cnt->n_blocks, bin.nb_cap);
    LaneCell L;
    L.dx = sc->dx;
    L.inv_dx = sc->inv_dx;
    L.kD = sc->Dinv * sc->dx;
    L.kS = -sc->dt * sc->inv_dx;

    // prologue: descriptors of chunks 0 and 1, meta of chunk 0
    CellChunkIter it;
    it.init(bin, nb, vb);
    int b0, c0, n0, cells0, b1, c1, n1, cells1;
    it.step(bin, nb, b0, c0, n0, cells0);
    it.step(bin, nb, b1, c1, n1, cells1);
    if (t == 0) {
        S.abort = 0;
        mbar_init(&S.bar, kP2GThreads / 32);
        mbar_init_fence();
    }
#pragma unroll
    for (int q = 0; q < kRawWords; ++q)
        if (t == q) S.plane[q] = raw_plane(st, aux, q);
    for (int q = t; q < kItems; q += kP2GThreads) make_item(q, S.item[q]);
    issue_p2g_meta(S.o[0], S.cs[0], &S.bkey[0], t, b0, c0, n0, bin);
    cp_async_commit();
    bool first = true;  // first chunk of its page
    int done = -1;      // page whose tile is ready to be written

    for (int k = 0;; ++k) {
        const int m = k & 1;
        cp_async_wait_all();
        // the sums and the tile were accessed by this thread; bulk copies follow
        fence_proxy_async_shared();
        __syncthreads();
        if (t == 0 && done >= 0)
            bulk_copy_s2g(tile + (int64_t)done * kP2GChannels * kWindowNodes, S.tile, (unsigned)sizeof(S.tile));
        done = -1;
        if (n0 <= 0) break;
        const int len = window_length(n0);
        const int64_t w0 = window_start(S.o[m], n0, st.stride, len);
        if (lane == 0) issue_staging(S.plane, &S.bar, stage, w0, len, warp);
        issue_p2g_meta(S.o[m ^ 1], S.cs[m ^ 1], &S.bkey[m ^ 1], t, b1, c1, n1, bin);
        cp_async_commit();
        bool outside = false;
        for (int p = t; p < n0; p += kP2GThreads) {
            const int64_t r = (int64_t)S.o[m][p] - w0;
            outside = outside || r < 0 || r >= len;
        }
        // this lane's cell: the fuller (or, in the group's other warp, the lighter) of cells lane and lane + 32
        int cell, lo, hi;
        {
            const int* cs = S.cs[m];
            const bool upper_fuller = cs[lane + 33] - cs[lane + 32] > cs[lane + 1] - cs[lane];
            cell = upper_fuller != lighter ? lane + 32 : lane;
            lo = max(cs[cell], c0) - c0;
            hi = min(cs[cell + 1], c0 + n0) - c0;
            set_lane_cell(L, S.bkey[m], cell);
        }
        if (!mbar_wait(&S.bar, (unsigned)m)) S.abort = 1;
        outside = __syncthreads_or(outside);
        if (S.abort) break;
        if (outside) sort_staged(S.plane, S.o[m], stage, n0, w0, len);
        const int win = (int)w0;

        if (cells0 & 64)
            cell_sums<false>(stage, sums, S.o[m], win, group, cell, lo, hi, 1, true, L);
        else
            shared_cell_sums(stage, sums, S.o[m], S.cs[m], S.bkey[m], win, c0, n0, cells0, group, lighter, L.dx, L.inv_dx,
                             L.kD, L.kS);
        __syncthreads();
        // Gather: window column (a, b), slot and half of the column's six nodes per item.  A node sums its
        // cell columns (cx, cy) = (a - i, b - j) in ascending order (compensated), each column's cells
        // first.  The upper half is the mirror image: node 5 - z takes cell 3 - cz at stencil node 2 - k.
        // Threads past the first 152 take a second, short item.
        for (int it0 = t; it0 < kItems; it0 = it0 < kP2GThreads ? 2 * kP2GThreads - 1 - it0 : kItems) {
            const uint32_t w0 = S.item[it0][0], w1 = S.item[it0][1];
            P2 sum[3];
            gather_item(sums, w0, sum);
            R* t0 = S.tile + (w1 & 0xffff);
            R* t1 = S.tile + (w1 >> 16);
            const int dz = ((w0 >> 19) & 1) ? -1 : 1;
            const bool two = (w1 >> 16) != 0xffff;
            if (first) {
#pragma unroll
                for (int z = 0; z < 3; ++z) {
                    t0[z * dz] = sum[z].x;
                    if (two) t1[z * dz] = sum[z].y;
                }
            } else {
#pragma unroll
                for (int z = 0; z < 3; ++z) {
                    t0[z * dz] += sum[z].x;
                    if (two) t1[z * dz] += sum[z].y;
                }
            }
        }
        first = (cells0 & CellChunkIter::kLastChunk) != 0;
        if (first) done = b0;
        b0 = b1; c0 = c1; n0 = n1; cells0 = cells1;
        it.step(bin, nb, b1, c1, n1, cells1);
    }
    cp_async_wait_all();
    if (t == 0) bulk_store_wait();
    if (S.abort) {
        // A staging copy may still be in flight: wait for it (bounded) before
        // the CTA's shared memory goes away, and report.
        if (t == 0) {
            raise_flag(cnt, GMPM_FLAG_COPY_TIMEOUT);
            mbar_wait(&S.bar, 0u);
            mbar_wait(&S.bar, 1u);
        }
    }
}

__global__ void __launch_bounds__(kP2GThreads, kCtasPerSm)
    k_p2g(const SceneDev<R>* sc, PState<R> st, PAux<R> aux, BinDev bin, R* tile,
            Counters* cnt, double* diag) {
    depend_on_previous();
    // the sums that the grid stage adds to
    if (blockIdx.x == 0 && threadIdx.x < 4) diag[threadIdx.x] = 0.0;
    p2g_body(own_blocks(), sc, st, aux, bin, tile, cnt);
}

// Batched launch: the same body for the scene that owns this CTA.
__global__ void __launch_bounds__(kP2GThreads, kCtasPerSm)
    k_batch_p2g(const SceneArgs<R>* __restrict__ A, const int32_t* __restrict__ start, int ns) {
    VB vb;
    const SceneArgs<R>& a = A[scene_of_block(start, ns, vb)];
    p2g_body(vb, a.sc, a.in, a.aux, a.bin, reinterpret_cast<R*>(a.grid.tile), a.cnt);
}

constexpr size_t kSmem = p2g_stage_bytes() + sizeof(P2GMeta);

}  // namespace

template <>
cudaError_t prepare_p2g<float>() {
    cudaError_t e = cudaFuncSetAttribute(k_p2g, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_batch_p2g, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    return e;
}

template <>
int p2g_ctas<float>(int nb_cap, int sms) {
    return max(1, min(nb_cap, sms * kCtasPerSm));
}

template <>
cudaError_t launch_batch_p2g<float>(const SceneArgs<float>* A, const BatchPlan& P, cudaStream_t s) {
    return launch_kernel(k_batch_p2g, dim3((unsigned)P.total[BM_P2G]), dim3(kP2GThreads), kSmem, s, A, P.start[BM_P2G],
                         P.n_scenes);
}

template <>
cudaError_t launch_p2g<float>(const SceneDev<float>* sc, const PState<float>& st, const PAux<float>& aux, BinDev bin,
                               GridDev grid, Counters* cnt, LaunchCfg cfg, cudaStream_t stream) {
    return launch_dependent(k_p2g, dim3((unsigned)p2g_ctas<float>(bin.nb_cap, cfg.num_sms)), dim3(kP2GThreads), kSmem, stream, sc, st,
                            aux, bin, reinterpret_cast<float*>(grid.tile), cnt, grid.diag);
}

}  // namespace gmpm
