// What the FP32 and the FP64 P2G share: the raw particle planes they stage, the
// sequence of page chunks, and the window of previous slots a chunk is staged from.
#pragma once
#include <cstdint>

#include "async_copy.cuh"
#include "kernels.h"

namespace gmpm {

// Raw particle planes, in staging order.
enum RawField : int {
    RW_X = 0, RW_V = 3, RW_B = 6, RW_SIG = 15, RW_C = 21, RW_M = 22, RW_VOL = 23, RW_FP = 24, RW_Q = 25,
    kRawWords = 28
};

// Device pointer of raw plane q.
template <typename R>
__device__ __forceinline__ const R* raw_plane(const PState<R>& st, const PAux<R>& aux, int q) {
    if (q < RW_V) return st.x[q - RW_X];
    if (q < RW_B) return aux.v[q - RW_V];
    if (q < RW_SIG) return aux.B[q - RW_B];
    if (q < RW_C) return aux.sigma[q - RW_SIG];
    if (q == RW_C) return st.c;
    if (q == RW_M) return st.m;
    if (q == RW_VOL) return aux.vol;
    if (q == RW_FP) return aux.FP;
    return aux.q[q - RW_Q];
}

// Chunk sequence of one CTA: its pages b + k g (b, g: the CTA's index and the
// CTA count of its scene's share of the launch), each cut into runs of CH
// slots.  Every thread runs the same iterator.
template <int CH>
struct ChunkIter {
    int page, next, end;  // current page, next run start, page end
    int nbs, nbe;         // slot range of the following page (loaded one page ahead)
    int stride;           // CTAs of the scene's share of the launch
    __device__ void init(const BinDev& bin, int nb, VB vb) {
        page = vb.b;
        stride = vb.g;
        next = end = 0;
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
    // Next chunk (page, first slot, count, last chunk of its page); count 0 when done.
    __device__ void step(const BinDev& bin, int nb, int& b, int& s0, int& n, int& last) {
        while (page < nb && next >= end) {
            page += stride;
            next = nbs;
            end = nbe;
            if (page < nb) preload(bin, nb);
        }
        if (page < nb) {
            b = page;
            s0 = next;
            n = min(CH, end - next);
            next += CH;
            last = next >= end;
        } else {
            b = -1;
            s0 = n = last = 0;
        }
    }
};

// Margin of a staging window on either side of its chunk.
constexpr int kMargin = 64;

// Start of the staging window (of len elements) of a chunk: the median over
// three particles of (previous slot - slot) estimates the chunk's shift between
// the orders.
__device__ __forceinline__ int64_t window_start(const int32_t* o, int n, int64_t stride, int len) {
    const int64_t d0 = o[0], d1 = (int64_t)o[n / 2] - n / 2, d2 = (int64_t)o[n - 1] - (n - 1);
    const int64_t med = max(min(d0, d1), min(max(d0, d1), d2));
    int64_t w = (med - kMargin) & ~(int64_t)3;
    w = min(w, stride - len);
    return max(w, (int64_t)0);
}

}  // namespace gmpm
