// pgd_kernels.cuh -- device helpers shared by the decomposition kernels.
#pragma once

#include <stdint.h>

#include "pgd_gb300.h"

// First index i in [0, len) with a[i] >= x (len if none); a sorted ascending.
__device__ __forceinline__ int pgd_lower_bound(const int32_t *a, int len, int32_t x) {
    int lo = 0, hi = len;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ bool pgd_contains(const int32_t *a, int len, int32_t x) {
    int i = pgd_lower_bound(a, len, x);
    return i < len && a[i] == x;
}

__device__ __forceinline__ unsigned long long pgd_warp_sum(unsigned long long x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

__device__ __forceinline__ int pgd_warp_incl_scan(int x) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// Last row r in [lo, hi) with off[r] <= p, by the whole warp (the same for all lanes).
__device__ __forceinline__ int64_t pgd_warp_row(const int64_t *off, int64_t lo, int64_t hi, int64_t p, int lane) {
    while (hi - lo > 1) {
        const int64_t step = (hi - lo + 31) / 32;
        const int64_t at = min(lo + (lane + 1) * step, hi);
        const int k = __popc(__ballot_sync(0xffffffffu, at < hi && __ldg(off + at) <= p));
        const int64_t nlo = lo + k * step;
        hi = min(nlo + step, hi);
        lo = nlo;
    }
    return lo;
}

// Row of slot p, one of a warp's consecutive slots p0..p1: the rows of p0 and p1
// are found by searches of the whole warp, p's by a short one between them.  All
// lanes call.
__device__ __forceinline__ int64_t pgd_slot_row(const int64_t *off, int64_t n, int64_t p0, int64_t p1, int64_t p,
                                                int lane) {
    int64_t lo = pgd_warp_row(off, 0, n, p0, lane), hi = lo + 1;
    if (off[hi] <= p1) hi = pgd_warp_row(off, lo, n, p1, lane) + 1;
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (off[mid] <= p) lo = mid;
        else hi = mid;
    }
    return lo;
}

// First entry of each row above the diagonal, and how many there are (0 for row N).
static __global__ void pgd_upper_rows(const int64_t *off, const int32_t *adj, int64_t N, uint32_t *first,
                                      uint32_t *count) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v <= N; v += (int64_t)gridDim.x * blockDim.x) {
        uint32_t c = 0;
        if (v < N) {
            const int64_t o = off[v];
            const int d = (int)(off[v + 1] - o);
            const int at = pgd_lower_bound(adj + o, d, (int32_t)v);
            first[v] = (uint32_t)(o + at);
            c = (uint32_t)(d - at);
        }
        count[v] = c;
    }
}

// Ascending bitonic sort of P words in shared memory (P a power of two, at least
// 64) by the whole block.  Exchanges at most 32 apart stay within the 64 words of
// a warp's turn, so only the wider ones meet at the block's barrier.
__device__ __forceinline__ void pgd_block_sort(uint64_t *w, int P) {
    for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < (P >> 1); i += blockDim.x) {
                const int lo = ((i & ~(stride - 1)) << 1) | (i & (stride - 1)), hi = lo + stride;
                const uint64_t x = w[lo], y = w[hi];
                if ((x > y) == ((lo & size) == 0)) {
                    w[lo] = y;
                    w[hi] = x;
                }
            }
            // the next exchange is block-wide after this one, or the first of a larger size
            if (stride > 32 || (stride == 1 && size >= 64)) __syncthreads();
            else __syncwarp();
        }
    }
    __syncthreads();
}

// Exclusive prefix sum over a block of up to 1024 threads; *total gets the sum.
// sh: 33 words.  All threads call.
__device__ __forceinline__ int pgd_block_excl_scan(int x, int *sh, int *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    const int incl = pgd_warp_incl_scan(x);
    if (lane == 31) sh[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        const int v = lane < nw ? sh[lane] : 0;
        const int s = pgd_warp_incl_scan(v);
        sh[lane] = s - v;
        if (lane == 31) sh[32] = s;
    }
    __syncthreads();
    const int r = sh[wid] + incl - x;
    *total = sh[32];
    __syncthreads();
    return r;
}

// Graphs of at most this many pairs and vertices are built, ordered and ranked by
// one block per stage, with their sorts in shared memory: what bounds them is the
// number of launches and waits, not the work.  Build, order and counts of
// G(96, 0.06) take 145 us against 270 us with the grid-wide stages; 2,048 pairs of
// 300 vertices 230 us against 320 us for 2,049; 2,048 of 8,192 vertices 307 us
// against 381 us for 8,193.  At 4,096 pairs one SM sorts as long as the launches
// take (369 against 347 us), so the line lies below that.
constexpr int64_t kSmallPairs = 2048;
constexpr int64_t kSmallVertices = 8192;
constexpr int kSmallThreads = 1024;
inline int pgd_small_words(int64_t n) {   // words of a sort of n
    int p = 64;
    while (p < n) p <<= 1;
    return p;
}

// (unsigned long long)(x / 2.0) as the reference computes it: conversion to
// double (round to nearest), scale, truncate.  Below 2^53 the conversion and
// the halving are exact, so the result is x >> 1; only larger x take the
// double path (FP64 is slow on this part, and every edge needs several).
__device__ __forceinline__ unsigned long long pgd_half_d(unsigned long long x) {
    if ((x >> 53) == 0) return x >> 1;
    return __double2ull_rz(__dmul_rn(__ull2double_rn(x), 0.5));
}

// Per-edge closed forms of solve_graphlet_equations (graphlet_core.cpp:
// 1326-1364), added into the 15 partial sums.  Types as in the reference:
// degrees signed 64-bit, t and the sums unsigned 64-bit.
__device__ __forceinline__ void pgd_edge_sums(unsigned long long *s, long long dv, long long du,
                                              unsigned long long t, long long m, long long n) {
    typedef unsigned long long ull;
    ull star = (ull)dv - t - 1;
    star = star + (ull)du - t - 1;
    const ull disc = (ull)n - (star + t) - 2;
    const ull sv = (ull)dv - t - 1, su = (ull)du - t - 1;
    s[0] += t;
    s[1] += star;
    s[2] += disc;
    s[5] += pgd_half_d((t + star) * (t + star - 1));      // N1
    s[6] += pgd_half_d(star * (star - 1));                // N2
    s[7] += pgd_half_d(t * (t - 1));                      // N3
    s[8] += t * star;                                     // N4
    s[9] += sv * su;                                      // N5
    s[10] += (sv * (sv - 1)) / 2 + (su * (su - 1)) / 2;   // N6
    s[11] += (ull)(m - dv - du + 1);                      // N7
    s[12] += pgd_half_d(disc * (disc - 1));               // N8
    s[13] += star * disc;                                 // N9
    s[14] += t * disc;                                    // N10
}

// Column c of the per-edge output row (micro stores graphlet_core.cpp:
// 1559-1575 and the 2-star of the writer, graphlet_core.h:353-355).
__device__ __forceinline__ unsigned long long pgd_micro_col(int c, long long dv, long long du,
                                                           unsigned long long t, unsigned long long k4,
                                                           unsigned long long c4) {
    typedef unsigned long long ull;
    const long long sv = dv - (long long)t - 1, su = du - (long long)t - 1;
    switch (c) {
    case 0: return t;
    case 1: return ((ull)dv - t) + ((ull)du - t) - 2;
    case 2: return k4;
    case 3: {
        // (ull)((double)(t(t-1)) * 0.5 - (double)k4): exact below 2^53
        const ull tt = t * (t - 1);
        if ((tt >> 53) == 0 && (k4 >> 53) == 0) return (tt >> 1) - k4;
        return __double2ull_rz(__dsub_rn(__dmul_rn(__ull2double_rn(tt), 0.5), __ull2double_rn(k4)));
    }
    case 4: return 0;  // local_4_tailed_tris is never written (graphlet_core.cpp:1501)
    case 5: return c4;
    case 6: {
        // (ull)((double)a + (double)(su(su-1)) * 0.5), a = (ull)((double)(sv(sv-1)) * 0.5):
        // exact while every operand and the sum stay below 2^53
        const long long pv = sv * (sv - 1), pu = su * (su - 1);
        const long long lim = 1ll << 53;
        if (pv >= 0 && pv < lim && pu >= 0 && pu < lim) {
            const ull a = (ull)pv >> 1, b = (ull)pu >> 1;
            if (((a + b) >> 53) == 0) return a + b;
        }
        ull a = __double2ull_rz(__dmul_rn(__ll2double_rn(pv), 0.5));
        return __double2ull_rz(__dadd_rn(__ull2double_rn(a), __dmul_rn(__ll2double_rn(pu), 0.5)));
    }
    default: return (ull)(sv * su) - c4;
    }
}
