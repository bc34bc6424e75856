// size_rules.h -- choices by size that host code makes before a launch: plain
// functions of numbers, so that tests reach sizes that no graph of theirs has.
#pragma once

#include <math.h>
#include <stdint.h>

inline int pgd_bit_length(uint64_t x) {
    int b = 0;
    while (x) { b++; x >>= 1; }
    return b;
}

// Bits of an id in a packed (row, column) word: ids up to max_id (-1: none), and
// max_id + 1 for the row of what sorts behind every edge.  At most 32: two fit a word.
inline int pgd_id_bits(int64_t max_id) {
    const int b = pgd_bit_length((uint64_t)(max_id + 1));
    return b > 0 ? b : 1;
}

// k-core: by one block or a cluster of sixteen in one launch, or by steps of the
// whole device.  The cluster saves a captured graph (0.33 ms with its read-backs)
// and 3 us a step, and has a tenth of the device's bandwidth: about 65 ps more per
// row entry, and three quarters of that per vertex scanned.  A step of 46,000
// entries costs the same on both; the line lies lower because steps may widen
// again (a random graph of 65,536 vertices and 16.7 M entries 1.55 ms at 16,000,
// 2.2 ms from 24,000 on, 1.56 ms without the cluster).
constexpr int64_t kCoreLightWeight = 6000000;   // entries and vertices that cost what the captured graph does
constexpr int64_t kCoreNarrowWeight = 16000;    // entries and vertices of a narrow step, on average
constexpr int64_t kCoreIndexRoom = 1 << 16;     // vertices are counted in 32 bits, with strides of at most this

inline bool pgd_core_fits(int64_t n) { return n <= 0x7fffffffll - kCoreIndexRoom; }

// Graphs that the cluster takes from the start.  Milliseconds, cluster / device, on
// both sides of the line: G(n, p) of 2^18 vertices with 5.24 M entries 1.04 / 1.13,
// 6.29 M 1.10 / 0.94; of 2^20 with 4.19 M 1.07 / 1.18, 7.34 M 1.60 / 1.30; half a
// million pairs among 4 M vertices 1.03 / 1.27, among 16 M 4.08 / 3.47.
inline bool pgd_core_light(int64_t n, int64_t entries) {
    return pgd_core_fits(n) && entries + n / 4 * 3 <= kCoreLightWeight;
}

// Whether `steps` steps of the whole device, which scanned and removed so many
// vertices, were narrow: the cluster then takes the rest.  Milliseconds, device
// alone / with the cluster: R-MAT 20 13.5 / 9.1, R-MAT 22 with 2 edges per vertex
// 7.1 / 5.5, a 2000 x 2000 grid 11.2 / 9.0, geometric graphs of 500,000 vertices
// and degree 60 and 100 10.2 / 9.7 and 15.8 / 14.7, BA of 400,000 2.85 / 2.20; a
// random graph of 1M vertices and degree 50 and other wide ones stay: 2.46 / 2.46
// (5.4 in the cluster from the start).
inline bool pgd_core_narrow(int64_t n, int64_t entries, int64_t steps, int64_t scanned, int64_t removed) {
    return pgd_core_fits(n) &&
           0.75 * (double)scanned + (double)removed * ((double)entries / (double)n) <= (double)(steps * kCoreNarrowWeight);
}

// Whether a batch decomposes a graph with whole adjacency rows as bits and a
// common-neighbour matrix: at most dense_max vertices, average degree at least n/16.
inline bool pgd_dense_member(int64_t n, int64_t m, int dense_max) { return m > 0 && n <= dense_max && 32 * m >= n * n; }

// Whether k of a graph's m edges are decomposed edge by edge (decompose.cu), or by
// the passes over the whole graph (rank_path.cu), whose cost hardly depends on k.
//
// Below 1/2048 of the edges always edge by edge: microseconds for order and counts
// of 1/10000 of RMAT-20 27447 edge by edge, 32621 by the passes.  From there on the
// passes, edge by edge against whole-graph for 1/2000, 1/500 and 1/66 of the edges:
// RMAT-16 2151, 2298, 2609 / 699, 702, 771; RMAT-20 39110, 55900, 83642 / 32673,
// 32721, 32978; 1M-vertex BA 3257, 3452, 3909 / 1315, 1334, 1422; rgg-20 4345, 4368,
// 4714 / 3333, 3336, 3466.
//
// Dense graphs (average degree d at least 0.15 n) are the exception: their passes
// are bound by the triangles, of which there are about m d p / 3 with p = d / n, at
// 20 + d / 60 ps each; edge by edge it is 1.4 ps for each of the m d list entries of
// the triangle pass, 2.6 ps for those of the anchors met (k edges meet 1 - exp(-k/n)
// of n), and 38 ps for those of the sampled edges.  Microseconds edge by edge /
// whole-graph, G(1000, 0.5): 1/2048 638 / 950, 1/256 882 / 961, 1/64 1120 / 947;
// G(1000, 0.9): 1/2048 1259 / 3427, 1/16 2785 / 3479, 1/4 4763 / 3546; G(2000, 0.5):
// 1/64 4917 / 5179, 1/16 6033 / 5243; G(3000, 0.5): 1/16 20374 / 27159, 1/8 28133 /
// 27304; G(5000, 0.2): 1/2048 5602 / 7344, 1/512 8760 / 7396; G(250, 0.9) and
// G(1000, 0.25): the passes at any share from 1/2048.
inline bool pgd_sample_edgewise(int64_t n, int64_t m, int64_t k) {
    if (k < m / 2048) return true;
    if (k > m / 4) return false;
    const double d = 2.0 * (double)m / (double)n, p = d / (double)n, md = (double)m * d;
    if (!(p >= 0.15)) return false;
    const double f = 1.0 - exp(-(double)k / (double)n), share = (double)k / (double)m;
    const double edgewise = 300.0 + 1e-6 * md * (1.4 + 2.6 * f + 38.0 * share);
    const double whole = 150.0 + 1e-6 * md * p / 3.0 * (20.0 + d / 60.0);
    return edgewise < whole;
}
