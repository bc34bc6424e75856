// rank_path.cu -- per-edge graphlet counts of sparse graphs in degree-rank
// order: triangles and 4-cliques from each vertex's up-neighbourhood, 4-cycles
// from wedges whose highest-ranked vertex is an end.
//
// Replaces the OpenMP edge loop of graphlet_decomposition[_micro]
// (graphlet_core.cpp:1408-1424 and :1549-1577) with its helpers
// triangles_and_wedges / cycle / clique (:1069-1240).  That loop rescans the
// neighbourhoods of both ends for every edge; here every triangle, 4-clique
// and wedge is met once (the wedges twice) and credited to its edges.
//
// Vertices are renumbered by (degree descending, id descending); a row lists
// its neighbours' ranks in ascending order, so its first entries N+(x) are the
// neighbours above x.  With T(e) the common neighbours of an edge e's ends,
// t = |T|, k4 the edges inside T, and c4 the induced 4-cycles through e:
//   * triangles {a, x, y}, a the lowest: y in N+(a) n N+(x).  Pass 1 adds one to
//     t of the three edges.  Pass 2 repeats it with the adjacency F of N+(a) as
//     a bit matrix: |F_x & F_y| is the number of 4-cliques {a, z, x, y}, each
//     credited to its six edges, and the other two edges' t go to
//       D(e) = sum over w in T(e) of t of the edges from w to e's two ends.
//   * 4-cycles: the top vertex u of a cycle meets its opposite w through
//     wedges u - v - w with v and w below u.  For each u a counter per w counts
//     them; a second walk adds count(w) - 1 to edges (u, v) and (v, w).  That
//     gives C4(e), the 4-cycles through e with or without chords, and
//       c4 = C4 - D + 2 t + 2 k4
//     (a cycle p, q, w, x through e = (p, q) has the chord (p, w) iff w is in
//     T, of which there are sum_T (t(w, p) - 1), likewise for x and q, and both
//     chords 2 k4 times).
// t, k4 and c4 are at most m < 2^31, and everything else is used modulo 2^32,
// so all partial results are 32-bit.
//
// The numbers on R-MAT scale 20 (15.7 M edges): 5.65e9 wedges, 4.4e9 list
// entries probed per triangle pass, 4.2e8 triangles -- against 4.6e10 histogram
// entries and 9e10 list entries and bitmap words for the per-edge method of
// decompose.cu, which stays for small samples of the edges and for the
// allocation-free entry point.
#include <stddef.h>

#include <algorithm>
#include <cub/cub.cuh>

#include "pgd_kernels.cuh"
#include "rank_path.h"

namespace {

constexpr int kThreads = 256;
constexpr uint32_t kFull = 0xffffffffu;

inline int grid_for(int64_t n, int per_block = kThreads, int cap = 1 << 20) {
    int64_t g = (n + per_block - 1) / per_block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

inline int bits_for(int64_t x) {   // bits that hold every value below x (at least one)
    int b = 1;
    while (b < 63 && (int64_t(1) << b) < x) b++;
    return b;
}

// ---------------------------------------------------------------------------
// work classes

enum {
    kEgoWarp = 0,    // |N+(a)| in [2, 32]: a warp per vertex
    kEgoA,           // (32, 256]
    kEgoB,           // (256, 512]
    kEgoC,           // (512, 1024]
    kEgoGlobal,      // beyond: the tables in global memory
    kCycWarp,        // 2 .. kCycWarpMax wedges: a warp per vertex
    kCycHash,        // .. kCycHashMax wedges: a block per vertex, hashed counters
    kClasses         // more wedges: items of k_cycle_direct
};
constexpr int kEgoWarpMax = 32, kEgoAMax = 256, kEgoBMax = 512, kEgoCMax = 1024;
constexpr int kEgoMax[] = {kEgoWarpMax, kEgoAMax, kEgoBMax, kEgoCMax};
constexpr int kCycWarpMax = 512;
constexpr int kCycHashMax = 4096;
constexpr int kMaxRanges = 8192;
constexpr int64_t kKeepBytes = 16ll << 30;     // largest bound of the triangle lists kept between the passes
constexpr int64_t kTableBytes = 8ll << 30;     // largest lists and tables of the blocks of kEgoGlobal
constexpr int64_t kListFloor = 256ll << 20;    // lists and tables that are taken without asking for the room (about what
                                               // the edge-by-edge kernels take)
constexpr int64_t kBposBytes = 4ll << 30;      // largest table of range boundaries per row
constexpr uint32_t kDirectWords = 50 * 1024;   // counter words of one item: 200 KB of shared memory

// Sizes found on the device while the graph is built.
struct RankMeta {
    uint32_t tier[6];        // ranks below tier[i] have degree >= 65536, 256, 16, 4, 2, 1
    uint32_t tcode[5];       // bit address at which tier i + 1 ends (counter widths 32, 16, 8, 4, 2)
    uint32_t max_up;
    uint32_t nlist[kClasses];
    unsigned long long direct_wedges;   // wedges of the vertices beyond the lists
    unsigned long long pairs;           // sum of |N+(a)| (|N+(a)| - 1) / 2
    uint32_t bound[kMaxRanges + 1];   // range boundaries (ranks); not there where no vertex has items
};
constexpr size_t kMetaHead = offsetof(RankMeta, bound);
static_assert(kMetaHead <= kPinBytes, "the sizes fit the read-back buffer");

// Bit address of the counter of rank r.  A counter of w never exceeds deg(w):
// 32, 16, 8, 4 or 2 bits by degree (wide ones first, so none straddles a word).
__device__ __forceinline__ uint32_t code_of(const RankMeta *M, uint32_t r) {
    uint32_t lo = 0, c = 0;
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const uint32_t hi = M->tier[i];
        if (r < hi) return c + ((r - lo) << (5 - i));
        lo = hi;
        c = M->tcode[i];
    }
    return c;
}

__device__ __forceinline__ uint32_t mask_of(const RankMeta *M, uint32_t code) {
    if (code >= M->tcode[2]) return code < M->tcode[3] ? 0xfu : 0x3u;
    if (code >= M->tcode[1]) return 0xffu;
    return code >= M->tcode[0] ? 0xffffu : 0xffffffffu;
}

__device__ __forceinline__ uint32_t lower_bound_u(const int32_t *a, uint32_t lo, uint32_t hi, int32_t x) {
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (__ldg(a + mid) < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// First lane whose inclusive prefix exceeds it (all 32 lanes call).
__device__ __forceinline__ int owner_of(int incl, int it) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const int pre = __shfl_sync(kFull, incl, lo + step - 1);
        if (pre <= it) lo += step;
    }
    return lo;
}

// The rows of a warp's lanes (len entries each, possibly none) end to end: their
// entries are taken 32 at a time, in order.  A row is known by its place among
// those with entries, so that the owner of an entry follows from one OR of the
// starts that fall into the 32 and a popcount, not from a 5-step search by
// shuffles (a tenth of R-MAT 17's edges 2.53 -> 2.46 ms, a geometric graph of 1M
// vertices 10.46 -> 10.34 ms, rows included).
struct FlatRows {
    int start, place, total;   // first entry and place of this lane's row; entries in all
    int before = 0;            // rows begun before the entries taken next
    bool some;
    __device__ __forceinline__ FlatRows(int len, int lane) {
        const int incl = pgd_warp_incl_scan(len);
        total = __shfl_sync(kFull, incl, 31);
        start = incl - len;
        some = len > 0;
        place = __popc(__ballot_sync(kFull, some) & ((1u << lane) - 1));
    }
    // place of the row of entry b + lane; call with b = 0, 32, 64, ...
    __device__ __forceinline__ int owner(int b, int lane) {
        const uint32_t p = (uint32_t)(start - b);
        const uint32_t starts = __reduce_or_sync(kFull, some && p < 32 ? 1u << p : 0u);
        const int own = before + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
        before += __popc(starts);
        return own;
    }
};

// Row of each slot p = p0 + lane of one warp (lanes with p >= nnz get a valid
// row too).  Rows without entries come last in rank order, so 32 consecutive
// slots span at most 32 rows: one 32-way search finds the first, a 5-step
// search over the next row ends the rest.
__device__ __forceinline__ int rows_of_warp(const uint32_t *roff, int64_t n, uint32_t p0, uint32_t p, int lane) {
    int64_t lo = 0, hi = n;   // roff[lo] <= p0 < roff[hi]
    while (hi - lo > 1) {
        const int64_t step = (hi - lo + 31) / 32;
        const int64_t at = min(lo + (lane + 1) * step, hi);
        const unsigned m = __ballot_sync(kFull, at < hi && __ldg(roff + at) <= p0);
        const int k = __popc(m);
        const int64_t nlo = lo + k * step;
        hi = min(nlo + step, hi);
        lo = nlo;
    }
    const uint32_t end = __ldg(roff + min(lo + 1 + lane, n));
    const int own = owner_of((int)min(end - p0, 0x7fffffffu), (int)(p - p0));
    return (int)min(lo + own, n - 1);
}

// ---------------------------------------------------------------------------
// building

// Sort keys of the ranks; also clears the sizes.
__global__ void k_rank_keys2(const int32_t *deg, const int32_t *vgraph, const uint8_t *vmask, int64_t n,
                             int32_t max_degree, int vb, uint64_t *keys, RankMeta *M) {
    if (blockIdx.x == 0 && threadIdx.x < 6) M->tier[threadIdx.x] = 0;
    if (blockIdx.x == 0 && threadIdx.x < kClasses) M->nlist[threadIdx.x] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        M->max_up = 0;
        M->direct_wedges = 0;
        M->pairs = 0;
    }
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t d = vmask && vmask[vgraph[v]] ? 0 : deg[v];
        keys[v] = ((uint64_t)(uint32_t)(max_degree - d) << vb) | (uint64_t)(n - 1 - v);
    }
}

// Ranks from the sorted keys, the degree tiers (where the degree falls below a
// tier's), and zeroes for what k_rank_slots and k_rank_wedges fill.
__global__ void k_rank_scatter2(const uint64_t *sorted, int64_t n, int32_t max_degree, int vb, int32_t *vrank,
                                int32_t *rv, uint32_t *rdeg, int32_t *rup, uint32_t *bend, uint32_t *wd, RankMeta *M) {
    constexpr uint32_t lim[6] = {65536, 256, 16, 4, 2, 1};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x) {
        if (i == n) {
            rdeg[n] = 0;
            continue;
        }
        const uint64_t k = sorted[i];
        const int32_t v = (int32_t)(n - 1 - (int64_t)(k & ((1ull << vb) - 1)));
        const uint32_t d = (uint32_t)(max_degree - (int32_t)(k >> vb));
        const uint32_t dn = i + 1 < n ? (uint32_t)(max_degree - (int32_t)(sorted[i + 1] >> vb)) : 0;
        vrank[v] = (int32_t)i;
        rv[i] = v;
        rdeg[i] = d;
        rup[i] = 0;
        bend[i] = 0;
        wd[i] = 0;
#pragma unroll
        for (int t = 0; t < 6; t++)
            if (d >= lim[t] && dn < lim[t]) M->tier[t] = (uint32_t)i + 1;
    }
}

// The entries in rank order of their row, each as (rank of the neighbour, rank
// of the row): stably sorted by the first, the second ones are the rows of the
// rank-ordered graph, ascending.
__global__ void k_rank_entries(const uint32_t *roff, const int32_t *rv, const int64_t *off, const int32_t *adj,
                               const int32_t *vrank, int64_t n, int64_t nnz, uint32_t *key, int32_t *val) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; p0 < nnz; p0 += stride) {
        const int64_t p = min(p0 + lane, nnz - 1);
        const int r = rows_of_warp(roff, n, (uint32_t)p0, (uint32_t)p, lane);
        if (p0 + lane < nnz) {
            key[p] = (uint32_t)vrank[adj[off[rv[r]] + (p - (int64_t)roff[r])]];
            val[p] = r;
        }
    }
}

// Range boundaries: `ranges` parts of about equal weight, a rank's weight being
// half its share of the entries and half its share of the counter bits (so a
// range holds at most 2 / ranges of the bits).
__global__ void k_rank_bounds(const uint32_t *roff, int ranges, RankMeta *M) {
    const uint32_t n2 = M->tier[4];
    const double fe = 0.5 / (double)max(1u, roff[n2]), fb = 0.5 / (double)max(1u, M->tcode[4]);
    for (int k = threadIdx.x; k <= ranges; k += blockDim.x) {
        const double want = (double)k / ranges;
        uint32_t lo = 0, hi = n2;   // first rank whose prefix weight reaches want
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            if (fe * roff[mid] + fb * code_of(M, mid) < want) lo = mid + 1;
            else hi = mid;
        }
        M->bound[k] = k == 0 ? 0 : (k == ranges ? n2 : lo);
    }
}

// Per slot: the entry's counter address; the row's count of entries above it and
// its first entry of degree 1 (those come last); and, from the side of the lower
// end, the slots of the two directions.
__global__ void k_rank_slots(const uint32_t *roff, const int32_t *radj, int64_t n, int64_t nnz, RankMeta *M,
                             uint32_t *wcode, uint32_t *tw, int32_t *rup, uint32_t *bend) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // where each tier's counters end, from the tiers (then kept for the others)
    uint32_t lo[6], end[6];
    lo[0] = end[0] = 0;
#pragma unroll
    for (int i = 0; i < 5; i++) {
        lo[i + 1] = M->tier[i];
        end[i + 1] = end[i] + ((lo[i + 1] - lo[i]) << (5 - i));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
#pragma unroll
        for (int i = 0; i < 5; i++) M->tcode[i] = end[i + 1];
    const int32_t n2 = (int32_t)lo[5];
    for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; p0 < nnz; p0 += stride) {
        const int64_t p = min(p0 + lane, nnz - 1);
        const int r = rows_of_warp(roff, n, (uint32_t)p0, (uint32_t)p, lane);
        if (p0 + lane >= nnz) continue;
        const int32_t x = radj[p];
        uint32_t c = end[5];
#pragma unroll
        for (int i = 4; i >= 0; i--)
            if ((uint32_t)x < lo[i + 1]) c = end[i] + (((uint32_t)x - lo[i]) << (5 - i));
        wcode[p] = c;
        const bool first = p == (int64_t)roff[r], last = p + 1 == (int64_t)roff[r + 1];
        if (x >= n2 ? first || radj[p - 1] < n2 : last) bend[r] = (uint32_t)(x >= n2 ? p : p + 1);
        if (x < r) {
            const uint32_t s = lower_bound_u(radj, roff[x], roff[x + 1], r);
            tw[p] = s;
            tw[s] = (uint32_t)p;
            if (last || radj[p + 1] > r) {
                const uint32_t up = (uint32_t)p + 1 - roff[r];
                rup[r] = (int32_t)up;
                if (up > 32) atomicMax(&M->max_up, up);
            }
        }
    }
}

__global__ void k_rank_eslot(const int32_t *ev, const int32_t *eu, const int32_t *vrank, const uint32_t *roff,
                             const int32_t *rup, const int32_t *radj, const int32_t *vgraph, const uint8_t *vmask,
                             int64_t m, uint32_t *eslot) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = ev[e];
        if (vmask && vmask[vgraph[v]]) {
            eslot[e] = kFull;   // not read
            continue;
        }
        const int32_t a = vrank[v], b = vrank[eu[e]];
        const int32_t r = max(a, b), x = min(a, b);
        eslot[e] = lower_bound_u(radj, roff[r], roff[r] + (uint32_t)rup[r], x);
    }
}

// First entry of each row at or beyond each inner range boundary.
__global__ void k_rank_bpos(const uint32_t *roff, const int32_t *radj, int n2, int ranges, const RankMeta *M,
                            uint32_t *bpos) {
    const int64_t total = (int64_t)n2 * (ranges - 1);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int k = 1 + (int)(i / n2), v = (int)(i % n2);
        bpos[i] = lower_bound_u(radj, roff[v], roff[v + 1], (int32_t)M->bound[k]);
    }
}

// Wedges of every top vertex u (its lower neighbours' entries below u), with
// one atomic per warp where its slots belong to one row.
__global__ void k_rank_wedges(const uint32_t *roff, const int32_t *radj, const uint32_t *tw, const uint32_t *bend,
                              int64_t n, const RankMeta *M, uint32_t *wd) {
    const int lane = threadIdx.x & 31;
    const int32_t n2 = (int32_t)M->tier[4];
    const int64_t nnz2 = roff[n2];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; p0 < nnz2; p0 += stride) {
        const int64_t p = min(p0 + lane, nnz2 - 1);
        const int u = rows_of_warp(roff, n, (uint32_t)p0, (uint32_t)p, lane);
        uint32_t c = 0;
        const int32_t v = radj[p];
        if (p0 + lane < nnz2 && v > u && v < n2) c = bend[v] - tw[p] - 1;
        const int u0 = __shfl_sync(kFull, u, 0);
        if (__all_sync(kFull, u == u0)) {
            c = __reduce_add_sync(kFull, c);
            if (lane == 0 && c) atomicAdd(wd + u, c);
        } else if (c) {
            atomicAdd(wd + u, c);
        }
    }
}

__device__ __forceinline__ void list_append(bool in, int32_t v, int32_t *list, uint32_t *count, int lane) {
    const unsigned m = __ballot_sync(kFull, in);
    if (!m) return;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(count, (uint32_t)__popc(m));
    at = __shfl_sync(kFull, at, 0);
    if (in) list[at + __popc(m & ((1u << lane) - 1))] = v;
}

// Every vertex into the lists of its classes, and a place for its triangles:
// hbase[a], with room for every pair of N+(a).
__global__ void k_rank_lists(const int32_t *rup, const uint32_t *wd, int64_t n, int32_t *lists,
                             unsigned long long *hbase, RankMeta *M) {
    const int lane = threadIdx.x & 31;
    const int32_t n2 = (int32_t)M->tier[4];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    unsigned long long direct = 0;
    for (int64_t x0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; x0 < n2; x0 += stride) {
        const int64_t x = x0 + lane;
        const int up = x < n2 ? rup[x] : 0;
        const uint32_t w = x < n2 ? wd[x] : 0;
        const int ec = up < 2 ? -1 : up <= kEgoMax[0] ? 0 : up <= kEgoMax[1] ? 1 : up <= kEgoMax[2] ? 2 : up <= kEgoMax[3] ? 3 : 4;
#pragma unroll
        for (int c = 0; c < kCycWarp; c++) list_append(ec == c, (int32_t)x, lists + (int64_t)c * n, &M->nlist[c], lane);
        list_append(w >= 2 && w <= kCycWarpMax, (int32_t)x, lists + (int64_t)kCycWarp * n, &M->nlist[kCycWarp], lane);
        list_append(w > kCycWarpMax && w <= kCycHashMax, (int32_t)x, lists + (int64_t)kCycHash * n, &M->nlist[kCycHash],
                    lane);
        if (w > kCycHashMax) direct += w;
        const unsigned long long pairs = (unsigned long long)up * (unsigned)(up - (up > 0)) / 2;
        unsigned long long incl = pairs;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        unsigned long long at = 0;
        if (lane == 31 && incl) at = atomicAdd(&M->pairs, incl);
        at = __shfl_sync(kFull, at, 31);
        if (x < n2) hbase[x] = at + incl - pairs;
    }
    direct = pgd_warp_sum(direct);
    if (lane == 0 && direct) atomicAdd(&M->direct_wedges, direct);
}

// The whole of the above for a graph of at most 2 kSmallPairs entries and
// kSmallVertices vertices, by one block: twelve launches of a few microseconds
// each become one.  Ids take 14 bits.
constexpr int kSmallIdBits = 14;
static_assert(kSmallVertices < 1 << kSmallIdBits, "ids of a small graph");

struct RankSmallArgs {
    const int64_t *off;
    const int32_t *adj, *deg, *ev, *eu;
    int n, nnz, m, max_degree;
    int pv, pe;               // words of the two sorts
    uint32_t *roff;
    int32_t *rup;
    uint32_t *bend;
    int32_t *radj;
    uint32_t *wcode;
    uint32_t *tw, *eslot;
    int32_t *lists;
    unsigned long long *hbase;
    uint32_t *wd;
    RankMeta *M, *host;       // the sizes, on the device and in page-locked memory
};
inline size_t rank_small_bytes(int n, int pv, int pe) {
    return (size_t)std::max(pv, pe) * 8 + ((size_t)n + 1) * 8 + (size_t)n * 2 + (size_t)pe * 2 + 16;
}

__global__ void __launch_bounds__(kSmallThreads) k_rank_small(RankSmallArgs A) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    __shared__ int sh[33];
    __shared__ uint32_t s_tier[6], s_code[6], s_n[kClasses], s_up, s_pairs;
    __shared__ unsigned int s_direct;
    constexpr uint32_t idm = (1u << kSmallIdBits) - 1;
    constexpr uint32_t lim[6] = {65536, 256, 16, 4, 2, 1};
    const int n = A.n, nnz = A.nnz, tid = threadIdx.x;
    uint64_t *w = (uint64_t *)s_dyn;
    uint32_t *roff = (uint32_t *)(w + max(A.pv, A.pe)), *wd = roff + n + 1;
    uint16_t *vr = (uint16_t *)(wd + n + 1), *rad = vr + n;
    if (tid < 6) s_tier[tid] = 0;
    if (tid < kClasses) s_n[tid] = 0;
    if (tid == 0) {
        s_up = s_pairs = 0;
        s_direct = 0;
        A.wd[n] = 0;
    }
    // ranks and degree tiers
    for (int v = tid; v < A.pv; v += kSmallThreads)
        w[v] = v < n ? ((uint64_t)(uint32_t)(A.max_degree - A.deg[v]) << kSmallIdBits) | (uint64_t)(n - 1 - v) : ~0ull;
    __syncthreads();
    pgd_block_sort(w, A.pv);
    for (int i = tid; i < n; i += kSmallThreads) {
        const uint32_t d = (uint32_t)(A.max_degree - (int)(w[i] >> kSmallIdBits));
        const uint32_t dn = i + 1 < n ? (uint32_t)(A.max_degree - (int)(w[i + 1] >> kSmallIdBits)) : 0;
        vr[n - 1 - (int)(w[i] & idm)] = (uint16_t)i;
        roff[i] = d;
        wd[i] = 0;
        A.rup[i] = 0;
        A.bend[i] = 0;
        A.wd[i] = 0;
#pragma unroll
        for (int t = 0; t < 6; t++)
            if (d >= lim[t] && dn < lim[t]) s_tier[t] = (uint32_t)i + 1;
    }
    __syncthreads();
    {   // row offsets: each thread a contiguous part
        const int per = (n + kSmallThreads - 1) / kSmallThreads, b0 = min(n, tid * per), b1 = min(n, b0 + per);
        int c = 0, total = 0;
        for (int i = b0; i < b1; i++) c += (int)roff[i];
        int at = pgd_block_excl_scan(c, sh, &total);
        for (int i = b0; i < b1; i++) {
            const int d = (int)roff[i];
            roff[i] = (uint32_t)at;
            A.roff[i] = (uint32_t)at;
            at += d;
        }
        if (tid == 0) {
            roff[n] = (uint32_t)total;
            A.roff[n] = (uint32_t)total;
            uint32_t c0 = 0, lo = 0;
            s_code[0] = 0;
            for (int t = 0; t < 5; t++) {
                c0 += (s_tier[t] - lo) << (5 - t);
                lo = s_tier[t];
                s_code[t + 1] = c0;
            }
        }
    }
    // rows in rank order
    for (int p = tid; p < A.pe; p += kSmallThreads) {
        uint64_t x = ~0ull;
        if (p < nnz) {
            int lo = 0, hi = n;   // last row with off <= p
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (A.off[mid] <= p) lo = mid;
                else hi = mid;
            }
            x = ((uint64_t)vr[lo] << kSmallIdBits) | vr[A.adj[p]];
        }
        w[p] = x;
    }
    __syncthreads();
    pgd_block_sort(w, A.pe);
    for (int p = tid; p < nnz; p += kSmallThreads) {
        const uint32_t x = (uint32_t)(w[p] & idm);
        rad[p] = (uint16_t)x;
        A.radj[p] = (int32_t)x;
    }
    __syncthreads();
    const uint32_t n2 = s_tier[4];
    auto find = [&](uint32_t r, uint32_t x) {   // slot of x in row r
        uint32_t lo = roff[r], hi = roff[r + 1];
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (rad[mid] < x) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    for (int p = tid; p < nnz; p += kSmallThreads) {
        const uint32_t r = (uint32_t)(w[p] >> kSmallIdBits), x = rad[p];
        uint32_t c = s_code[5];
#pragma unroll
        for (int i = 4; i >= 0; i--)
            if (x < s_tier[i]) c = s_code[i] + ((x - (i ? s_tier[i - 1] : 0)) << (5 - i));
        A.wcode[p] = c;
        const bool first = (uint32_t)p == roff[r], last = (uint32_t)p + 1 == roff[r + 1];
        if (x >= n2 ? first || rad[p - 1] < n2 : last) A.bend[r] = (uint32_t)(x >= n2 ? p : p + 1);
        if (x < r) {
            const uint32_t s = find(x, r);
            A.tw[p] = s;
            A.tw[s] = (uint32_t)p;
            if (last || rad[p + 1] > r) {
                const uint32_t up = (uint32_t)p + 1 - roff[r];
                A.rup[r] = (int32_t)up;
                atomicMax(&s_up, up);
            }
        }
    }
    for (int e = tid; e < A.m; e += kSmallThreads) {
        const uint32_t a = vr[A.ev[e]], b = vr[A.eu[e]];
        A.eslot[e] = find(max(a, b), min(a, b));
    }
    __syncthreads();
    // wedges below each vertex, and the lists
    for (int p = tid; p < nnz; p += kSmallThreads) {
        const uint32_t u = (uint32_t)(w[p] >> kSmallIdBits), v = rad[p];
        if (v > u && v < n2) atomicAdd(wd + u, A.bend[v] - A.tw[p] - 1);
    }
    __syncthreads();
    for (int x = tid; x < (int)n2; x += kSmallThreads) {
        const int up = A.rup[x];
        const uint32_t c = wd[x];
        const int ec = up < 2 ? -1 : up <= kEgoWarpMax ? 0 : up <= kEgoAMax ? 1 : up <= kEgoBMax ? 2 : up <= kEgoCMax ? 3 : 4;
        const int cc = c < 2 || c > kCycHashMax ? -1 : c <= kCycWarpMax ? (int)kCycWarp : (int)kCycHash;
        if (ec >= 0) A.lists[(int64_t)ec * n + atomicAdd(&s_n[ec], 1u)] = x;
        if (cc >= 0) A.lists[(int64_t)cc * n + atomicAdd(&s_n[cc], 1u)] = x;
        if (c > kCycHashMax) atomicAdd(&s_direct, c);
        A.hbase[x] = atomicAdd(&s_pairs, (uint32_t)up * (uint32_t)(up - (up > 0)) / 2);
        A.wd[x] = c;
    }
    __syncthreads();
    if (tid < 2) {
        RankMeta *M = tid ? A.host : A.M;
        for (int i = 0; i < 6; i++) M->tier[i] = s_tier[i];
        for (int i = 0; i < 5; i++) M->tcode[i] = s_code[i + 1];
        for (int i = 0; i < kClasses; i++) M->nlist[i] = s_n[i];
        M->max_up = s_up;
        M->direct_wedges = s_direct;
        M->pairs = s_pairs;
    }
}

// Ranges [k, end) of u's next item: as many as its counters and its share of
// the wedges allow (at least one).
__device__ __forceinline__ int next_piece(const RankMeta *M, uint32_t u, int k, int ranges, int per_item) {
    const uint32_t c0 = code_of(M, max(M->bound[k], u + 1)) & ~31u;
    int e = k + 1;
    while (e < ranges && e - k < per_item && (code_of(M, M->bound[e + 1]) - c0 + 31) / 32 <= kDirectWords) e++;
    return e;
}

// Items of the vertices with many wedges: mode 0 counts them per vertex, mode 1
// writes them.  A vertex whose wedges exceed a fixed part of all is split by
// ranges of the wedge's end, so that no item keeps one block busy to the end.
__global__ void k_rank_items(const uint32_t *wd, int n2, int ranges, const RankMeta *M, int parts,
                             uint32_t *count, const uint32_t *pos, int2 *items) {
    const unsigned long long target = max(65536ull, M->direct_wedges / (unsigned)parts);
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x <= n2; x += (int64_t)gridDim.x * blockDim.x) {
        uint32_t c = 0;
        if (x < n2 && wd[x] > kCycHashMax) {
            const uint32_t u = (uint32_t)x;
            int k = 0;   // first range that reaches beyond u
            while (k + 1 < ranges && M->bound[k + 1] <= u + 1) k++;
            const int split = (int)min((unsigned long long)(ranges - k), wd[x] / target + 1);
            const int per_item = (ranges - k + split - 1) / split;
            while (k < ranges) {
                const int e = next_piece(M, u, k, ranges, per_item);
                if (items) items[pos[x] + c] = make_int2((int)u, k | (e << 16));
                c++;
                k = e;
            }
        }
        if (count) count[x] = c;
    }
}

// ---------------------------------------------------------------------------
// 4-cycles

struct CycArgs {
    const uint32_t *roff;
    const int32_t *rup;
    const int32_t *radj;
    const uint32_t *wcode;
    const uint32_t *tw;
    const uint32_t *bend;
    const uint32_t *bpos;
    int n2;
    int ranges;
    const RankMeta *M;
    const int32_t *list;
    const int2 *items;
    uint32_t count;
    uint32_t grab;      // k_cycle_warp: vertices a warp takes at a time
    unsigned long long *next;
    uint32_t *cyc;      // per slot
};

// Shared scratch of a block's walk over the rows of up to NT middle vertices.
template <int NT>
struct Walk {
    int pre[NT];          // inclusive prefix sums of the rows' lengths
    uint32_t start[NT];   // first entry taken of each row
    uint32_t acc[NT];     // what the second walk found for (u, v)
    int wtot[NT / 32];
};

template <int NT>
__device__ __forceinline__ int walk_search(const int *pre, int i) {   // first t with pre[t] > i
    int lo = 0;
#pragma unroll
    for (int step = NT / 2; step > 0; step >>= 1)
        if (pre[lo + step - 1] <= i) lo += step;
    return lo;
}

// Applies fn(code, position) to every wedge end w of u: the rows of NT middle vertices v at a time are concatenated and every warp
// takes an equal contiguous share, so short and long rows keep all lanes busy.
// fn's results are added per v and, in the second walk (ACC), written to the
// slot u -> v.  All threads of the block call; returns behind a barrier.
template <int NT, bool ACC, typename Fn>
__device__ __forceinline__ void walk_wedges(const CycArgs &A, Walk<NT> &W, uint32_t u, Fn fn) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t j0 = A.roff[u] + (uint32_t)A.rup[u];
    const uint32_t j1 = A.bend[u];
    for (uint32_t c0 = j0; c0 < j1; c0 += NT) {
        const uint32_t j = c0 + threadIdx.x;
        int len = 0;
        uint32_t s0 = 0;
        if (j < j1) {
            const int32_t v = __ldg(A.radj + j);
            s0 = __ldg(A.tw + j) + 1;
            len = (int)(__ldg(A.bend + v) - s0);
        }
        const int incl = pgd_warp_incl_scan(len);
        if (lane == 31) W.wtot[wid] = incl;
        __syncthreads();
        const int wt = lane < NT / 32 ? W.wtot[lane] : 0;
        const int wincl = pgd_warp_incl_scan(wt);
        const int total = __shfl_sync(kFull, wincl, 31);
        W.pre[threadIdx.x] = __shfl_sync(kFull, wincl - wt, wid) + incl;
        W.start[threadIdx.x] = s0;
        if (ACC) W.acc[threadIdx.x] = 0;
        __syncthreads();
        const int share = (total + NT / 32 - 1) / (NT / 32);
        const int lo = min(total, wid * share), hi = min(total, lo + share);
        int base = lo < hi ? walk_search<NT>(W.pre, lo) : 0;
        for (int s = lo; s < hi;) {
            const int own_end = min(W.pre[base], hi);
            if (own_end - s >= 64) {
                // one row covers the next entries: straight, four per lane
                const uint32_t row0 = W.start[base] - (uint32_t)(base ? W.pre[base - 1] : 0);
                uint32_t a = 0;
                for (; s + 128 <= own_end; s += 128) {
                    const uint32_t q = row0 + (uint32_t)(s + lane);
                    const uint32_t w0 = __ldg(A.wcode + q), w1 = __ldg(A.wcode + q + 32), w2 = __ldg(A.wcode + q + 64),
                                   w3 = __ldg(A.wcode + q + 96);
                    a += fn(w0, q) + fn(w1, q + 32) + fn(w2, q + 64) + fn(w3, q + 96);
                }
                for (; s < own_end; s += 32) {
                    const uint32_t q = row0 + (uint32_t)(s + lane);
                    if (s + lane < own_end) a += fn(__ldg(A.wcode + q), q);
                }
                s = own_end;
                if (ACC) {
                    a = __reduce_add_sync(kFull, a);
                    if (lane == 0 && a) atomicAdd(&W.acc[base], a);
                }
                if (s < hi) base = walk_search<NT>(W.pre, s);
                continue;
            }
            const int cand = base + lane < NT ? W.pre[base + lane] : 0x7fffffff;
            const int last = __shfl_sync(kFull, cand, 31);
            const int iA = s + lane, iB = s + 32 + lane;
            const bool vA = iA < hi, vB = iB < hi;
            int ownA = base + owner_of(cand, iA), ownB = base + owner_of(cand, iB);
            if (vA && iA >= last) ownA = walk_search<NT>(W.pre, iA);
            if (vB && iB >= last) ownB = walk_search<NT>(W.pre, iB);
            uint32_t qA = 0, qB = 0, wA = 0, wB = 0;
            if (vA) {
                qA = W.start[ownA] + (uint32_t)(iA - (ownA ? W.pre[ownA - 1] : 0));
                wA = __ldg(A.wcode + qA);
            }
            if (vB) {
                qB = W.start[ownB] + (uint32_t)(iB - (ownB ? W.pre[ownB - 1] : 0));
                wB = __ldg(A.wcode + qB);
            }
            if (vA) {
                const uint32_t a = fn(wA, qA);
                if (ACC && a) atomicAdd(&W.acc[ownA], a);
            }
            if (vB) {
                const uint32_t a = fn(wB, qB);
                if (ACC && a) atomicAdd(&W.acc[ownB], a);
            }
            __syncwarp();
            s += 64;
            if (s < hi) base = min(__shfl_sync(kFull, ownB, 31), NT - 1);
        }
        __syncthreads();
        if (ACC && j < j1) {
            const uint32_t a = W.acc[threadIdx.x];
            if (a) atomicAdd(A.cyc + j, a);
        }
        __syncthreads();
    }
}

// Rows of vertices of degree >= kCoopRow are dealt to all warps of
// k_cycle_direct in pieces of 128 entries; of the others a warp takes about
// kGrabEntries entries at a time.
constexpr int kCoopRow = 4096;
constexpr int kGrabEntries = 4096;

// fn(code, position) over the entries p0 + lane, p0 + 32 + lane, ... below n of
// the 128 starting at s + p0, with their loads in flight together.
template <typename Fn>
__device__ __forceinline__ uint32_t take_128(const uint32_t *wcode, uint32_t s, int n, int p0, int lane, Fn fn) {
    const uint32_t q = s + (uint32_t)(p0 + lane);
    const uint32_t *w = wcode + q;
    const int left = n - p0 - lane;
    uint32_t a = 0;
    if (n - p0 >= 128) {
        const uint32_t w0 = __ldg(w), w1 = __ldg(w + 32), w2 = __ldg(w + 64), w3 = __ldg(w + 96);
        a = fn(w0, q) + fn(w1, q + 32) + fn(w2, q + 64) + fn(w3, q + 96);
    } else {
        uint32_t w0 = 0, w1 = 0, w2 = 0, w3 = 0;
        if (left > 0) w0 = __ldg(w);
        if (left > 32) w1 = __ldg(w + 32);
        if (left > 64) w2 = __ldg(w + 64);
        if (left > 96) w3 = __ldg(w + 96);
        if (left > 0) a += fn(w0, q);
        if (left > 32) a += fn(w1, q + 32);
        if (left > 64) a += fn(w2, q + 64);
        if (left > 96) a += fn(w3, q + 96);
    }
    return a;
}

// Applies fn(code, position) to every wedge end w of u in the ranges [k0, k1)
// and, in the second walk (ACC), adds its results per v to the slot u -> v.
// The rows of the middle vertices v come longest first.  The warps share the
// pieces of the longest rows in turn; then they take 1 to 32 rows at a time from
// a counter, rows of 64 or more entries one after the other, the rest flattened
// over the lanes.  No barrier inside: warps only meet between the two walks.
// (Sharing rows from 1,024 entries costs more turns than it balances: R-MAT 20
// 30.0 against 25.3 ms; one block-wide prefix sum per 1,024 rows with equal
// shares for the warps spent a third of its time at its barriers.)
template <int NT, bool ACC, typename Fn>
__device__ __forceinline__ void walk_rows(const CycArgs &A, uint32_t u, int k0, int k1, uint32_t *next, uint32_t *acc,
                                          Fn fn) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t j0 = A.roff[u] + (uint32_t)A.rup[u];
    const uint32_t j1 = A.bend[u];
    // the part of row radj[j] that ends wedges of u in the ranges: start and length
    auto row_of = [&](uint32_t j, uint32_t &s0) {
        const int32_t v = __ldg(A.radj + j);
        s0 = __ldg(A.tw + j) + 1;
        uint32_t e0 = __ldg(A.bend + v);
        if (A.bpos) {
            if (k1 < A.ranges) e0 = __ldg(A.bpos + (int64_t)(k1 - 1) * A.n2 + v);
            if (k0 > 0) s0 = max(s0, __ldg(A.bpos + (int64_t)(k0 - 1) * A.n2 + v));
        } else {
            if (k1 < A.ranges) e0 = lower_bound_u(A.radj, s0, max(s0, e0), (int32_t)A.M->bound[k1]);
            if (k0 > 0) s0 = lower_bound_u(A.radj, s0, max(s0, e0), (int32_t)A.M->bound[k0]);
        }
        return e0 > s0 ? (int)(e0 - s0) : 0;
    };
    int turn = wid;   // pieces of 128 until this warp's next one
    uint32_t jb = j0;
    for (; jb < j1; jb += 32) {
        const int32_t v0 = __ldg(A.radj + jb);   // the longest row left
        if (__ldg(A.roff + v0 + 1) - __ldg(A.roff + v0) < (uint32_t)kCoopRow) break;
        uint32_t s0 = 0;
        const int len = jb + lane < j1 ? row_of(jb + lane, s0) : 0;
        unsigned m = __ballot_sync(kFull, len > 0);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const uint32_t s = __shfl_sync(kFull, s0, src);
            const int n = __shfl_sync(kFull, len, src);
            const int pieces = (n + 127) >> 7;
            uint32_t a = 0;
            const bool any = turn < pieces;
            for (; turn < pieces; turn += NT / 32) a += take_128(A.wcode, s, n, turn << 7, lane, fn);
            turn -= pieces;
            if (ACC && any) {
                __syncwarp();
                a = __reduce_add_sync(kFull, a);
                if (lane == 0 && a) atomicAdd(A.cyc + jb + src, a);
            }
        }
    }
    uint32_t *off = acc + 32;
    uint32_t grab = 1;
    while (true) {
        uint32_t c0 = 0;
        if (lane == 0) c0 = atomicAdd(next, grab);
        c0 = __shfl_sync(kFull, c0, 0);
        if (jb >= j1 || c0 >= j1 - jb) break;
        c0 += jb;
        uint32_t s0 = 0;
        int len = (uint32_t)lane < grab && c0 + lane < j1 ? row_of(c0 + lane, s0) : 0;
        const uint32_t taken = grab;
        const int longest = __reduce_max_sync(kFull, len);   // the next rows are hardly longer
        grab = longest <= kGrabEntries / 32 ? 32 : max(1u, (uint32_t)(kGrabEntries / longest));
        uint32_t mine = 0;
        if (ACC) acc[lane] = 0;
        unsigned m = __ballot_sync(kFull, len >= 64);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const uint32_t s = __shfl_sync(kFull, s0, src);
            const int n = __shfl_sync(kFull, len, src);
            uint32_t a = 0;
            for (int p = 0; p < n; p += 128) a += take_128(A.wcode, s, n, p, lane, fn);
            if (ACC) {
                __syncwarp();
                a = __reduce_add_sync(kFull, a);
                if (lane == src) mine = a;
            }
        }
        if (len >= 64) len = 0;
        FlatRows F(len, lane);
        if (len) off[F.place] = s0 - (uint32_t)F.start;   // slot = off + flattened index
        __syncwarp();
        const int total = F.total;
        constexpr int kFly = 4;   // loads in flight (two: sample of R-MAT 17 2.46, now 2.44 ms)
        for (int b = 0; b < total; b += 32 * kFly) {
            int own[kFly];
            uint32_t q[kFly], w[kFly];
#pragma unroll
            for (int k = 0; k < kFly; k++) {
                own[k] = F.owner(b + 32 * k, lane);
                q[k] = off[own[k]] + (uint32_t)(b + 32 * k + lane);
                w[k] = b + 32 * k + lane < total ? __ldg(A.wcode + q[k]) : 0;
            }
#pragma unroll
            for (int k = 0; k < kFly; k++) {
                if (b + 32 * k + lane < total) {
                    const uint32_t a = fn(w[k], q[k]);
                    if (ACC && a) atomicAdd(acc + own[k], a);
                }
            }
            __syncwarp();
        }
        if (ACC) {
            __syncwarp();
            if (len) mine += acc[F.place];
            if ((uint32_t)lane < taken && c0 + lane < j1 && mine) atomicAdd(A.cyc + c0 + lane, mine);
            __syncwarp();
        }
    }
}

// Many wedges: one block per (u, ranges of w), a counter per w in shared
// memory at its bit address.  Graphs whose counters all fit in 100 or 50 KB run
// it with 2 or 4 smaller blocks per SM, which hide each other's barriers.
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_cycle_direct(CycArgs A) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    __shared__ uint32_t s_acc[NT / 32][64];   // a warp's sums and slots per row
    __shared__ uint32_t s_item, s_next[2];
    const RankMeta *M = A.M;
    uint32_t *acc = s_acc[threadIdx.x >> 5];
    while (true) {
        if (threadIdx.x == 0) {
            s_item = (uint32_t)atomicAdd(A.next, 1ull);
            s_next[0] = s_next[1] = 0;
        }
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= A.count) break;
        const int2 it = A.items[item];
        const uint32_t u = (uint32_t)it.x;
        const int k0 = it.y & 0xffff, k1 = it.y >> 16;
        const uint32_t first = code_of(M, max(M->bound[k0], u + 1)), end = code_of(M, M->bound[k1]);
        const uint32_t c0 = first & ~31u, words = (end - c0 + 31) / 32;
        for (uint32_t i = threadIdx.x; i < words; i += NT) s_dyn[i] = 0;
        // the item's counter widths: mostly two, below and from thr
        int tier = 0;
        while (tier < 4 && M->tcode[tier] <= first) tier++;
        const uint32_t thr = M->tcode[tier];
        const bool two = end <= thr || tier >= 3 || end <= M->tcode[tier + 1];
        const uint32_t mlo = mask_of(M, first), mhi = mask_of(M, thr);
        __syncthreads();
        walk_rows<NT, false>(A, u, k0, k1, &s_next[0], acc, [&](uint32_t c, uint32_t) {
            atomicAdd(s_dyn + ((c - c0) >> 5), 1u << (c & 31));
            return 0u;
        });
        __syncthreads();
        if (two) {
            walk_rows<NT, true>(A, u, k0, k1, &s_next[1], acc, [&](uint32_t c, uint32_t q) {
                const uint32_t k = ((s_dyn[(c - c0) >> 5] >> (c & 31)) & (c < thr ? mlo : mhi)) - 1;
                if (k) atomicAdd(A.cyc + q, k);
                return k;
            });
        } else {
            walk_rows<NT, true>(A, u, k0, k1, &s_next[1], acc, [&](uint32_t c, uint32_t q) {
                const uint32_t k = ((s_dyn[(c - c0) >> 5] >> (c & 31)) & mask_of(M, c)) - 1;
                if (k) atomicAdd(A.cyc + q, k);
                return k;
            });
        }
        __syncthreads();
    }
}

// Hashed counters: open addressing, at most half full.
__device__ __forceinline__ uint32_t hash_of(uint32_t key, int shift) { return (key * 0x9E3779B1u) >> shift; }

__device__ __forceinline__ uint32_t hash_find_add(uint32_t *keys, uint32_t key, uint32_t mask, int shift) {
    uint32_t h = hash_of(key, shift);
    while (true) {
        const uint32_t k = keys[h];
        if (k == key) return h;
        if (k == kFull) {
            const uint32_t old = atomicCAS(keys + h, kFull, key);
            if (old == kFull || old == key) return h;
        }
        h = (h + 1) & mask;
    }
}

__device__ __forceinline__ uint32_t hash_find(const uint32_t *keys, uint32_t key, uint32_t mask, int shift) {
    uint32_t h = hash_of(key, shift);
    while (keys[h] != key) h = (h + 1) & mask;   // the key is in the table
    return h;
}

constexpr int kHashThreads = 512;
constexpr int kHashSlots = 2 * kCycHashMax;
constexpr int kHashSmem = kHashSlots * 6 + (int)sizeof(Walk<kHashThreads>);

// A middling number of wedges: one block per u, hashed 16-bit counters (a
// counter holds at most kCycHashMax).
__global__ void __launch_bounds__(kHashThreads, 4) k_cycle_hash(CycArgs A) {
    constexpr int kSlots = kHashSlots;
    extern __shared__ __align__(16) uint32_t s_dyn[];
    uint32_t *s_key = s_dyn, *s_cnt = s_dyn + kSlots;
    Walk<kHashThreads> &W = *(Walk<kHashThreads> *)(s_dyn + kSlots + kSlots / 2);
    __shared__ uint32_t s_item;
    while (true) {
        if (threadIdx.x == 0) s_item = (uint32_t)atomicAdd(A.next, 1ull);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= A.count) break;
        const uint32_t u = (uint32_t)A.list[item];
        for (int i = threadIdx.x; i < kSlots; i += kHashThreads) s_key[i] = kFull;
        for (int i = threadIdx.x; i < kSlots / 2; i += kHashThreads) s_cnt[i] = 0;
        __syncthreads();
        constexpr int shift = 32 - 13;
        static_assert(kSlots == 1 << 13, "hash width");
        walk_wedges<kHashThreads, false>(A, W, u, [&](uint32_t c, uint32_t) {
            const uint32_t h = hash_find_add(s_key, c, kSlots - 1, shift);
            atomicAdd(s_cnt + (h >> 1), 1u << ((h & 1) << 4));
            return 0u;
        });
        walk_wedges<kHashThreads, true>(A, W, u, [&](uint32_t c, uint32_t q) {
            const uint32_t h = hash_find(s_key, c, kSlots - 1, shift);
            const uint32_t k = ((s_cnt[h >> 1] >> ((h & 1) << 4)) & 0xffffu) - 1;
            if (k) atomicAdd(A.cyc + q, k);
            return k;
        });
        __syncthreads();
    }
}

constexpr int kWarpThreads = 256;
constexpr int kWarpSlots = 2 * kCycWarpMax;
constexpr int kWarpWords = kWarpSlots + kWarpSlots / 2 + 64;   // keys, 16-bit counters, sums and slots per row
constexpr int kWarpSmem = kWarpThreads / 32 * kWarpWords * 4;
static_assert(kWarpSlots == 1 << 10, "largest table of a warp");

// Few wedges: one warp per u.
__global__ void __launch_bounds__(kWarpThreads) k_cycle_warp(CycArgs A) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t *key = s_dyn + wid * kWarpWords, *cnt = key + kWarpSlots, *acc = cnt + kWarpSlots / 2,
             *off = acc + 32;
    const uint32_t *bend = A.bend;
    while (true) {
        uint32_t i0 = 0;
        if (lane == 0) i0 = (uint32_t)atomicAdd(A.next, (unsigned long long)A.grab);
        i0 = __shfl_sync(kFull, i0, 0);
        if (i0 >= A.count) break;
        const uint32_t i1 = min(i0 + A.grab, A.count);
        for (uint32_t i = i0; i < i1; i++) {
            const uint32_t u = (uint32_t)A.list[i];
            const uint32_t j0 = A.roff[u] + (uint32_t)A.rup[u], j1 = bend[u];
            int bits = 0;   // log2 of the table's slots, 0 until the first rows are known
            for (int pass = 0; pass < 2; pass++) {
                for (uint32_t c0 = j0; c0 < j1; c0 += 32) {
                    const uint32_t j = c0 + lane;
                    int len = 0;
                    uint32_t s0 = 0;
                    if (j < j1) {
                        s0 = __ldg(A.tw + j) + 1;
                        len = (int)(__ldg(bend + __ldg(A.radj + j)) - s0);
                    }
                    FlatRows F(len, lane);
                    const int total = F.total;
                    if (!bits) {
                        // all wedges within these rows: a table twice their number, else the largest
                        bits = c0 + 32 >= j1 ? max(5, 33 - __clz(max(total, 2) - 1)) : 10;
                        for (int k = lane; k < (1 << bits); k += 32) key[k] = kFull;
                        for (int k = lane; k < (1 << bits) / 2; k += 32) cnt[k] = 0;
                    }
                    acc[lane] = 0;
                    if (F.some) off[F.place] = s0 - (uint32_t)F.start;   // slot = off + flattened index
                    __syncwarp();
                    const uint32_t mask = (1u << bits) - 1;
                    const int shift = 32 - bits;
                    for (int b = 0; b < total; b += 32) {
                        const int it = b + lane;
                        const int own = F.owner(b, lane);
                        if (it < total) {
                            const uint32_t q = off[own] + (uint32_t)it;
                            const uint32_t c = __ldg(A.wcode + q);
                            if (pass == 0) {
                                const uint32_t h = hash_find_add(key, c, mask, shift);
                                atomicAdd(cnt + (h >> 1), 1u << ((h & 1) << 4));
                            } else {
                                const uint32_t h = hash_find(key, c, mask, shift);
                                const uint32_t k = ((cnt[h >> 1] >> ((h & 1) << 4)) & 0xffffu) - 1;
                                if (k) {
                                    atomicAdd(A.cyc + q, k);
                                    atomicAdd(acc + own, k);
                                }
                            }
                        }
                    }
                    __syncwarp();
                    if (pass == 1 && F.some && acc[F.place]) atomicAdd(A.cyc + j, acc[F.place]);
                    __syncwarp();
                }
            }
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// triangles (pass 1) and 4-cliques with the sums of t (pass 2)

struct EgoArgs {
    const uint32_t *roff;
    const int32_t *rup;
    const int32_t *radj;
    const int32_t *list;
    uint32_t count;
    uint32_t grab;              // k_ego_warp: vertices a warp takes at a time
    unsigned long long *next;
    uint32_t *t;                // per slot of the lower end: triangles
    unsigned long long *dk;     // per slot of the lower end: D << 32 | k4
    uint2 *hits;                // triangles ({i << 16 | j, slot x -> y}): at hbase[a], or a list per block
    const unsigned long long *hbase;
    uint32_t *hcount;           // triangles of a, where they are kept from pass 1 to pass 2 (else null)
    int64_t hits_stride;
    uint8_t *tables;            // kEgoGlobal: tables of each block
    int64_t tables_stride;
};

// |N+(a)| = d <= 32: a warp per vertex.  The pairs (i, j), j < i, of N+(a) are
// dealt to the lanes; y = N+(a)[j] is searched in N+(x), x = N+(a)[i].
template <int PASS>
__global__ void __launch_bounds__(kWarpThreads) k_ego_warp(EgoArgs A) {
    constexpr int kPairs = 32 * 31 / 2;
    constexpr int kW = kWarpThreads / 32;
    __shared__ uint16_t s_pair[kPairs];
    __shared__ uint32_t s_a[kW][32], s_b[kW][32], s_f[kW][32], s_t[kW][32];
    __shared__ uint32_t s_slot[PASS == 2 ? kW : 1][PASS == 2 ? kPairs : 1];
    __shared__ uint16_t s_hit[PASS == 2 ? kW : 1][PASS == 2 ? kPairs : 1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int i = 1 + (int)threadIdx.x; i < 32; i += kWarpThreads)
        for (int j = 0; j < i; j++) s_pair[i * (i - 1) / 2 + j] = (uint16_t)(i << 8 | j);
    __syncthreads();
    uint32_t *ca = s_a[wid], *cb = s_b[wid], *f = s_f[wid], *ta = s_t[wid];
    while (true) {
        uint32_t i0 = 0;
        if (lane == 0) i0 = (uint32_t)atomicAdd(A.next, (unsigned long long)A.grab);
        i0 = __shfl_sync(kFull, i0, 0);
        if (i0 >= A.count) break;
        const uint32_t i1 = min(i0 + A.grab, A.count);
        for (uint32_t ii = i0; ii < i1; ii++) {
            const uint32_t a = (uint32_t)A.list[ii];
            const int d = A.rup[a];
            const uint32_t ra = A.roff[a];
            int32_t x = 0;
            uint32_t rx = 0;
            int ux = 0;
            if (lane < d) {
                x = __ldg(A.radj + ra + lane);
                rx = __ldg(A.roff + x);
                ux = __ldg(A.rup + x);
            }
            ca[lane] = 0;
            if (PASS == 2) {
                cb[lane] = 0;
                f[lane] = 0;
                ta[lane] = lane < d ? A.t[ra + lane] : 0;
            }
            __syncwarp();
            const int np = d * (d - 1) / 2;
            int nh = 0;
            const unsigned long long hb = PASS == 1 && A.hcount ? A.hbase[a] : 0;
            for (int b = 0; b < np; b += 32) {
                const bool act = b + lane < np;
                const int pr = act ? s_pair[b + lane] : 0x0100;
                const int i = pr >> 8, j = pr & 255;
                const int32_t y = __shfl_sync(kFull, x, j);
                const uint32_t r0 = __shfl_sync(kFull, rx, i);
                const int ui = __shfl_sync(kFull, ux, i);
                bool hit = false;
                uint32_t pos = 0;
                if (act) {
                    pos = lower_bound_u(A.radj, r0, r0 + (uint32_t)ui, y);
                    hit = pos < r0 + (uint32_t)ui && __ldg(A.radj + pos) == y;
                }
                if (PASS == 1) {
                    const unsigned m = A.hcount ? __ballot_sync(kFull, hit) : 0;
                    if (hit) {
                        atomicAdd(A.t + pos, 1u);
                        atomicAdd(ca + i, 1u);
                        atomicAdd(ca + j, 1u);
                        if (m) A.hits[hb + nh + __popc(m & ((1u << lane) - 1))] = make_uint2((uint32_t)i << 16 | j, pos);
                    }
                    nh += __popc(m);
                } else {
                    const unsigned m = __ballot_sync(kFull, hit);
                    if (hit) {
                        const int at = nh + __popc(m & ((1u << lane) - 1));
                        s_slot[wid][at] = pos;
                        s_hit[wid][at] = (uint16_t)pr;
                        atomicOr(f + i, 1u << j);
                        atomicOr(f + j, 1u << i);
                    }
                    nh += __popc(m);
                }
            }
            __syncwarp();
            if (PASS == 1) {
                if (lane < d && ca[lane]) atomicAdd(A.t + ra + lane, ca[lane]);
                if (A.hcount && lane == 0) A.hcount[a] = (uint32_t)nh;
            } else {
                for (int h = lane; h < nh; h += 32) {
                    const uint32_t pos = s_slot[wid][h];
                    const int i = s_hit[wid][h] >> 8, j = s_hit[wid][h] & 255;
                    const uint32_t c = (uint32_t)__popc(f[i] & f[j]);
                    const uint32_t tij = A.t[pos], ti = ta[i], tj = ta[j];
                    atomicAdd(A.dk + pos, ((unsigned long long)(ti + tj) << 32) + c);
                    atomicAdd(ca + i, c);
                    atomicAdd(ca + j, c);
                    atomicAdd(cb + i, tj + tij);
                    atomicAdd(cb + j, ti + tij);
                }
                __syncwarp();
                if (lane < d && (ca[lane] | cb[lane]))
                    atomicAdd(A.dk + ra + lane, ((unsigned long long)cb[lane] << 32) + (ca[lane] >> 1));
            }
            __syncwarp();
        }
    }
}

// Table sizes of the block kernels for up to dmax neighbours.
__host__ __device__ __forceinline__ int ego_hash_bits(int dmax) {   // a table at least 4 times as large
    int b = 7;
    while ((1 << b) < 4 * dmax) b++;
    return b;
}
// 64-bit words of a row of F: odd, so that rows spread over the banks
__host__ __device__ __forceinline__ int ego_row_words(int dmax) { return ((dmax + 63) / 64) | 1; }

// Ranks below this have their index in N(+)(a) in a direct table, most entries
// of the lists being of high rank; the others are looked up in the hash table.
constexpr int kTopRanks = 8192;

// One block's tables: [F] hash keys, N+(a)'s rows (start, length), list,
// counts, [sums of t, t of (a, x)], hash indices, direct table
struct EgoTables {
    unsigned long long *F;
    uint32_t *hkey, *rs;
    int32_t *ru, *ls;
    uint32_t *ck, *cd, *ta;
    uint16_t *hidx, *top;
};
__host__ __device__ __forceinline__ int64_t ego_layout(uint8_t *base, int dmax, bool lookup, bool counts2,
                                                       EgoTables *T) {
    uint8_t *p = base;
    auto take = [&](int64_t bytes) {
        uint8_t *q = p;
        p += bytes;
        return q;
    };
    const int hb = ego_hash_bits(dmax);
    T->F = (unsigned long long *)take(counts2 ? (int64_t)dmax * 8 * ego_row_words(dmax) : 0);
    T->ck = (uint32_t *)take((int64_t)dmax * 4);
    T->cd = (uint32_t *)take(counts2 ? (int64_t)dmax * 4 : 0);
    T->ta = (uint32_t *)take(counts2 ? (int64_t)dmax * 4 : 0);
    T->hkey = (uint32_t *)take(lookup ? (int64_t)4 << hb : 0);
    T->rs = (uint32_t *)take(lookup ? (int64_t)dmax * 4 : 0);
    T->ru = (int32_t *)take(lookup ? (int64_t)dmax * 4 : 0);
    T->ls = (int32_t *)take(lookup ? (int64_t)dmax * 4 : 0);
    T->hidx = (uint16_t *)take(lookup ? (int64_t)2 << hb : 0);
    T->top = (uint16_t *)take(lookup ? (int64_t)2 * kTopRanks : 0);
    return ((p - base) + 127) & ~(int64_t)127;
}
inline int64_t ego_table_bytes(int dmax, bool lookup, bool counts2) {
    EgoTables T;
    return ego_layout(nullptr, dmax, lookup, counts2, &T);
}

// The second half of pass 2: each triangle {a, x, y} (indices i, j; slot x -> y)
// with c = |F_i & F_j| 4-cliques.  All threads of the block call.
template <int NT>
__device__ __forceinline__ void clique_hits(const EgoArgs &A, const uint2 *hits, uint32_t nh, const EgoTables &T, int W,
                                            int WS) {
    const int lane = threadIdx.x & 31;
    for (uint32_t h0 = threadIdx.x - lane; h0 < nh; h0 += NT) {
        const uint32_t h = h0 + lane;
        uint32_t c = 0, di = 0;
        int i = -1;
        if (h < nh) {
            const uint2 e = hits[h];
            const uint32_t tij = A.t[e.y];
            i = (int)(e.x >> 16);
            const int j = (int)(e.x & 0xffff);
            const unsigned long long *fi = T.F + (int64_t)i * WS, *fj = T.F + (int64_t)j * WS;
            for (int w = 0; w < W; w++) c += (uint32_t)__popcll(fi[w] & fj[w]);
            const uint32_t ti = T.ta[i], tj = T.ta[j];
            atomicAdd(A.dk + e.y, ((unsigned long long)(ti + tj) << 32) + c);
            if (c) atomicAdd(T.ck + j, c);
            atomicAdd(T.cd + j, ti + tij);
            di = tj + tij;
        }
        // most warps hold one x: reduce its sums first
        const int i0 = __shfl_sync(kFull, i, 0);
        if (__all_sync(kFull, i == i0 || i < 0)) {
            c = __reduce_add_sync(kFull, c);
            di = __reduce_add_sync(kFull, di);
            if (lane == 0) {
                if (c) atomicAdd(T.ck + i0, c);
                atomicAdd(T.cd + i0, di);
            }
        } else if (i >= 0) {
            if (c) atomicAdd(T.ck + i, c);
            atomicAdd(T.cd + i, di);
        }
    }
}

// Index in N+(a) of the vertex of rank y, -1 if it is not among them (last: the
// largest rank asked for).
__device__ __forceinline__ int ego_find(const EgoTables &T, int32_t y, int32_t last, int shift, uint32_t hmask) {
    if (y < kTopRanks) return (int)T.top[y] - 1;
    if (y > last) return -1;
    uint32_t h = hash_of((uint32_t)y, shift), k;
    while ((k = T.hkey[h]) != (uint32_t)y && k != kFull) h = (h + 1) & hmask;
    return k == (uint32_t)y ? (int)T.hidx[h] : -1;
}

// The same without a list: the rows of N+(a) looked up once more, a warp per row
// from the counter *next (index of the last row at the start).
__device__ __forceinline__ void clique_rows(const EgoArgs &A, const EgoTables &T, int W, int WS, int shift,
                                            uint32_t hmask, int *next) {
    const int lane = threadIdx.x & 31;
    while (true) {
        int i = 0;
        if (lane == 0) i = atomicSub(next, 1);
        i = __shfl_sync(kFull, i, 0);
        if (i < 1) break;
        const uint32_t r0 = T.rs[i], ti = T.ta[i];
        const int len = T.ru[i];
        const int32_t last = T.ls[i - 1];
        const unsigned long long *fi = T.F + (int64_t)i * WS;
        uint32_t ci = 0, di = 0;
        for (int b = 0; b < len; b += 32) {
            const uint32_t pos = r0 + (uint32_t)(b + lane);
            const int32_t y = b + lane < len ? __ldg(A.radj + pos) : 0x7fffffff;
            const int j = ego_find(T, y, last, shift, hmask);
            if (j >= 0) {
                const unsigned long long *fj = T.F + (int64_t)j * WS;
                uint32_t c = 0;
                for (int w = 0; w < W; w++) c += (uint32_t)__popcll(fi[w] & fj[w]);
                const uint32_t tij = A.t[pos], tj = T.ta[j];
                atomicAdd(A.dk + pos, ((unsigned long long)(ti + tj) << 32) + c);
                if (c) atomicAdd(T.ck + j, c);
                atomicAdd(T.cd + j, ti + tij);
                ci += c;
                di += tj + tij;
            }
            if (__shfl_sync(kFull, y, 31) > last) break;   // ascending: nothing more at or below last
        }
        ci = __reduce_add_sync(kFull, ci);
        di = __reduce_add_sync(kFull, di);
        if (lane == 0) {
            if (ci) atomicAdd(T.ck + i, ci);
            if (di) atomicAdd(T.cd + i, di);
        }
    }
}

// |N+(a)| = d in a block's range: a block per vertex.  The indices of N+(a) go
// into the lookup tables; each warp takes vertices x of N+(a) and looks the
// entries of N+(x) up (searching N+(a)'s entries in N+(x) where that takes fewer
// instructions is bound by the searches' latency: with 32 entries a turn 5.0 against
// 5.4 ms for the smaller class on R-MAT 20, 2.9 against 2.1 ms for the next).  PASS 1
// counts the triangles and, where there is room, keeps them for k_clique_block;
// PASS 2 (else) lists them again, with F, or only finds them again (clique_rows).
template <int PASS, int NT, bool GLOBAL>
__global__ void __launch_bounds__(NT) k_ego_block(EgoArgs A, int dmax) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    __shared__ uint32_t s_item;
    __shared__ uint32_t s_nhit;
    __shared__ int s_row;
    const int lane = threadIdx.x & 31;
    const int hb = ego_hash_bits(dmax), shift = 32 - hb;
    const uint32_t hmask = (1u << hb) - 1;
    EgoTables T;
    ego_layout(GLOBAL ? A.tables + (int64_t)blockIdx.x * A.tables_stride : (uint8_t *)s_dyn, dmax, true, PASS == 2, &T);
    const int WS = ego_row_words(dmax);
    uint32_t *F32 = (uint32_t *)T.F;
    for (int i = threadIdx.x; i < kTopRanks / 2; i += NT) ((uint32_t *)T.top)[i] = 0;
    while (true) {
        if (threadIdx.x == 0) {
            s_item = (uint32_t)atomicAdd(A.next, 1ull);
            s_nhit = 0;
        }
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= A.count) break;
        const uint32_t a = (uint32_t)A.list[item];
        const int d = A.rup[a];
        const uint32_t ra = A.roff[a];
        const int W = (d + 63) >> 6;
        uint2 *hits = nullptr;
        if (PASS == 2) hits = A.hits ? A.hits + (int64_t)blockIdx.x * A.hits_stride : nullptr;
        else if (A.hcount) hits = A.hits + A.hbase[a];
        if (threadIdx.x == 0) s_row = d - 1;
        for (int i = threadIdx.x; i <= (int)hmask; i += NT) T.hkey[i] = kFull;
        if (PASS == 2)
            for (int i = threadIdx.x; i < d * WS; i += NT) T.F[i] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < d; i += NT) {
            const int32_t x = __ldg(A.radj + ra + i);
            T.ls[i] = x;
            T.rs[i] = __ldg(A.roff + x);
            T.ru[i] = __ldg(A.rup + x);
            T.ck[i] = 0;
            if (PASS == 2) {
                T.cd[i] = 0;
                T.ta[i] = A.t[ra + i];
            }
            if (x < kTopRanks) {
                T.top[x] = (uint16_t)(i + 1);
            } else {
                uint32_t h = hash_of((uint32_t)x, shift);
                while (atomicCAS(T.hkey + h, kFull, (uint32_t)x) != kFull) h = (h + 1) & hmask;
                T.hidx[h] = (uint16_t)i;
            }
        }
        __syncthreads();
        while (true) {
            int i = 0;
            if (lane == 0) i = atomicSub(&s_row, 1);
            i = __shfl_sync(kFull, i, 0);
            if (i < 1) break;   // the first neighbour has none of the others above it
            const uint32_t r0 = T.rs[i];
            const int len = T.ru[i];
            uint32_t found = 0;
            const int32_t last = T.ls[i - 1];
            auto find = [&](int32_t y) { return ego_find(T, y, last, shift, hmask); };
            // 64 entries a turn: two loads in flight, one place among the hits for both
            // (R-MAT 20: 5.42 -> 4.70 ms for the smaller class, 2.12 -> 1.64 ms for the
            // next; bound by issue.  Short rows end to end over the lanes instead: 5.72 ms)
            for (int b = 0; b < len; b += 64) {
                const uint32_t pos = r0 + (uint32_t)(b + lane);
                const int32_t yA = b + lane < len ? __ldg(A.radj + pos) : 0x7fffffff;
                const int32_t yB = b + 32 + lane < len ? __ldg(A.radj + pos + 32) : 0x7fffffff;
                const int jA = find(yA), jB = b + 32 < len ? find(yB) : -1;
                const unsigned mA = __ballot_sync(kFull, jA >= 0), mB = __ballot_sync(kFull, jB >= 0);
                if (mA | mB) {
                    const uint32_t nA = (uint32_t)__popc(mA), nB = (uint32_t)__popc(mB);
                    if (hits) {
                        uint32_t at = 0;
                        if (lane == 0) at = atomicAdd(&s_nhit, nA + nB);
                        at = __shfl_sync(kFull, at, 0);
                        const unsigned below = (1u << lane) - 1;
                        if (jA >= 0) hits[at + __popc(mA & below)] = make_uint2((uint32_t)i << 16 | (uint32_t)jA, pos);
                        if (jB >= 0)
                            hits[at + nA + __popc(mB & below)] = make_uint2((uint32_t)i << 16 | (uint32_t)jB, pos + 32);
                    }
                    auto credit = [&](int j, uint32_t p) {
                        if (PASS == 1) {
                            atomicAdd(A.t + p, 1u);
                            atomicAdd(T.ck + j, 1u);
                        } else {
                            atomicOr(F32 + (int64_t)i * 2 * WS + (j >> 5), 1u << (j & 31));
                            atomicOr(F32 + (int64_t)j * 2 * WS + (i >> 5), 1u << (i & 31));
                        }
                    };
                    if (jA >= 0) credit(jA, pos);
                    if (jB >= 0) credit(jB, pos + 32);
                    found += nA + nB;
                }
                if (__shfl_sync(kFull, yB, 31) > last) break;   // ascending: nothing more at or below last
            }
            if (PASS == 1 && lane == 0 && found) atomicAdd(T.ck + i, found);
        }
        __syncthreads();
        if (PASS == 2) {
            if (hits) {
                clique_hits<NT>(A, hits, s_nhit, T, W, WS);
            } else {
                if (threadIdx.x == 0) s_row = d - 1;
                __syncthreads();
                clique_rows(A, T, W, WS, shift, hmask, &s_row);
            }
            __syncthreads();
        } else if (A.hcount && threadIdx.x == 0) {
            A.hcount[a] = s_nhit;
        }
        for (int i = threadIdx.x; i < d; i += NT) {
            if (PASS == 1) {
                if (T.ck[i]) atomicAdd(A.t + ra + i, T.ck[i]);
            } else if (T.ck[i] | T.cd[i]) {
                atomicAdd(A.dk + ra + i, ((unsigned long long)T.cd[i] << 32) + (T.ck[i] >> 1));
            }
            if (T.ls[i] < kTopRanks) T.top[T.ls[i]] = 0;
        }
        __syncthreads();
    }
}

// Pass 2 from the triangles that pass 1 kept: F from the list, then the list again.
template <int NT, bool GLOBAL>
__global__ void __launch_bounds__(NT) k_clique_block(EgoArgs A, int dmax) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    __shared__ uint32_t s_item;
    EgoTables T;
    ego_layout(GLOBAL ? A.tables + (int64_t)blockIdx.x * A.tables_stride : (uint8_t *)s_dyn, dmax, false, true, &T);
    const int WS = ego_row_words(dmax);
    uint32_t *F32 = (uint32_t *)T.F;
    while (true) {
        if (threadIdx.x == 0) s_item = (uint32_t)atomicAdd(A.next, 1ull);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= A.count) break;
        const uint32_t a = (uint32_t)A.list[item];
        const int d = A.rup[a];
        const uint32_t ra = A.roff[a], nh = A.hcount[a];
        const int W = (d + 63) >> 6;
        const uint2 *hits = A.hits + A.hbase[a];
        for (int i = threadIdx.x; i < d * WS; i += NT) T.F[i] = 0;
        for (int i = threadIdx.x; i < d; i += NT) {
            T.ck[i] = 0;
            T.cd[i] = 0;
            T.ta[i] = A.t[ra + i];
        }
        __syncthreads();
        for (uint32_t h = threadIdx.x; h < nh; h += NT) {
            const uint32_t e = hits[h].x;
            const int i = (int)(e >> 16), j = (int)(e & 0xffff);
            atomicOr(F32 + (int64_t)i * 2 * WS + (j >> 5), 1u << (j & 31));
            atomicOr(F32 + (int64_t)j * 2 * WS + (i >> 5), 1u << (i & 31));
        }
        __syncthreads();
        clique_hits<NT>(A, hits, nh, T, W, WS);
        __syncthreads();
        for (int i = threadIdx.x; i < d; i += NT)
            if (T.ck[i] | T.cd[i])
                atomicAdd(A.dk + ra + i, ((unsigned long long)T.cd[i] << 32) + (T.ck[i] >> 1));
        __syncthreads();
    }
}

// |N+(a)| <= 32: a warp per vertex, F one 32-bit word per row.
__global__ void __launch_bounds__(kWarpThreads) k_clique_warp(EgoArgs A) {
    constexpr int kW = kWarpThreads / 32;
    __shared__ uint32_t s_a[kW][32], s_b[kW][32], s_f[kW][32], s_t[kW][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t *ca = s_a[wid], *cb = s_b[wid], *f = s_f[wid], *ta = s_t[wid];
    while (true) {
        uint32_t i0 = 0;
        if (lane == 0) i0 = (uint32_t)atomicAdd(A.next, (unsigned long long)A.grab);
        i0 = __shfl_sync(kFull, i0, 0);
        if (i0 >= A.count) break;
        const uint32_t i1 = min(i0 + A.grab, A.count);
        for (uint32_t ii = i0; ii < i1; ii++) {
            const uint32_t a = (uint32_t)A.list[ii];
            const uint32_t nh = A.hcount[a];
            if (!nh) continue;
            const int d = A.rup[a];
            const uint32_t ra = A.roff[a];
            const uint2 *hits = A.hits + A.hbase[a];
            ca[lane] = cb[lane] = f[lane] = 0;
            ta[lane] = lane < d ? A.t[ra + lane] : 0;
            __syncwarp();
            for (uint32_t h = lane; h < nh; h += 32) {
                const uint32_t e = hits[h].x;
                atomicOr(f + (e >> 16), 1u << (e & 31));
                atomicOr(f + (e & 31), 1u << (e >> 16));
            }
            __syncwarp();
            for (uint32_t h = lane; h < nh; h += 32) {
                const uint2 e = hits[h];
                const int i = (int)(e.x >> 16), j = (int)(e.x & 0xffff);
                const uint32_t c = (uint32_t)__popc(f[i] & f[j]);
                const uint32_t tij = A.t[e.y], ti = ta[i], tj = ta[j];
                atomicAdd(A.dk + e.y, ((unsigned long long)(ti + tj) << 32) + c);
                atomicAdd(ca + i, c);
                atomicAdd(ca + j, c);
                atomicAdd(cb + i, tj + tij);
                atomicAdd(cb + j, ti + tij);
            }
            __syncwarp();
            if (lane < d && (ca[lane] | cb[lane]))
                atomicAdd(A.dk + ra + lane, ((unsigned long long)cb[lane] << 32) + (ca[lane] >> 1));
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// closing: t, k4, c4 of each position, its closed forms and its row

struct CloseArgs {
    pgd_rank_out o;
    const uint32_t *eslot;
    const uint32_t *tw;
    const uint32_t *t;
    const unsigned long long *dk;
    const uint32_t *cyc;
};

__device__ __forceinline__ void flush_warp(unsigned long long *acc, unsigned long long *dst, int lane) {
#pragma unroll
    for (int i = 0; i < PGD_NSUMS; i++) {
        const unsigned long long v = pgd_warp_sum(acc[i]);
        if (lane == 0 && v) atomicAdd(dst + i, v);
        acc[i] = 0;
    }
}

// A warp takes a contiguous part of the positions, 32 at a time; in a batch
// they belong to few graphs, whose sums are flushed when the graph changes.
__global__ void __launch_bounds__(kThreads) k_rank_close(CloseArgs A) {
    const pgd_rank_out &o = A.o;
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t steps = (o.npos + 31) / 32, per = (steps + nw - 1) / nw;
    const int64_t e1 = min(o.npos, (w + 1) * per * 32);
    unsigned long long acc[PGD_NSUMS];
#pragma unroll
    for (int i = 0; i < PGD_NSUMS; i++) acc[i] = 0;
    int cur = -1;   // graph of the sums held (batch)
    long long n = o.n, m = o.m;
    for (int64_t e0 = w * per * 32; e0 < e1; e0 += 32) {
        const int64_t e = e0 + lane;
        bool act = e < e1;
        int g = 0;
        if (o.egraph) {
            if (act) g = o.egraph[e];
            if (act && o.gdense && o.gdense[g]) act = false;
        }
        long long dv = 0, du = 0;
        unsigned long long t = 0, k4 = 0, c4 = 0;
        if (act) {
            const int32_t id = o.order[e];
            const uint32_t j = __ldg(A.eslot + id);
            dv = __ldg(o.deg + __ldg(o.ev + id));
            du = __ldg(o.deg + __ldg(o.eu + id));
            const uint32_t tt = __ldg(A.t + j);
            const unsigned long long x = __ldg(A.dk + j);
            const uint32_t cc = __ldg(A.cyc + j) + __ldg(A.cyc + __ldg(A.tw + j));
            t = tt;
            k4 = (uint32_t)x;
            c4 = cc - (uint32_t)(x >> 32) + 2 * tt + 2 * (uint32_t)x;
        }
        unsigned todo = __ballot_sync(kFull, act);
        while (todo) {
            const int g0 = o.egraph ? __shfl_sync(kFull, g, __ffs(todo) - 1) : 0;
            if (o.egraph && g0 != cur) {
                if (cur >= 0) flush_warp(acc, o.sums + (int64_t)cur * PGD_NSUMS, lane);
                cur = g0;
                n = o.gnm[2 * (int64_t)g0];
                m = o.gnm[2 * (int64_t)g0 + 1];
            }
            const bool mine = act && (!o.egraph || g == g0);
            if (mine) {
                pgd_edge_sums(acc, dv, du, t, m, n);
                acc[3] += k4;
                acc[4] += c4;
            }
            todo &= ~__ballot_sync(kFull, mine);
        }
        if (act && o.micro) {
            ulonglong2 *row = (ulonglong2 *)(o.micro + e * PGD_NMICRO);
#pragma unroll
            for (int c = 0; c < PGD_NMICRO; c += 2) {
                ulonglong2 v;
                v.x = pgd_micro_col(c, dv, du, t, k4, c4);
                v.y = pgd_micro_col(c + 1, dv, du, t, k4, c4);
                row[c / 2] = v;
            }
        }
    }
    if (o.egraph) {
        if (cur >= 0) flush_warp(acc, o.sums + (int64_t)cur * PGD_NSUMS, lane);
        return;
    }
    __shared__ unsigned long long red[kThreads / 32][PGD_NSUMS];
#pragma unroll
    for (int i = 0; i < PGD_NSUMS; i++) {
        const unsigned long long v = pgd_warp_sum(acc[i]);
        if (lane == 0) red[threadIdx.x >> 5][i] = v;
    }
    __syncthreads();
    if (threadIdx.x < PGD_NSUMS) {
        unsigned long long s = 0;
        for (int i = 0; i < kThreads / 32; i++) s += red[i][threadIdx.x];
        if (s) atomicAdd(o.sums + threadIdx.x, s);
    }
}

// Stream-ordered temporaries released on every return path.
struct Tmp {
    pgd_ctx *ctx;
    void *held[16];   // more than any caller takes
    int k = 0;
    explicit Tmp(pgd_ctx *c) : ctx(c) {}
    Tmp(const Tmp &) = delete;
    Tmp &operator=(const Tmp &) = delete;
    ~Tmp() {
        while (k) pgd_tmp_free(ctx, held[--k]);
    }
    template <typename T>
    pgd_status alloc(T **out, size_t bytes) {
        void *p = nullptr;
        const pgd_status st = pgd_tmp_alloc(ctx, &p, bytes);
        if (st == PGD_OK) {
            held[k++] = p;
            *out = (T *)p;
        }
        return st;
    }
};

}  // namespace

// ---------------------------------------------------------------------------

void pgd_rank_free(pgd_graph *g, pgd_rank_graph *R) {
    while (R->nheld) {
        R->nheld--;
        pgd_graph_free(g, R->held[R->nheld], R->held_bytes[R->nheld]);
    }
    *R = pgd_rank_graph();
}

void pgd_rank_drop(pgd_graph *g) {
    if (!g->ranked) return;
    pgd_rank_free(g, g->ranked);
    delete g->ranked;
    g->ranked = nullptr;
}

#define RB_TRY(expr)                   \
    do {                               \
        if ((st = (expr)) != PGD_OK) { \
            pgd_rank_free(g, R);       \
            return st;                 \
        }                              \
    } while (0)
#define RB_CUDA(call)                                     \
    do {                                                  \
        const cudaError_t e__ = (call);                   \
        if (e__ != cudaSuccess) {                         \
            pgd_rank_free(g, R);                          \
            return pgd_cuda_fail(ctx, e__, #call);        \
        }                                                 \
    } while (0)

// Ranks, rows, slots, wedges and lists of a graph of any size; *wd_out, *tmp_out and
// *tb_out get the wedge counts and CUB's temporary storage, held by tg.
static pgd_status rank_build_large(pgd_graph *g, int64_t nnz, const int32_t *vgraph, const uint8_t *vmask,
                                   pgd_rank_graph *R, RankMeta *M, Tmp &tg, uint32_t **wd_out, void **tmp_out,
                                   size_t *tb_out) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    pgd_status st;
    const int64_t n = g->n, m = g->m;
    const size_t nb = (n + 1) * sizeof(uint32_t), eb = nnz * sizeof(uint32_t);
    uint64_t *keys = nullptr, *keys2 = nullptr;
    int32_t *vrank = nullptr, *rv = nullptr, *val = nullptr;
    uint32_t *rdeg = nullptr, *key = nullptr, *key2 = nullptr;
    const int vb = bits_for(n), db = bits_for((int64_t)g->max_degree + 1);
    size_t tb1 = 0, tb2 = 0, tb3 = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, tb1, keys, keys2, n, 0, vb + db, s);
    cub::DeviceScan::ExclusiveSum(nullptr, tb2, rdeg, R->roff, n + 1, s);
    cub::DeviceRadixSort::SortPairs(nullptr, tb3, key, key2, val, R->radj, nnz, 0, vb, s);
    const size_t tb = *tb_out = std::max(tb1, std::max(tb2, tb3));
    pgd_pieces W;
    W.add(2 * nb); W.add(2 * nb); W.add(nb); W.add(nb); W.add(nb); W.add(nb); W.add(eb); W.add(eb); W.add(eb); W.add(tb);
    if ((st = tg.alloc(&W.base, W.bytes))) return st;
    keys = W.take<uint64_t>(2 * nb);
    keys2 = W.take<uint64_t>(2 * nb);
    vrank = W.take<int32_t>(nb);
    rv = W.take<int32_t>(nb);
    rdeg = W.take<uint32_t>(nb);
    uint32_t *wd = *wd_out = W.take<uint32_t>(nb);
    key = W.take<uint32_t>(eb);
    key2 = W.take<uint32_t>(eb);
    val = W.take<int32_t>(eb);
    void *tmp = *tmp_out = W.take<void>(tb);
    // ranks and row offsets
    PGD_LAUNCH(ctx, k_rank_keys2, grid_for(n), kThreads, 0, g->deg, vgraph, vmask, n, g->max_degree, vb, keys, M);
    PGD_CUDA(ctx, cub::DeviceRadixSort::SortKeys(tmp, *tb_out, keys, keys2, n, 0, vb + db, s));
    PGD_LAUNCH(ctx, k_rank_scatter2, grid_for(n + 1), kThreads, 0, keys2, n, g->max_degree, vb, vrank, rv, rdeg, R->rup,
               R->bend, wd, M);
    PGD_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, *tb_out, rdeg, R->roff, n + 1, s));
    // rows in rank order
    PGD_LAUNCH(ctx, k_rank_entries, grid_for(nnz), kThreads, 0, R->roff, rv, g->off, g->adj, vrank, n, nnz, key, val);
    PGD_CUDA(ctx, cub::DeviceRadixSort::SortPairs(tmp, *tb_out, key, key2, val, R->radj, nnz, 0, vb, s));
    PGD_LAUNCH(ctx, k_rank_slots, grid_for(nnz), kThreads, 0, R->roff, R->radj, n, nnz, M, R->wcode, R->tw, R->rup,
               R->bend);
    PGD_LAUNCH(ctx, k_rank_eslot, grid_for(m), kThreads, 0, g->ev, g->eu, vrank, R->roff, R->rup, R->radj, vgraph,
               vmask, m, R->eslot);
    // wedges per vertex and the work lists
    PGD_LAUNCH(ctx, k_rank_wedges, grid_for(nnz), kThreads, 0, R->roff, R->radj, R->tw, R->bend, n, M, wd);
    PGD_LAUNCH(ctx, k_rank_lists, grid_for(n), kThreads, 0, R->rup, wd, n, R->lists, R->hbase, M);
    PGD_CUDA(ctx, cudaGetLastError());
    PGD_CUDA(ctx, pgd_fetch(ctx, 0, M, kMetaHead));
    PGD_CUDA(ctx, cudaStreamSynchronize(s));
    return PGD_OK;
}

// Blocks of k_cycle_direct per SM: as many as all counters fit in.
static int direct_factor(int64_t words) { return words < kDirectWords / 4 ? 4 : words < kDirectWords / 2 ? 2 : 1; }

pgd_status pgd_rank_build(pgd_graph *g, int64_t nnz, const int32_t *vgraph, const uint8_t *vmask, pgd_rank_graph *R) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    pgd_status st;
    const int64_t n = g->n, m = g->m;
    *R = pgd_rank_graph();
    R->n = n;
    R->nnz = nnz;
    if (nnz == 0) return PGD_OK;
    auto keep = [&](auto **p, size_t bytes) -> pgd_status {
        const pgd_status e = pgd_graph_alloc(g, (void **)p, bytes);
        if (e == PGD_OK) {
            R->held[R->nheld] = *p;
            R->held_bytes[R->nheld++] = bytes;
        }
        return e;
    };
    // kept arrays in one allocation; the range boundaries behind the sizes only where
    // vertices are likely to have items
    const bool one_block = !vgraph && nnz <= 2 * kSmallPairs && n <= kSmallVertices;
    const size_t meta_bytes = one_block ? kMetaHead : sizeof(RankMeta);
    pgd_pieces K;
    const size_t nb = (n + 1) * sizeof(uint32_t), eb = nnz * sizeof(uint32_t), mb = m * sizeof(int32_t),
                 lb = (size_t)kClasses * n * sizeof(int32_t), hb = n * sizeof(unsigned long long);
    K.add(meta_bytes); K.add(nb); K.add(nb); K.add(nb); K.add(eb); K.add(eb); K.add(eb); K.add(mb); K.add(lb); K.add(hb);
    RB_TRY(keep(&K.base, K.bytes));
    RankMeta *M = K.take<RankMeta>(meta_bytes);
    R->meta = M;
    R->roff = K.take<uint32_t>(nb);
    R->rup = K.take<int32_t>(nb);
    R->bend = K.take<uint32_t>(nb);
    R->radj = K.take<int32_t>(eb);
    R->wcode = K.take<uint32_t>(eb);
    R->tw = K.take<uint32_t>(eb);
    R->eslot = K.take<uint32_t>(mb);
    R->lists = K.take<int32_t>(lb);
    R->hbase = K.take<unsigned long long>(hb);
    Tmp tg(ctx);
    uint32_t *wd = nullptr;
    void *tmp = nullptr;
    size_t tb = 0;
    if (one_block) {
        RankSmallArgs A{};
        A.off = g->off;
        A.adj = g->adj;
        A.deg = g->deg;
        A.ev = g->ev;
        A.eu = g->eu;
        A.n = (int)n;
        A.nnz = (int)nnz;
        A.m = (int)m;
        A.max_degree = g->max_degree;
        A.pv = pgd_small_words(n);
        A.pe = pgd_small_words(nnz);
        A.roff = R->roff;
        A.rup = R->rup;
        A.bend = R->bend;
        A.radj = R->radj;
        A.wcode = R->wcode;
        A.tw = R->tw;
        A.eslot = R->eslot;
        A.lists = R->lists;
        A.hbase = R->hbase;
        A.M = M;
        A.host = (RankMeta *)ctx->pin;
        cub::DeviceScan::ExclusiveSum(nullptr, tb, wd, wd, n + 1, s);
        pgd_pieces W;
        W.add(nb); W.add(tb);
        RB_TRY(tg.alloc(&W.base, W.bytes));
        A.wd = wd = W.take<uint32_t>(nb);
        tmp = W.take<void>(tb);
        PGD_LAUNCH(ctx, k_rank_small, 1, kSmallThreads, rank_small_bytes((int)n, A.pv, A.pe), A);
        RB_CUDA(cudaGetLastError());
        RB_CUDA(cudaStreamSynchronize(s));
    } else {
        RB_TRY(rank_build_large(g, nnz, vgraph, vmask, R, M, tg, &wd, &tmp, &tb));
    }
    RankMeta h;
    memcpy((void *)&h, ctx->pin, kMetaHead);
    const int n2 = R->n2 = (int32_t)h.tier[4];
    R->max_up = (int32_t)std::max((uint32_t)kEgoMax[kEgoWarp], h.max_up);
    for (int i = 0; i < kClasses; i++) R->nlist[i] = h.nlist[i];
    R->pairs = (int64_t)h.pairs;
    if (n2 == 0 || h.direct_wedges == 0) return PGD_OK;
    // items of the vertices with many wedges, by ranges of the wedges' ends:
    // fine enough to balance the items, and at most half an item's counters each
    const int64_t words = R->words = ((int64_t)h.tcode[4] + 31) / 32;
    R->nranges = (int32_t)std::min<int64_t>(kMaxRanges, std::max<int64_t>(16, 2 * (2 * words / kDirectWords + 1)));
    if (one_block) {   // the sizes again, with room for the boundaries
        RankMeta *full = nullptr;
        RB_TRY(keep(&full, sizeof(RankMeta)));
        RB_CUDA(cudaMemcpyAsync(full, M, kMetaHead, cudaMemcpyDeviceToDevice, s));
        R->meta = M = full;
    }
    PGD_LAUNCH(ctx, k_rank_bounds, 1, 128, 0, R->roff, R->nranges, M);
    const int64_t bpos_bytes = (int64_t)(R->nranges - 1) * n2 * (int64_t)sizeof(uint32_t);
    // the table is left out where the budget or the device has no room for it
    const std::string err = ctx->err;
    const int64_t bpos_most = (int64_t)std::min<uint64_t>(kBposBytes, ctx->list_limit / 4);
    st = bpos_bytes <= bpos_most ? keep(&R->bpos, (size_t)bpos_bytes) : PGD_ENOMEM;
    if (st == PGD_ENOMEM) {
        R->bpos = nullptr;
        ctx->err = err;
    } else {
        RB_TRY(st);
        PGD_LAUNCH(ctx, k_rank_bpos, grid_for((int64_t)n2 * (R->nranges - 1)), kThreads, 0, R->roff, R->radj, n2,
                   R->nranges, M, R->bpos);
    }
    uint32_t *count = nullptr, *pos = nullptr;
    RB_TRY(tg.alloc(&count, 2 * ((size_t)n2 + 1) * sizeof(uint32_t)));
    pos = count + n2 + 1;
    const int parts = ctx->num_sms * 4 * (1 + direct_factor(words));
    PGD_LAUNCH(ctx, k_rank_items, grid_for(n2 + 1), kThreads, 0, wd, n2, R->nranges, M, parts, count,
               (const uint32_t *)nullptr, (int2 *)nullptr);
    RB_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, count, pos, (int64_t)n2 + 1, s));
    RB_CUDA(pgd_fetch(ctx, 0, pos + n2, sizeof(uint32_t)));
    RB_CUDA(cudaStreamSynchronize(s));
    R->nitems = pgd_pinned<uint32_t>(ctx, 0);
    RB_TRY(keep(&R->items, (size_t)R->nitems * sizeof(int2)));
    PGD_LAUNCH(ctx, k_rank_items, grid_for(n2 + 1), kThreads, 0, wd, n2, R->nranges, M, parts, (uint32_t *)nullptr,
               (const uint32_t *)pos, R->items);
    RB_CUDA(cudaGetLastError());
    return PGD_OK;
}

// Vertices a warp takes from a list at a time: one while there are warps to
// spare (a short list then spreads over the whole device), else four.
static uint32_t grab_for(const pgd_ctx *ctx, uint32_t count) { return count > 64u * (uint32_t)ctx->num_sms ? 4 : 1; }

static int warp_blocks(const pgd_ctx *ctx, uint32_t count, uint32_t grab, int per_sm) {
    const int64_t per_block = (int64_t)(kWarpThreads / 32) * grab;
    return (int)std::min<int64_t>((count + per_block - 1) / per_block, (int64_t)per_sm * ctx->num_sms);
}

// Blocks per SM of a block class, and whether the class has so few vertices
// that each gets a block of 1024 threads (at most two waves of them): a short
// list is bound by its largest vertex, not by the device.
static int ego_blocks_per_sm(int c) { return c == kEgoA ? 8 : c == kEgoB ? 3 : 1; }
static bool ego_wide(const pgd_ctx *ctx, const pgd_rank_graph &R, int c) {
    return R.nlist[c] <= 2u * (uint32_t)ctx->num_sms;
}
static int ego_grid(const pgd_ctx *ctx, const pgd_rank_graph &R, int c) {
    return (int)std::min<int64_t>(R.nlist[c], (int64_t)(ego_wide(ctx, R, c) ? 2 : ego_blocks_per_sm(c)) * ctx->num_sms);
}

// What the ego classes hold beside the counts per slot: the tables of the largest
// neighbourhoods, and every triangle of pass 1, kept for pass 2; or a list of each
// block of pass 2, which then finds its triangles again; or no list, and it finds
// them twice.  A request of G(3000, 0.5): 32 ms with its 8.8 GB kept, 32 to 34 ms
// without a list, 370 ms with a list for as few blocks as 120 MB hold; one of R-MAT
// 16 3.8 and 4.0 ms.
struct EgoMemory {
    bool keep = false;
    int64_t hits = 0;             // triangles in the lists
    int gblocks = 0;              // blocks of kEgoGlobal
    int64_t table_bytes = 0;      // each one's tables
    int64_t bytes() const { return hits * (int64_t)sizeof(uint2) + gblocks * table_bytes; }
};

// The fastest of them that takes at most `limit` bytes (and at least one block's tables).
static EgoMemory ego_memory(const pgd_ctx *ctx, const pgd_rank_graph &R, int64_t limit) {
    EgoMemory E;
    const int64_t hit = sizeof(uint2), most = std::min<int64_t>(ctx->num_sms, R.nlist[kEgoGlobal]);
    auto blocks_in = [&](int64_t bytes, int64_t each) {
        return most ? (int)std::max<int64_t>(1, std::min(most, bytes / each)) : 0;
    };
    const int64_t per = (int64_t)R.max_up * (R.max_up - 1) / 2;
    if (most) E.table_bytes = ego_table_bytes(R.max_up, true, true);
    E.gblocks = blocks_in(kTableBytes, per * hit + E.table_bytes);
    E.hits = R.pairs;
    E.keep = R.pairs * hit <= kKeepBytes && E.bytes() <= limit;
    if (E.keep) return E;
    E.hits = per * E.gblocks;
    for (int c : {kEgoA, kEgoB, kEgoC}) {
        const int64_t dmax = std::min(kEgoMax[c], (int)R.max_up);
        E.hits = std::max(E.hits, ego_grid(ctx, R, c) * (dmax * (dmax - 1) / 2));
    }
    if (E.bytes() <= limit) return E;
    E.hits = 0;
    E.gblocks = blocks_in(std::min(kTableBytes, limit), E.table_bytes);
    return E;
}

// Bytes that lists and tables may take: what the context was given (a quarter of it
// is for the range positions), else kListFloor and beyond it at most what is left
// of its budget and half of the device's free memory.
static int64_t ego_room(const pgd_ctx *ctx) {
    if (ctx->list_limit != UINT64_MAX) return (int64_t)std::min<uint64_t>(ctx->list_limit / 4 * 3, INT64_MAX / 2);
    size_t free_b = 0, total_b = 0;
    uint64_t reserved = 0, used = 0;   // the pool's: what it holds and does not use is free as well
    cudaMemPool_t pool;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) free_b = 0;
    if (cudaDeviceGetDefaultMemPool(&pool, ctx->device) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
        reserved = used = 0;
    cudaGetLastError();
    const uint64_t left = ctx->budget > ctx->resident ? ctx->budget - ctx->resident : 0;
    const uint64_t room = std::min<uint64_t>(left, (free_b + (reserved - used)) / 2);
    return std::max<int64_t>(kListFloor, (int64_t)std::min<uint64_t>(room, INT64_MAX / 2));
}

// The ego classes' launches: pass 1, pass 2 that lists the triangles again, or
// (kept) pass 2 from the triangles of pass 1.
static void ego_pass(pgd_ctx *ctx, const pgd_rank_graph &R, EgoArgs A, int pass, unsigned long long *ctr,
                     uint8_t *tables, const EgoMemory &mem) {
    const bool kept = pass == 2 && mem.keep;
    auto args = [&](int c) {
        EgoArgs B = A;
        B.list = R.lists + (int64_t)c * R.n;
        B.count = R.nlist[c];
        B.next = ctr + c;
        B.grab = grab_for(ctx, B.count);
        return B;
    };
#define EGO_BLOCK(NT, G, grid, smem, B, dmax)                                                    \
    do {                                                                                         \
        if (pass == 1) PGD_LAUNCH(ctx, (k_ego_block<1, NT, G>), grid, NT, smem, B, dmax);        \
        else if (kept) PGD_LAUNCH(ctx, (k_clique_block<NT, G>), grid, NT, smem, B, dmax);        \
        else PGD_LAUNCH(ctx, (k_ego_block<2, NT, G>), grid, NT, smem, B, dmax);                  \
    } while (0)
    if (R.nlist[kEgoGlobal]) {
        EgoArgs B = args(kEgoGlobal);
        B.hits_stride = (int64_t)R.max_up * (R.max_up - 1) / 2;
        B.tables = tables;
        B.tables_stride = mem.table_bytes;
        EGO_BLOCK(1024, true, mem.gblocks, 0, B, R.max_up);
    }
    for (int c : {kEgoC, kEgoB, kEgoA}) {
        if (!R.nlist[c]) continue;
        EgoArgs B = args(c);
        const int dmax = std::min(kEgoMax[c], (int)R.max_up);
        B.hits_stride = (int64_t)dmax * (dmax - 1) / 2;
        const int blocks = ego_grid(ctx, R, c);
        const size_t smem = (size_t)ego_table_bytes(dmax, !kept, pass == 2);
        if (c == kEgoC || ego_wide(ctx, R, c)) EGO_BLOCK(1024, false, blocks, smem, B, dmax);
        else if (c == kEgoB) EGO_BLOCK(512, false, blocks, smem, B, dmax);
        else EGO_BLOCK(256, false, blocks, smem, B, dmax);
    }
#undef EGO_BLOCK
    if (R.nlist[kEgoWarp]) {
        EgoArgs B = args(kEgoWarp);
        const int blocks = warp_blocks(ctx, B.count, B.grab, 8);
        if (pass == 1) PGD_LAUNCH(ctx, k_ego_warp<1>, blocks, kWarpThreads, 0, B);
        else if (kept) PGD_LAUNCH(ctx, k_clique_warp, blocks, kWarpThreads, 0, B);
        else PGD_LAUNCH(ctx, k_ego_warp<2>, blocks, kWarpThreads, 0, B);
    }
}

cudaError_t pgd_rank_limits() {
    constexpr cudaFuncAttribute kDyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_cycle_direct<1024>, kDyn, kDirectWords * 4);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_rank_small, kDyn,
                                 (int)rank_small_bytes((int)kSmallVertices, (int)kSmallVertices, 2 * (int)kSmallPairs));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cycle_direct<512>, kDyn, kDirectWords * 2);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cycle_direct<256>, kDyn, kDirectWords);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cycle_hash, kDyn, kHashSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cycle_warp, kDyn, kWarpSmem);
    const int cmax = kEgoMax[kEgoC];
    const int c1 = (int)ego_table_bytes(cmax, true, false), c2 = (int)ego_table_bytes(cmax, true, true),
              b2 = (int)ego_table_bytes(kEgoMax[kEgoB], true, true), k2 = (int)ego_table_bytes(cmax, false, true);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_ego_block<1, 1024, false>, kDyn, c1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_ego_block<2, 1024, false>, kDyn, c2);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_ego_block<2, 512, false>, kDyn, b2);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_clique_block<1024, false>, kDyn, k2);
    return e;
}

// Runs the 4-cycle kernels on the context's second stream, beside the triangle
// passes; the first stream waits for it before anything they used is freed.
struct SideStream {
    pgd_ctx *ctx;
    cudaStream_t main;
    bool forked = false;
    explicit SideStream(pgd_ctx *c) : ctx(c), main(c->stream) {}
    cudaError_t fork() {
        cudaError_t e = cudaEventRecord(ctx->ev_fork, main);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->side, ctx->ev_fork, 0);
        forked = e == cudaSuccess;
        return e;
    }
    cudaError_t join() {
        if (!forked) return cudaSuccess;
        forked = false;
        cudaError_t e = cudaEventRecord(ctx->ev_join, ctx->side);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(main, ctx->ev_join, 0);
        return e;
    }
    ~SideStream() {
        ctx->stream = main;
        join();
    }
};

static pgd_status cycle_pass(pgd_ctx *ctx, const pgd_rank_graph &R, CycArgs C, unsigned long long *ctr) {
    const int nsm = ctx->num_sms;
    PGD_CUDA(ctx, cudaEventRecord(ctx->evh0, ctx->stream));
    if (R.nitems) {
        CycArgs B = C;
        B.items = R.items;
        B.count = R.nitems;
        B.next = ctr;
        const int f = direct_factor(R.words);
        const int blocks = (int)std::min<int64_t>(R.nitems, (int64_t)f * nsm);
        const size_t smem = std::min<size_t>(kDirectWords * 4 / f, (size_t)(R.words + 1) * 4);
        if (f == 1) PGD_LAUNCH(ctx, k_cycle_direct<1024>, blocks, 1024, smem, B);
        else if (f == 2) PGD_LAUNCH(ctx, k_cycle_direct<512>, blocks, 512, smem, B);
        else PGD_LAUNCH(ctx, k_cycle_direct<256>, blocks, 256, smem, B);
    }
    if (R.nlist[kCycHash]) {
        CycArgs B = C;
        B.list = R.lists + (int64_t)kCycHash * R.n;
        B.count = R.nlist[kCycHash];
        B.next = ctr + 1;
        PGD_LAUNCH(ctx, k_cycle_hash, (int)std::min<int64_t>(B.count, 4 * (int64_t)nsm), kHashThreads, kHashSmem, B);
    }
    if (R.nlist[kCycWarp]) {
        CycArgs B = C;
        B.list = R.lists + (int64_t)kCycWarp * R.n;
        B.count = R.nlist[kCycWarp];
        B.grab = grab_for(ctx, B.count);
        B.next = ctr + 2;
        PGD_LAUNCH(ctx, k_cycle_warp, warp_blocks(ctx, B.count, B.grab, 4), kWarpThreads, kWarpSmem, B);
    }
    PGD_CUDA(ctx, cudaEventRecord(ctx->evh1, ctx->stream));
    PGD_CUDA(ctx, cudaGetLastError());
    return PGD_OK;
}

pgd_status pgd_rank_decompose(pgd_ctx *ctx, const pgd_rank_graph &R, const pgd_rank_out &out) {
    cudaStream_t s = ctx->stream;
    pgd_status st;
    if (out.npos == 0 || R.nnz == 0) return PGD_OK;
    const int nsm = ctx->num_sms;
    // one allocation: counters, dk, t, cyc (zeroed), then the lists and tables, in
    // smaller ones where there is no room
    constexpr int kCounters = 16;   // [0..5) pass 1, [5..10) pass 2, [10..13) 4-cycles
    auto up128 = [](int64_t x) { return (x + 127) & ~(int64_t)127; };
    const int64_t zeroed = kCounters * 8 + R.nnz * 16, at_count = up128(zeroed);
    int64_t at_hits = 0, at_tables = 0;
    EgoMemory mem = ego_memory(ctx, R, INT64_MAX / 2);
    if (mem.bytes() > kListFloor || ctx->list_limit != UINT64_MAX) mem = ego_memory(ctx, R, ego_room(ctx));
    Tmp tg(ctx);
    uint8_t *work = nullptr;
    const std::string err = ctx->err;
    while (true) {
        at_hits = at_count + up128(mem.keep ? (int64_t)R.n2 * 4 : 0);
        at_tables = at_hits + up128(mem.hits * (int64_t)sizeof(uint2));
        st = tg.alloc(&work, (size_t)(at_tables + mem.gblocks * mem.table_bytes));
        const int64_t had = mem.bytes();
        if (st != PGD_ENOMEM || (mem = ego_memory(ctx, R, had / 4)).bytes() >= had) break;
        ctx->err = err;
    }
    if (st) return st;
    unsigned long long *ctr = (unsigned long long *)work, *dk = ctr + kCounters;
    uint32_t *t = (uint32_t *)(dk + R.nnz), *cyc = t + R.nnz;
    PGD_CUDA(ctx, cudaMemsetAsync(work, 0, zeroed, s));
    SideStream side(ctx);   // joined before tg frees
    PGD_CUDA(ctx, side.fork());
    CycArgs C{};
    C.roff = R.roff;
    C.rup = R.rup;
    C.radj = R.radj;
    C.wcode = R.wcode;
    C.tw = R.tw;
    C.bend = R.bend;
    C.bpos = R.bpos;
    C.n2 = R.n2;
    C.ranges = R.nranges;
    C.M = (const RankMeta *)R.meta;
    C.cyc = cyc;
    ctx->stream = ctx->side;
    st = cycle_pass(ctx, R, C, ctr + 10);
    ctx->stream = s;
    if (st) return st;
    EgoArgs E{};
    E.roff = R.roff;
    E.rup = R.rup;
    E.radj = R.radj;
    E.t = t;
    E.dk = dk;
    E.hits = mem.hits ? (uint2 *)(work + at_hits) : nullptr;
    E.hbase = R.hbase;
    E.hcount = mem.keep ? (uint32_t *)(work + at_count) : nullptr;
    PGD_CUDA(ctx, cudaEventRecord(ctx->evt0, s));
    ego_pass(ctx, R, E, 1, ctr, work + at_tables, mem);
    ego_pass(ctx, R, E, 2, ctr + 5, work + at_tables, mem);
    PGD_CUDA(ctx, cudaEventRecord(ctx->evt1, s));
    PGD_CUDA(ctx, side.join());
    CloseArgs Z;
    Z.o = out;
    Z.eslot = R.eslot;
    Z.tw = R.tw;
    Z.t = t;
    Z.dk = dk;
    Z.cyc = cyc;
    PGD_LAUNCH(ctx, k_rank_close, (int)std::min<int64_t>(grid_for(out.npos), 8 * (int64_t)nsm), kThreads, 0, Z);
    PGD_CUDA(ctx, cudaGetLastError());
    return PGD_OK;
}
