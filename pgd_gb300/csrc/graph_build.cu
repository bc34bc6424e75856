// graph_build.cu -- device-side graph construction and ordering.
//
// Replaces, on the GPU, the reference's host-side preparation of the graph:
//   read_* + remove_multiple_edges (graphlet_core.cpp:291-556)  -> pgd_build_from_pairs
//   the CSR constructor (graphlet_core.h:156-160)                -> pgd_build_from_csr
//   vertex_degrees (graphlet_core.cpp:877-891)                   -> k_degrees
//   order_vertex_neighbors + create_edge_list_arrays (:929-949, :1846-1953) -> pgd_dev_preprocess
//   compute_cores (:958-1018)                                    -> pgd_dev_cores (parallel peeling)
//   compute_assortativity (:1029-1057)                           -> pgd_dev_assortativity
//   sort_edges + get_ordering_value (:774-867)                   -> pgd_dev_sort_edges
//
// The compute CSR keeps every row sorted by neighbour id (what the
// decomposition kernels search).  The reference's own neighbour order only
// decides edge ids and hence the E_ordered tie-break; it is reproduced as a
// per-entry "insertion rank" and a segmented sort, never materialised.
#include <cub/cub.cuh>
#include <vector>

#include "cluster_ptx.cuh"
#include "pgd_internal.h"
#include "pgd_kernels.cuh"
#include "size_rules.h"

namespace {

constexpr int kThreads = 256;

inline int grid_for(int64_t n, int per_block = kThreads, int cap = 1 << 20) {
    int64_t g = (n + per_block - 1) / per_block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

// ---------------------------------------------------------------------------
// Edge-pair intake.

__global__ void k_pair_stats(const int32_t *src, const int32_t *dst, int64_t k, int *max_id,
                             unsigned long long *self_loops, unsigned long long *bad) {
    int local_max = -1;
    unsigned long long loops = 0, nbad = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x) {
        int a = src[i], b = dst[i];
        if (a < 0 || b < 0) { nbad++; continue; }
        if (a == b) { loops++; continue; }
        local_max = max(local_max, max(a, b));
    }
    for (int o = 16; o > 0; o >>= 1) {
        local_max = max(local_max, __shfl_xor_sync(0xffffffffu, local_max, o));
        loops += __shfl_xor_sync(0xffffffffu, loops, o);
        nbad += __shfl_xor_sync(0xffffffffu, nbad, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (local_max >= 0) atomicMax(max_id, local_max);
        if (loops) atomicAdd(self_loops, loops);
        if (nbad) atomicAdd(bad, nbad);
    }
}

// Pair i -> directed entries 2i (a->b) and 2i+1 (b->a) as row << cb | col, both
// carrying i as their insertion rank (vals may be null).  Self loops get a key
// that sorts after every edge.
__global__ void k_make_entries(const int32_t *src, const int32_t *dst, int64_t k, uint64_t sentinel, int cb,
                               uint64_t *keys, uint32_t *vals) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t a = (uint32_t)src[i], b = (uint32_t)dst[i];
        uint64_t k0 = sentinel, k1 = sentinel;
        if (a != b) {
            k0 = ((uint64_t)a << cb) | b;
            k1 = ((uint64_t)b << cb) | a;
        }
        *(ulonglong2 *)(keys + 2 * i) = ulonglong2{k0, k1};
        if (vals) *(uint2 *)(vals + 2 * i) = make_uint2((uint32_t)i, (uint32_t)i);
    }
}

// CSR input -> entries (row << cb | col), rank = position in the input.
__global__ void k_csr_entries(const int64_t *off, const int32_t *adj, int64_t n, int64_t nnz, int cb, uint64_t *keys,
                              uint32_t *vals, unsigned long long *bad) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x) {
        // row of position j: last r with off[r] <= j
        int64_t lo = 0, hi = n;  // off[lo] <= j < off[hi]
        while (hi - lo > 1) {
            int64_t mid = (lo + hi) >> 1;
            if (off[mid] <= j) lo = mid; else hi = mid;
        }
        int32_t c = adj[j];
        if (c < 0 || c >= n || c == lo) atomicAdd(bad, 1ull);
        keys[j] = ((uint64_t)(uint32_t)lo << cb) | (uint32_t)c;
        vals[j] = (uint32_t)j;
    }
}

// first-of-run flags over the sorted valid prefix (and a 0 behind it)
__global__ void k_unique_flags(const uint64_t *keys, int64_t valid, uint32_t *flags) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= valid; i += (int64_t)gridDim.x * blockDim.x)
        flags[i] = i < valid && (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

__global__ void k_scatter_unique(const uint64_t *keys, const uint32_t *vals, const uint32_t *flags,
                                 const uint32_t *pos, int64_t valid, int cb, int32_t *adj, int64_t *rank,
                                 int32_t *row) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < valid; i += (int64_t)gridDim.x * blockDim.x) {
        if (!flags[i]) continue;
        uint32_t p = pos[i];
        adj[p] = (int32_t)(keys[i] & ((1ull << cb) - 1));
        row[p] = (int32_t)(keys[i] >> cb);
        if (rank) rank[p] = vals[i];
    }
}

// off[r] = first entry of row r; rows without entries point at the next one.
__global__ void k_offsets(const int32_t *row, int64_t nnz, int64_t n, int64_t *off) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= nnz; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = (i < nnz) ? row[i] : n;
        int64_t rp = (i == 0) ? -1 : row[i - 1];
        for (int64_t x = rp + 1; x <= r; x++) off[x] = i;
    }
}

// Degrees and their maximum (*max_deg starts at 0).
__global__ void k_degrees(const int64_t *off, int64_t n, int32_t *deg, int *max_deg) {
    int top = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int d = (int)(off[v + 1] - off[v]);
        deg[v] = d;
        top = max(top, d);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0 && top > 0) atomicMax(max_deg, top);
}

// Per-vertex sum over neighbours of f(x), one warp per vertex.
// mode 0: degree (2-hop volume), 1: kcore1, 2: degree * kcore1.
__global__ void k_neigh_sum(const int64_t *off, const int32_t *adj, const int32_t *deg, const int32_t *core,
                            int64_t n, int mode, uint64_t *out) {
    int lane = threadIdx.x & 31;
    int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t v = w; v < n; v += nw) {
        uint64_t s = 0;
        for (int64_t j = off[v] + lane; j < off[v + 1]; j += 32) {
            int32_t x = adj[j];
            long long d = deg[x];
            long long k1 = (mode == 0) ? 0 : (x >= 1 ? core[x - 1] : 0);
            s += (uint64_t)(mode == 0 ? d : (mode == 1 ? k1 : d * k1));
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[v] = s;
    }
}

// Symmetry check for CSR input: (r,c) needs (c,r).
__global__ void k_check_symmetric(const int64_t *off, const int32_t *adj, const int32_t *row, int64_t nnz,
                                  unsigned long long *bad) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x) {
        int32_t r = row[j], c = adj[j];
        int64_t lo = off[c], hi = off[c + 1];
        while (lo < hi) {
            int64_t mid = (lo + hi) >> 1;
            if (adj[mid] < r) lo = mid + 1; else hi = mid;
        }
        if (lo >= off[c + 1] || adj[lo] != r) atomicAdd(bad, 1ull);
    }
}

__global__ void k_rows_of(const int64_t *off, int64_t n, int64_t nnz, int32_t *row) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x) {
        int64_t lo = 0, hi = n;
        while (hi - lo > 1) {
            int64_t mid = (lo + hi) >> 1;
            if (off[mid] <= j) lo = mid; else hi = mid;
        }
        row[j] = (int32_t)lo;
    }
}

// ---------------------------------------------------------------------------
// Neighbour order and edge ids.

// The entries above the diagonal in CSR order, each as one word that sorts into
// the order in which edges get their ids: by row, then by neighbour key, then by
// insertion rank, key and rank descending unless s2l (see k_neigh_keys).  vals
// gets the other endpoint.
template <typename K>
__global__ void k_neigh_words(const int64_t *off, const int32_t *adj, const int64_t *rank, const int32_t *deg,
                              const int32_t *core, const uint32_t *first, const uint32_t *base, int64_t n, int64_t nnz,
                              int kind, int descending, int db, int kb, K *keys, int32_t *vals) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; p0 < nnz; p0 += stride) {
        const int64_t p = min(p0 + lane, nnz - 1);
        const int64_t r = pgd_slot_row(off, n, p0, min(p0 + 31, nnz - 1), p, lane);
        const uint32_t f = first[r];
        if (p0 + lane >= nnz || (uint32_t)p < f) continue;
        const uint32_t i = base[r] + ((uint32_t)p - f);
        const int32_t c = adj[p];
        uint64_t key = 0;
        if (kind == PGD_NEIGH_DEG) key = (uint32_t)deg[c];
        else if (kind == PGD_NEIGH_KCORE) key = (uint32_t)(c >= 1 ? core[c - 1] : 0);
        uint64_t lo = (key << kb) | (uint64_t)rank[p];
        if (descending) lo = ((1ull << (db + kb)) - 1) - lo;
        keys[i] = (K)(((uint64_t)r << (db + kb)) | lo);
        vals[i] = c;
    }
}

// create_edge_list_arrays (graphlet_core.cpp:929-949) on the sorted words: e_v is
// the endpoint with the smaller degree, ties go to the larger id.
template <typename K>
__global__ void k_edge_assign(const K *keys, const int32_t *vals, const int32_t *deg, int64_t m, int shift, int32_t *ev,
                              int32_t *eu) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t r = (int32_t)((uint64_t)keys[i] >> shift), c = vals[i];
        const bool low = deg[r] < deg[c];
        ev[i] = low ? r : c;
        eu[i] = low ? c : r;
    }
}

// Composite within-row sort key: (neighbour key, insertion rank).  The
// reference's stable counting sort followed by a reversal
// (graphlet_core.cpp:1867-1875) orders a row by key descending with ties in
// reverse insertion order; --s2l_neigh keeps key ascending, ties in order.
__global__ void k_neigh_keys(const int32_t *adj, const int64_t *rank, const int32_t *deg, const int32_t *core,
                             int64_t nnz, int kind, uint64_t *keys, uint32_t *idx) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x) {
        int32_t c = adj[j];
        uint32_t key = 0;
        if (kind == PGD_NEIGH_DEG) key = (uint32_t)deg[c];
        else if (kind == PGD_NEIGH_KCORE) key = (uint32_t)(c >= 1 ? core[c - 1] : 0);
        keys[j] = ((uint64_t)key << 33) | (uint64_t)rank[j];
        idx[j] = (uint32_t)j;
    }
}

__global__ void k_edge_flags(const int32_t *row, const int32_t *adj, const uint32_t *perm, int64_t nnz,
                             uint32_t *flags) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x)
        flags[j] = (row[j] < adj[perm[j]]) ? 1u : 0u;
}

// create_edge_list_arrays (graphlet_core.cpp:929-949): e_v is the endpoint
// with the smaller degree, ties go to the larger id.
__global__ void k_edge_arrays(const int32_t *row, const int32_t *adj, const int32_t *deg, const uint32_t *perm,
                              const uint32_t *flags, const uint32_t *ids, int64_t nnz, int32_t *ev, int32_t *eu) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x) {
        if (!flags[j]) continue;
        int32_t r = row[j], c = adj[perm[j]];
        uint32_t id = ids[j];
        if (deg[r] < deg[c]) { ev[id] = r; eu[id] = c; }
        else { ev[id] = c; eu[id] = r; }
    }
}

// ---------------------------------------------------------------------------
// k-core peeling.  core[v] = -1 while v is alive.

__global__ void k_core_init(const int32_t *deg, int64_t n, int32_t *cur, int32_t *core, int32_t *alive) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        cur[v] = deg[v];
        core[v] = -1;
        alive[v] = (int32_t)v;
    }
}

__global__ void k_max_core(const int32_t *core, int64_t n_minus_1, int *out) {
    int local = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n_minus_1; v += (int64_t)gridDim.x * blockDim.x)
        local = max(local, core[v]);
    for (int o = 16; o > 0; o >>= 1) local = max(local, __shfl_xor_sync(0xffffffffu, local, o));
    if ((threadIdx.x & 31) == 0 && local > 0) atomicMax(out, local);
}

// ---------------------------------------------------------------------------
// Assortativity: int degree products as in the reference, double sums in a
// fixed order (block partials, then one block), so the result is repeatable.

__global__ void k_assort_partial(const int32_t *ev, const int32_t *eu, const int32_t *deg, int64_t m,
                                 double *partial) {
    __shared__ double s[3][kThreads / 32];
    double mu = 0, jd = 0, psi = 0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        unsigned dv = (unsigned)deg[ev[e]], du = (unsigned)deg[eu[e]];
        int p = (int)(dv * du);
        int q = (int)(dv * dv + du * du);
        mu += (double)p;
        jd += 0.5 * (double)(int)(dv + du);
        psi += 0.5 * (double)q;
    }
    for (int o = 16; o > 0; o >>= 1) {
        mu += __shfl_xor_sync(0xffffffffu, mu, o);
        jd += __shfl_xor_sync(0xffffffffu, jd, o);
        psi += __shfl_xor_sync(0xffffffffu, psi, o);
    }
    int wid = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) { s[0][wid] = mu; s[1][wid] = jd; s[2][wid] = psi; }
    __syncthreads();
    if (threadIdx.x < 3) {
        double t = 0;
        for (int i = 0; i < kThreads / 32; i++) t += s[threadIdx.x][i];
        partial[3 * blockIdx.x + threadIdx.x] = t;
    }
}

// ---------------------------------------------------------------------------
// Edge keys for sort_edges (graphlet_core.cpp:774-834).  The key is stored as
// int (Vertex, graphlet_vertex.h:42); order is key then id, id always
// descending (decr_bound / incr_bound, graphlet_vertex.h:57-75).

// The key of edge e (position i of the natural order), as the reference's int.
__device__ __forceinline__ int32_t edge_key(const int32_t *ev, const int32_t *eu, const int32_t *deg,
                                            const int32_t *core, const uint64_t *vsum, int64_t e, int64_t i, int kind) {
    const int32_t v = ev[e], u = eu[e];
    long long val = i;
    // core[] exists only for the k-core keys
    const bool kc = kind == PGD_ORD_KCORE || kind == PGD_ORD_KCORE_DEG;
    const int kv = (kc && v >= 1) ? core[v - 1] : 0, ku = (kc && u >= 1) ? core[u - 1] : 0;
    switch (kind) {
    case PGD_ORD_DEG: val = deg[u] + deg[v]; break;
    case PGD_ORD_KCORE: val = ku + kv; break;
    case PGD_ORD_KCORE_DEG: val = (int)((unsigned)(deg[u] + deg[v]) * (unsigned)(ku + kv)); break;
    case PGD_ORD_DEG_VOL:
    case PGD_ORD_KCORE_VOL:
    case PGD_ORD_KCORE_DEG_VOL: val = (long long)(vsum[u] + vsum[v]); break;
    case PGD_ORD_DEG_U: val = deg[u]; break;
    default: break;
    }
    return (int32_t)val;
}

// Every edge, last id first, with its key: a stable sort by the key alone then
// leaves ties in descending id order.  The sign bit is flipped where keys may
// be negative (32-bit keys), so that they sort as unsigned.
__global__ void k_edge_keys(const int32_t *ev, const int32_t *eu, const int32_t *deg, const int32_t *core,
                            const uint64_t *vsum, int64_t m, int kind, uint32_t flip, uint32_t *keys, int32_t *ids) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = m - 1 - i;
        keys[i] = (uint32_t)edge_key(ev, eu, deg, core, vsum, e, e, kind) ^ flip;
        ids[i] = (int32_t)e;
    }
}

// The sampled edge ids ids[0..count) (sort_edges with E_s, graphlet_core.cpp:
// 836-851; the natural key is the position in the sample): key above idb bits
// of the id, so that one sort orders by both.
__global__ void k_sample_keys(const int32_t *ev, const int32_t *eu, const int32_t *deg, const int32_t *core,
                              const uint64_t *vsum, const int32_t *ids, int64_t count, int kind, int s2l, uint32_t flip,
                              int idb, uint64_t *keys) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t e = (uint64_t)ids[i];
        const uint32_t k = (uint32_t)edge_key(ev, eu, deg, core, vsum, (int64_t)e, i, kind) ^ flip;
        keys[i] = ((uint64_t)k << idb) | (s2l ? ((1ull << idb) - 1 - e) : e);
    }
}

__global__ void k_keys_to_ids(const uint64_t *keys, int64_t m, int s2l, int idb, int32_t *order) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t lo = keys[e] & ((1ull << idb) - 1);
        order[e] = (int32_t)(s2l ? ((1ull << idb) - 1 - lo) : lo);
    }
}

}  // namespace

// ---------------------------------------------------------------------------

// The CSR of the sorted entries (row << cb | col), of which the first `valid` are
// edges.  vals (insertion ranks, below rank_limit) may be null: the graph then
// keeps none.
static pgd_status finish_csr(pgd_graph *g, uint64_t *keys, uint32_t *vals, int64_t valid, int cb, int64_t rank_limit,
                             bool dedup, bool csr_input) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    uint32_t *flags = nullptr, *pos = nullptr;
    int32_t *row = nullptr;
    pgd_status st;
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, flags, pos, (int64_t)valid + 1, s);
    const size_t vb = (valid + 1) * sizeof(uint32_t);
    pgd_pieces P;
    P.add(vb); P.add(vb); P.add(vb); P.add(tb);
    void *work = nullptr;
    if ((st = pgd_tmp_alloc(ctx, &work, P.bytes))) return st;
    struct Free {
        pgd_ctx *ctx;
        void *p;
        ~Free() { pgd_tmp_free(ctx, p); }
    } guard{ctx, work};
    P.base = (uint8_t *)work;
    flags = P.take<uint32_t>(vb);
    pos = P.take<uint32_t>(vb);
    row = P.take<int32_t>(vb);
    void *tmp = P.take<void>(tb);
    PGD_LAUNCH(ctx, k_unique_flags, grid_for(valid + 1), kThreads, 0, keys, valid, flags);
    PGD_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, tb, flags, pos, (int64_t)valid + 1, s));
    PGD_CUDA(ctx, pgd_fetch(ctx, 0, pos + valid, sizeof(uint32_t)));
    PGD_CUDA(ctx, cudaStreamSynchronize(s));
    const int64_t nnz = pgd_pinned<uint32_t>(ctx, 0);
    if (nnz != valid) {
        if (!dedup) {
            return pgd_fail(ctx, PGD_EINVAL, csr_input ? "CSR row lists a neighbour twice"
                                                       : "repeated pair without PGD_EDGES_DEDUP (multigraph input)");
        }
        g->duplicates = (valid - nnz) / 2;
    }
    g->m = nnz / 2;
    g->rank_limit = rank_limit;
    if ((st = pgd_graph_alloc(g, (void **)&g->adj, (nnz + 1) * sizeof(int32_t)))) return st;
    if (vals && (st = pgd_graph_alloc(g, (void **)&g->rank, (nnz + 1) * sizeof(int64_t)))) return st;
    if ((st = pgd_graph_alloc(g, (void **)&g->off, (g->n + 1) * sizeof(int64_t)))) return st;
    if ((st = pgd_graph_alloc(g, (void **)&g->deg, (g->n + 1) * sizeof(int32_t)))) return st;
    if (vals && (st = pgd_graph_alloc(g, (void **)&g->vol2, (g->n + 1) * sizeof(uint64_t)))) return st;
    // [0] the maximum degree, [1] entries without their reverse
    unsigned long long *ctr = ctx->d_ctr;
    PGD_CUDA(ctx, cudaMemsetAsync(ctr, 0, 2 * sizeof(unsigned long long), s));
    PGD_LAUNCH(ctx, k_scatter_unique, grid_for(valid), kThreads, 0, keys, vals, flags, pos, valid, cb, g->adj, g->rank,
               row);
    PGD_LAUNCH(ctx, k_offsets, grid_for(nnz + 1), kThreads, 0, row, nnz, g->n, g->off);
    PGD_LAUNCH(ctx, k_degrees, grid_for(g->n), kThreads, 0, g->off, g->n, g->deg, (int *)ctr);
    if (csr_input && nnz > 0)
        PGD_LAUNCH(ctx, k_check_symmetric, grid_for(nnz), kThreads, 0, g->off, g->adj, row, nnz, ctr + 1);
    PGD_CUDA(ctx, pgd_fetch(ctx, 0, ctr, 2 * sizeof(unsigned long long)));
    PGD_CUDA(ctx, cudaStreamSynchronize(s));
    if (pgd_pinned<unsigned long long>(ctx, 8))
        return pgd_fail(ctx, PGD_EINVAL, "CSR is not symmetric (undirected graphs list each edge both ways)");
    g->max_degree = pgd_pinned<int32_t>(ctx, 0);
    PGD_CUDA(ctx, cudaGetLastError());
    return PGD_OK;
}

// ---------------------------------------------------------------------------
// Small graphs: each stage by one block.

namespace {

struct SmallResult {
    int nnz, max_degree, loops;
};

// CSR of k <= kSmallPairs pairs (ids below n): words of row, column and pair index
// (ib bits) sorted in shared memory, the first of each run kept.
__global__ void __launch_bounds__(kSmallThreads) k_small_build(const int32_t *src, const int32_t *dst, int k, int n,
                                                               int cb, int ib, int P, int64_t *off, int32_t *adj,
                                                               int64_t *rank, int32_t *deg, SmallResult *out) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    uint64_t *w = (uint64_t *)s_dyn;
    __shared__ int sh[33], s_loops, s_max;
    if (threadIdx.x == 0) s_loops = s_max = 0;
    __syncthreads();
    for (int i = threadIdx.x; 2 * i < P; i += kSmallThreads) {
        uint64_t x = ~0ull, y = ~0ull;
        if (i < k) {
            const uint64_t a = (uint32_t)src[i], b = (uint32_t)dst[i];
            if (a != b) {
                x = (a << (cb + ib)) | (b << ib) | (uint64_t)i;
                y = (b << (cb + ib)) | (a << ib) | (uint64_t)i;
            } else {
                atomicAdd(&s_loops, 1);
            }
        }
        w[2 * i] = x;
        w[2 * i + 1] = y;
    }
    __syncthreads();
    pgd_block_sort(w, P);
    // each thread a contiguous part: its runs' first words, counted then written
    const int per = (P + kSmallThreads - 1) / kSmallThreads, b0 = min(P, (int)threadIdx.x * per), b1 = min(P, b0 + per);
    auto first = [&](int i) { return w[i] != ~0ull && (i == 0 || (w[i] >> ib) != (w[i - 1] >> ib)); };
    int c = 0, total = 0;
    for (int i = b0; i < b1; i++) c += first(i);
    int at = pgd_block_excl_scan(c, sh, &total);
    for (int i = b0; i < b1; i++) {
        if (!first(i)) continue;
        const int r = (int)(w[i] >> (cb + ib)), rp = i == 0 ? -1 : (int)(w[i - 1] >> (cb + ib));
        adj[at] = (int32_t)((w[i] >> ib) & ((1ull << cb) - 1));
        rank[at] = (int64_t)(w[i] & ((1ull << ib) - 1));
        for (int x = rp + 1; x <= r; x++) off[x] = at;
        at++;
    }
    // rows behind the last one with entries (the sentinels' row id is beyond n)
    const int valid = 2 * (k - s_loops);
    const int last = valid > 0 ? (int)(w[valid - 1] >> (cb + ib)) : -1;
    for (int x = last + 1 + (int)threadIdx.x; x <= n; x += kSmallThreads) off[x] = total;
    __syncthreads();
    int top = 0;
    for (int v = threadIdx.x; v < n; v += kSmallThreads) {
        const int d = (int)(off[v + 1] - off[v]);
        deg[v] = d;
        top = max(top, d);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0 && top > 0) atomicMax(&s_max, top);
    __syncthreads();
    if (threadIdx.x == 0) *out = SmallResult{total, s_max, s_loops};
}

// Edge arrays of a small graph: as k_neigh_words, one sort and k_edge_assign, with
// the other endpoint (cb bits) in the word.
__global__ void __launch_bounds__(kSmallThreads) k_small_edges(const int64_t *off, const int32_t *adj,
                                                               const int64_t *rank, const int32_t *deg,
                                                               const int32_t *core, int n, int nnz, int m, int kind,
                                                               int descending, int db, int kb, int cb, int P,
                                                               int32_t *ev, int32_t *eu) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    uint64_t *w = (uint64_t *)s_dyn;
    __shared__ int s_count;
    if (threadIdx.x == 0) s_count = 0;
    for (int i = m + (int)threadIdx.x; i < P; i += kSmallThreads) w[i] = ~0ull;
    __syncthreads();
    for (int p = threadIdx.x; p < nnz; p += kSmallThreads) {
        int lo = 0, hi = n;   // last row with off <= p
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (off[mid] <= p) lo = mid;
            else hi = mid;
        }
        const int32_t c = adj[p];
        if (c <= lo) continue;
        uint64_t key = 0;
        if (kind == PGD_NEIGH_DEG) key = (uint32_t)deg[c];
        else if (kind == PGD_NEIGH_KCORE) key = (uint32_t)(c >= 1 ? core[c - 1] : 0);
        uint64_t x = (key << kb) | (uint64_t)rank[p];
        if (descending) x = ((1ull << (db + kb)) - 1) - x;
        w[atomicAdd(&s_count, 1)] = ((((uint64_t)lo << (db + kb)) | x) << cb) | (uint64_t)c;
    }
    __syncthreads();
    pgd_block_sort(w, P);
    for (int i = threadIdx.x; i < m; i += kSmallThreads) {
        const int32_t r = (int32_t)(w[i] >> (db + kb + cb)), c = (int32_t)(w[i] & ((1ull << cb) - 1));
        const bool low = deg[r] < deg[c];
        ev[i] = low ? r : c;
        eu[i] = low ? c : r;
    }
}

// E_ordered of a small graph: (key, id) words, key descending unless s2l, ties by
// descending id.
__global__ void __launch_bounds__(kSmallThreads) k_small_order(const int32_t *ev, const int32_t *eu, const int32_t *deg,
                                                               const int32_t *core, const uint64_t *vsum, int m,
                                                               int kind, int s2l, int P, int32_t *order) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    uint64_t *w = (uint64_t *)s_dyn;
    for (int e = threadIdx.x; e < P; e += kSmallThreads) {
        uint64_t x = ~0ull;
        if (e < m) {
            uint32_t key = (uint32_t)edge_key(ev, eu, deg, core, vsum, e, e, kind) ^ 0x80000000u;
            if (!s2l) key = ~key;
            x = ((uint64_t)key << 16) | (uint64_t)(0xfffe - e);   // m < 65535; all ones stays last
        }
        w[e] = x;
    }
    __syncthreads();
    pgd_block_sort(w, P);
    for (int i = threadIdx.x; i < m; i += kSmallThreads) order[i] = 0xfffe - (int32_t)(w[i] & 0xffff);
}

}  // namespace

// A graph of at most kSmallPairs host pairs with ids below n: the pairs go through
// the context's page-locked buffer, which the kernel reads and answers in.
static pgd_status build_small(pgd_graph *g, const int32_t *h_src, const int32_t *h_dst, int64_t k, int64_t n, bool dedup) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    pgd_status st;
    // the buffer's last use was waited for (every fetch is); its second half holds the pairs
    int32_t *p_src = (int32_t *)(ctx->pin + kPinBytes / 2), *p_dst = p_src + kSmallPairs;
    memcpy(p_src, h_src, k * sizeof(int32_t));
    memcpy(p_dst, h_dst, k * sizeof(int32_t));
    g->n = n;
    g->rank_limit = k;
    if ((st = pgd_graph_alloc(g, (void **)&g->off, (n + 1) * sizeof(int64_t)))) return st;
    if ((st = pgd_graph_alloc(g, (void **)&g->deg, (n + 1) * sizeof(int32_t)))) return st;
    if ((st = pgd_graph_alloc(g, (void **)&g->vol2, (n + 1) * sizeof(uint64_t)))) return st;
    // entries: room for every pair, counted against the budget by what is kept
    int32_t *adj = nullptr;
    int64_t *rank = nullptr;
    if ((st = pgd_tmp_alloc(ctx, (void **)&adj, (2 * k + 1) * sizeof(int32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&rank, (2 * k + 1) * sizeof(int64_t)))) {
        pgd_tmp_free(ctx, adj);
        return st;
    }
    g->adj = adj;
    g->rank = rank;
    const int cb = std::max(1, pgd_bit_length((uint64_t)n)), ib = std::max(1, pgd_bit_length((uint64_t)k));
    const int P = pgd_small_words(2 * k);
    PGD_LAUNCH(ctx, k_small_build, 1, kSmallThreads, P * sizeof(uint64_t), p_src, p_dst, (int)k, (int)n, cb, ib, P, g->off,
               adj, rank, g->deg, (SmallResult *)ctx->pin);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    const SmallResult r = e == cudaSuccess ? pgd_pinned<SmallResult>(ctx, 0) : SmallResult{0, 0, 0};
    const int64_t valid = 2 * (k - r.loops);
    g->m = r.nnz / 2;
    const uint64_t bytes = (2 * (uint64_t)g->m + 1) * (sizeof(int32_t) + sizeof(int64_t));
    ctx->resident += bytes;
    g->bytes += bytes;
    if (e != cudaSuccess) return pgd_cuda_fail(ctx, e, "build of a small graph");
    if (ctx->resident > ctx->budget)
        return pgd_fail(ctx, PGD_ENOMEM, "HBM budget of the context exceeded (" + std::to_string(ctx->resident) + " > " +
                                             std::to_string(ctx->budget) + " bytes)");
    g->self_loops = r.loops;
    g->max_degree = r.max_degree;
    if (r.nnz != valid) {
        if (!dedup) return pgd_fail(ctx, PGD_EINVAL, "repeated pair without PGD_EDGES_DEDUP (multigraph input)");
        g->duplicates = (valid - r.nnz) / 2;
    }
    return PGD_OK;
}

// 16-byte words from a mapped host source, then the tail bytes
__global__ void k_copy_mapped(const uint4 *src, uint4 *dst, int64_t n16, const uint8_t *src_tail, uint8_t *dst_tail,
                              int tail) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n16; i += stride) dst[i] = src[i];
    if (blockIdx.x == 0 && threadIdx.x < tail) dst_tail[threadIdx.x] = src_tail[threadIdx.x];
}

cudaError_t pgd_h2d(pgd_ctx *ctx, void *dst, const void *src, size_t bytes) {
    if (!bytes) return cudaSuccess;
    const void *v = pgd_device_view(src);
    if (!v || ((uintptr_t)v & 15) || ((uintptr_t)dst & 15))
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream);
    const int64_t n16 = (int64_t)(bytes / 16);
    const int tail = (int)(bytes % 16);
    k_copy_mapped<<<ctx->num_sms * 8, kThreads, 0, ctx->stream>>>((const uint4 *)v, (uint4 *)dst, n16,
                                                                   (const uint8_t *)v + 16 * n16,
                                                                   (uint8_t *)dst + 16 * n16, tail);
    ctx->launches++;
    return cudaGetLastError();
}

pgd_status pgd_build_from_pairs(pgd_graph *g, const int32_t *h_src, const int32_t *h_dst, int64_t k, int64_t n_min,
                                bool dedup) {
    pgd_ctx *ctx = g->ctx;
    if (k < 0 || k > (int64_t)0x7fffffff) return pgd_fail(ctx, PGD_EINVAL, "pair count out of range (0..2^31-1)");
    pgd_status st;
    if (k > 0 && k <= kSmallPairs) {
        // the host reads the pairs here: after what the caller's own stream still has
        // to do, which may be what fills them (page-locked memory)
        if (!ctx->own_stream) PGD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        int32_t top = -1;   // largest id of an edge
        bool bad = false;
        for (int64_t i = 0; i < k; i++) {
            bad |= (h_src[i] | h_dst[i]) < 0;
            if (h_src[i] != h_dst[i]) top = std::max(top, std::max(h_src[i], h_dst[i]));
        }
        if (bad) return pgd_fail(ctx, PGD_EINVAL, "negative vertex id in edge list");
        const int64_t n = std::max<int64_t>(n_min, (int64_t)top + 1);
        if (n > 0 && n <= kSmallVertices) return build_small(g, h_src, h_dst, k, n, dedup);
    }
    int32_t *d_src = nullptr;
    const int64_t k1 = ((k > 0 ? k : 1) + 63) & ~(int64_t)63;   // both halves 256-byte aligned
    if ((st = pgd_tmp_alloc(ctx, (void **)&d_src, 2 * k1 * sizeof(int32_t)))) return st;
    int32_t *d_dst = d_src + k1;
    cudaError_t e = cudaSuccess;
    if (k > 0) {
        e = pgd_h2d(ctx, d_src, h_src, k * sizeof(int32_t));
        if (e == cudaSuccess) e = pgd_h2d(ctx, d_dst, h_dst, k * sizeof(int32_t));
    }
    st = e == cudaSuccess ? pgd_build_from_device_pairs(g, d_src, d_dst, k, n_min, dedup)
                          : pgd_cuda_fail(ctx, e, "upload of the pairs");
    pgd_tmp_free(ctx, d_src);
    return st;
}

pgd_status pgd_build_from_device_pairs(pgd_graph *g, const int32_t *d_src, const int32_t *d_dst, int64_t k,
                                       int64_t n_min, bool dedup, bool ranks) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    if (k < 0 || k > (int64_t)0x7fffffff) return pgd_fail(ctx, PGD_EINVAL, "pair count out of range (0..2^31-1)");
    pgd_status st;
    // stats: [0] max id (int), [1] self loops, [2] bad ids
    unsigned long long *stats = ctx->d_ctr;
    PGD_CUDA(ctx, cudaMemsetAsync(stats, 0, 3 * sizeof(unsigned long long), s));
    PGD_CUDA(ctx, cudaMemsetAsync(stats, 0xff, sizeof(int), s));  // max id = -1
    if (k > 0)
        PGD_LAUNCH(ctx, k_pair_stats, (int)std::min<int64_t>(grid_for(k), 8 * (int64_t)ctx->num_sms), kThreads, 0,
                   d_src, d_dst, k, (int *)stats, stats + 1, stats + 2);
    PGD_CUDA(ctx, pgd_fetch(ctx, 0, stats, 3 * sizeof(unsigned long long)));
    PGD_CUDA(ctx, cudaStreamSynchronize(s));
    const int64_t max_id = pgd_pinned<int>(ctx, 0);
    if (pgd_pinned<unsigned long long>(ctx, 16)) return pgd_fail(ctx, PGD_EINVAL, "negative vertex id in edge list");
    g->self_loops = pgd_pinned<int64_t>(ctx, 8);
    g->n = std::max<int64_t>(n_min, max_id + 1);
    // vertices are kept as 32-bit numbers from 0
    if (g->n > (int64_t)1 << 31) {
        g->n = 0;
        return pgd_fail(ctx, PGD_EINVAL, "vertex count out of range (0..2^31)");
    }
    const int64_t valid = 2 * (k - g->self_loops), ne = 2 * k;
    // a word holds row and column on the bits that ids up to max_id + 1 need
    const int cb = pgd_id_bits(max_id);
    const uint64_t sentinel = (uint64_t)(max_id + 1) << cb;
    uint64_t *keys = nullptr, *keys2 = nullptr;
    uint32_t *vals = nullptr, *vals2 = nullptr;
    size_t tb = 0;
    if (ranks) cub::DeviceRadixSort::SortPairs(nullptr, tb, keys, keys2, vals, vals2, ne, 0, 2 * cb, s);
    else cub::DeviceRadixSort::SortKeys(nullptr, tb, keys, keys2, ne, 0, 2 * cb, s);
    const size_t kbytes = ne * sizeof(uint64_t), vbytes = ranks ? ne * sizeof(uint32_t) : 0;
    pgd_pieces P1, P2;   // the inputs of the sort are freed after it, its outputs after the CSR is built
    P1.add(kbytes); P1.add(vbytes); P1.add(tb);
    P2.add(kbytes); P2.add(vbytes);
    void *w1 = nullptr, *w2 = nullptr;
    if ((st = pgd_tmp_alloc(ctx, &w1, P1.bytes))) return st;
    if ((st = pgd_tmp_alloc(ctx, &w2, P2.bytes))) {
        pgd_tmp_free(ctx, w1);
        return st;
    }
    P1.base = (uint8_t *)w1;
    P2.base = (uint8_t *)w2;
    keys = P1.take<uint64_t>(kbytes);
    keys2 = P2.take<uint64_t>(kbytes);
    if (ranks) {
        vals = P1.take<uint32_t>(vbytes);
        vals2 = P2.take<uint32_t>(vbytes);
    }
    void *tmp = P1.take<void>(tb);
    if (k > 0) {
        PGD_LAUNCH(ctx, k_make_entries, grid_for(k), kThreads, 0, d_src, d_dst, k, sentinel, cb, keys, vals);
        if (ranks) cub::DeviceRadixSort::SortPairs(tmp, tb, keys, keys2, vals, vals2, ne, 0, 2 * cb, s);
        else cub::DeviceRadixSort::SortKeys(tmp, tb, keys, keys2, ne, 0, 2 * cb, s);
    }
    pgd_tmp_free(ctx, w1);
    st = finish_csr(g, keys2, vals2, valid, cb, k, dedup, false);
    pgd_tmp_free(ctx, w2);
    return st;
}

pgd_status pgd_build_from_csr(pgd_graph *g, const int64_t *h_off, const int32_t *h_adj, int64_t n) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    if (n < 0 || n > (int64_t)0x7ffffffe) return pgd_fail(ctx, PGD_EINVAL, "vertex count out of range");
    if (h_off[0] != 0) return pgd_fail(ctx, PGD_EINVAL, "CSR offsets must start at 0");
    for (int64_t v = 0; v < n; v++)
        if (h_off[v + 1] < h_off[v]) return pgd_fail(ctx, PGD_EINVAL, "CSR offsets must not decrease");
    int64_t nnz = h_off[n];
    if (nnz > (int64_t)0x7fffffff) return pgd_fail(ctx, PGD_EINVAL, "too many CSR entries");
    g->n = n;
    pgd_status st;
    int64_t *d_off = nullptr;
    int32_t *d_adj = nullptr;
    uint64_t *keys = nullptr, *keys2 = nullptr;
    uint32_t *vals = nullptr, *vals2 = nullptr;
    int64_t nz1 = nnz > 0 ? nnz : 1;
    if ((st = pgd_tmp_alloc(ctx, (void **)&d_off, (n + 1) * sizeof(int64_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&d_adj, nz1 * sizeof(int32_t)))) return st;
    PGD_CUDA(ctx, cudaMemcpyAsync(d_off, h_off, (n + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, s));
    if (nnz) PGD_CUDA(ctx, cudaMemcpyAsync(d_adj, h_adj, nnz * sizeof(int32_t), cudaMemcpyHostToDevice, s));
    if ((st = pgd_tmp_alloc(ctx, (void **)&keys, nz1 * sizeof(uint64_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&keys2, nz1 * sizeof(uint64_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&vals, nz1 * sizeof(uint32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&vals2, nz1 * sizeof(uint32_t)))) return st;
    unsigned long long *bad = ctx->d_ctr;
    PGD_CUDA(ctx, cudaMemsetAsync(bad, 0, sizeof(unsigned long long), s));
    const int cb = std::max(1, pgd_bit_length((uint64_t)n));
    if (nnz) PGD_LAUNCH(ctx, k_csr_entries, grid_for(nnz), kThreads, 0, d_off, d_adj, n, nnz, cb, keys, vals, bad);
    unsigned long long h_bad = 0;
    PGD_CUDA(ctx, cudaMemcpyAsync(&h_bad, bad, sizeof(h_bad), cudaMemcpyDeviceToHost, s));
    PGD_CUDA(ctx, cudaStreamSynchronize(s));
    pgd_tmp_free(ctx, d_off);
    pgd_tmp_free(ctx, d_adj);
    if (h_bad) {
        pgd_tmp_free(ctx, keys); pgd_tmp_free(ctx, keys2); pgd_tmp_free(ctx, vals); pgd_tmp_free(ctx, vals2);
        return pgd_fail(ctx, PGD_EINVAL, "CSR neighbour id out of range or a self loop");
    }
    if (nnz) {
        const int end_bit = 2 * cb;
        size_t tb = 0;
        void *tmp = nullptr;
        cub::DeviceRadixSort::SortPairs(nullptr, tb, keys, keys2, vals, vals2, nnz, 0, end_bit, s);
        if ((st = pgd_tmp_alloc(ctx, &tmp, tb))) return st;
        cub::DeviceRadixSort::SortPairs(tmp, tb, keys, keys2, vals, vals2, nnz, 0, end_bit, s);
        pgd_tmp_free(ctx, tmp);
    }
    pgd_tmp_free(ctx, keys);
    pgd_tmp_free(ctx, vals);
    st = finish_csr(g, keys2, vals2, nnz, cb, nnz, false, true);
    pgd_tmp_free(ctx, keys2);
    pgd_tmp_free(ctx, vals2);
    return st;
}

// Edge ids by one sort of words of type K (rb bits of row, db of key, kb of rank).
template <typename K>
static pgd_status order_by_words(pgd_graph *g, int kind, bool descending, int rb, int db, int kb) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    pgd_status st;
    const int64_t n = g->n, m = g->m;
    uint32_t *first = nullptr, *count = nullptr, *base = nullptr;
    K *keys = nullptr;
    int32_t *vals = nullptr;
    size_t tb1 = 0, tb2 = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb1, first, first, n + 1, s);
    cub::DeviceRadixSort::SortPairs(nullptr, tb2, keys, keys, vals, vals, m, 0, rb + db + kb, s);
    const size_t nb = (n + 1) * sizeof(uint32_t), tb = std::max(tb1, tb2);
    pgd_pieces P;
    P.add(nb); P.add(nb); P.add(nb); P.add(2 * m * sizeof(K)); P.add(2 * m * sizeof(int32_t)); P.add(tb);
    void *work = nullptr;
    if ((st = pgd_tmp_alloc(ctx, &work, P.bytes))) return st;
    P.base = (uint8_t *)work;
    first = P.take<uint32_t>(nb);
    count = P.take<uint32_t>(nb);
    base = P.take<uint32_t>(nb);
    keys = P.take<K>(2 * m * sizeof(K));
    vals = P.take<int32_t>(2 * m * sizeof(int32_t));
    void *tmp = P.take<void>(tb);
    PGD_LAUNCH(ctx, pgd_upper_rows, grid_for(n + 1), kThreads, 0, g->off, g->adj, n, first, count);
    cub::DeviceScan::ExclusiveSum(tmp, tb1, count, base, n + 1, s);
    PGD_LAUNCH(ctx, k_neigh_words<K>, grid_for(2 * m), kThreads, 0, g->off, g->adj, g->rank, g->deg, g->core, first,
               base, n, 2 * m, kind, (int)descending, db, kb, keys, vals);
    cub::DeviceRadixSort::SortPairs(tmp, tb2, keys, keys + m, vals, vals + m, m, 0, rb + db + kb, s);
    PGD_LAUNCH(ctx, k_edge_assign<K>, grid_for(m), kThreads, 0, keys + m, vals + m, g->deg, m, db + kb, g->ev, g->eu);
    pgd_tmp_free(ctx, work);
    PGD_CUDA(ctx, cudaGetLastError());
    return PGD_OK;
}

pgd_status pgd_dev_preprocess(pgd_graph *g, int neigh_kind, int s2l) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    pgd_status st;
    int64_t nnz = 2 * g->m;
    if (!g->ev) {
        if ((st = pgd_graph_alloc(g, (void **)&g->ev, (g->m + 1) * sizeof(int32_t)))) return st;
        if ((st = pgd_graph_alloc(g, (void **)&g->eu, (g->m + 1) * sizeof(int32_t)))) return st;
    }
    if (nnz == 0) { g->preprocessed = true; return PGD_OK; }
    // The rank-ordered copy knows the edges by their ids (eslot), which change here.
    pgd_rank_drop(g);
    // One sort of the m entries above the diagonal by (row, key, rank) where a
    // 64-bit word holds them (32-bit where that does); else the rows' segments of
    // all 2m entries are sorted.
    const bool descend = (neigh_kind != PGD_NEIGH_ASREAD) && !s2l;
    const int rb = std::max(1, pgd_bit_length((uint64_t)g->n)), kb = std::max(1, pgd_bit_length((uint64_t)g->rank_limit));
    const int db = neigh_kind == PGD_NEIGH_ASREAD ? 0
                   : std::max(1, pgd_bit_length((uint64_t)(neigh_kind == PGD_NEIGH_DEG ? g->max_degree : g->max_core)));
    if (g->m <= kSmallPairs && g->n <= kSmallVertices && 2 * rb + db + kb <= 63) {
        const int P = pgd_small_words(g->m);
        PGD_LAUNCH(ctx, k_small_edges, 1, kSmallThreads, P * sizeof(uint64_t), g->off, g->adj, g->rank, g->deg, g->core,
                   (int)g->n, (int)nnz, (int)g->m, neigh_kind, (int)descend, db, kb, rb, P, g->ev, g->eu);
        PGD_CUDA(ctx, cudaGetLastError());
        g->preprocessed = true;
        g->sorted = false;
        g->has_micro = false;
        return PGD_OK;
    }
    if (rb + db + kb <= 64) {
        st = rb + db + kb <= 32 ? order_by_words<uint32_t>(g, neigh_kind, descend, rb, db, kb)
                                : order_by_words<uint64_t>(g, neigh_kind, descend, rb, db, kb);
        if (st) return st;
        g->preprocessed = true;
        g->sorted = false;
        g->has_micro = false;
        return PGD_OK;
    }
    int32_t *row = nullptr;
    uint64_t *keys = nullptr, *keys2 = nullptr;
    uint32_t *idx = nullptr, *perm = nullptr, *flags = nullptr, *ids = nullptr;
    if ((st = pgd_tmp_alloc(ctx, (void **)&row, nnz * sizeof(int32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&keys, nnz * sizeof(uint64_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&keys2, nnz * sizeof(uint64_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&idx, nnz * sizeof(uint32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&perm, nnz * sizeof(uint32_t)))) return st;
    PGD_LAUNCH(ctx, k_rows_of, grid_for(nnz), kThreads, 0, g->off, g->n, nnz, row);
    PGD_LAUNCH(ctx, k_neigh_keys, grid_for(nnz), kThreads, 0, g->adj, g->rank, g->deg, g->core, nnz, neigh_kind, keys, idx);
    bool descending = (neigh_kind != PGD_NEIGH_ASREAD) && !s2l;
    size_t tb = 0;
    void *tmp = nullptr;
    if (descending)
        cub::DeviceSegmentedSort::SortPairsDescending(nullptr, tb, keys, keys2, idx, perm, nnz, g->n, g->off,
                                                      g->off + 1, s);
    else
        cub::DeviceSegmentedSort::SortPairs(nullptr, tb, keys, keys2, idx, perm, nnz, g->n, g->off, g->off + 1, s);
    if ((st = pgd_tmp_alloc(ctx, &tmp, tb))) return st;
    if (descending)
        cub::DeviceSegmentedSort::SortPairsDescending(tmp, tb, keys, keys2, idx, perm, nnz, g->n, g->off,
                                                      g->off + 1, s);
    else
        cub::DeviceSegmentedSort::SortPairs(tmp, tb, keys, keys2, idx, perm, nnz, g->n, g->off, g->off + 1, s);
    pgd_tmp_free(ctx, tmp);
    pgd_tmp_free(ctx, keys);
    pgd_tmp_free(ctx, keys2);
    pgd_tmp_free(ctx, idx);
    if ((st = pgd_tmp_alloc(ctx, (void **)&flags, nnz * sizeof(uint32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&ids, nnz * sizeof(uint32_t)))) return st;
    PGD_LAUNCH(ctx, k_edge_flags, grid_for(nnz), kThreads, 0, row, g->adj, perm, nnz, flags);
    tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, flags, ids, nnz, s);
    if ((st = pgd_tmp_alloc(ctx, &tmp, tb))) return st;
    cub::DeviceScan::ExclusiveSum(tmp, tb, flags, ids, nnz, s);
    pgd_tmp_free(ctx, tmp);
    PGD_LAUNCH(ctx, k_edge_arrays, grid_for(nnz), kThreads, 0, row, g->adj, g->deg, perm, flags, ids, nnz, g->ev, g->eu);
    pgd_tmp_free(ctx, row);
    pgd_tmp_free(ctx, perm);
    pgd_tmp_free(ctx, flags);
    pgd_tmp_free(ctx, ids);
    PGD_CUDA(ctx, cudaGetLastError());
    g->preprocessed = true;
    g->sorted = false;
    g->has_micro = false;
    return PGD_OK;
}

// k-core of light graphs (pgd_core_light), and of others once their steps have
// become narrow (pgd_core_narrow): one cluster of sixteen blocks peels the graph in
// one launch.  What bounds it is the chain of steps (832 on R-MAT 20, 448 on R-MAT
// 16), each a few dependent L2 accesses and a barrier: the cluster's hardware
// barrier replaces two graph nodes per step (k_core_work and k_core_ctrl below,
// about 8 us together with their gaps), and no graph is captured and instantiated
// for the call (180 us).  Sixteen blocks rather than the portable eight for the
// steps that are not narrow: milliseconds of the whole call in the cluster with 8 /
// 16, R-MAT 20 12.1 / 8.0, BA of 400,000 2.8 / 2.0.
namespace {

constexpr int kCoreBlocks = 16;             // the largest cluster (beyond the portable eight)
constexpr int kCoreThreads = 1024;
static_assert(kCoreBlocks * kCoreThreads <= kCoreIndexRoom, "thread-strided loops over vertices stay below 2^31");
constexpr int kCoreLong = 1024;             // rows at least this long are shared by all warps

struct CoreSlot {
    unsigned int front, lng, alive;         // entries appended in this step
    int min_rest;                           // smallest count among the vertices left
};
struct CoreShared {
    CoreSlot slot[3];                       // by step modulo 3: written, read after the barrier, cleared a step later
    int max_core, failed;
};

__device__ __forceinline__ void core_append(bool in, int32_t v, int32_t *list, unsigned int *count, int lane) {
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (!m) return;
    unsigned at = 0;
    if (lane == 0) at = atomicAdd(count, (unsigned)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (in) list[at + __popc(m & ((1u << lane) - 1))] = v;
}

// visit(active, neighbour) over the rows of a frontier's entries 0..nf, by `warps`
// warps of which this is the w-th: as many vertices per warp as fill them (at
// most 32), whose offsets are then loaded together; rows of 64 or more entries
// one after the other, shorter ones flattened over the lanes.
// row(v, o, d) gives v's row.
template <typename Get, typename Row, typename Visit>
__device__ __forceinline__ void core_rows(const int32_t *adj, unsigned nf, int w, int warps, Get get, Row row,
                                          Visit visit) {
    const int lane = threadIdx.x & 31;
    const unsigned per = min(32u, max(1u, (nf + (unsigned)warps - 1) / (unsigned)warps));
    for (unsigned i0 = (unsigned)w * per; i0 < nf; i0 += (unsigned)warps * per) {
        int64_t o = 0;
        int d = 0;
        if ((unsigned)lane < per && i0 + lane < nf) {
            row(get(i0 + lane), o, d);
        }
        unsigned lm = __ballot_sync(0xffffffffu, d >= 64);
        while (lm) {
            const int src = __ffs(lm) - 1;
            lm &= lm - 1;
            const int64_t os = __shfl_sync(0xffffffffu, o, src);
            const int ds = __shfl_sync(0xffffffffu, d, src);
            for (int j = 0; j < ds; j += 128) {
                int32_t y[4];
#pragma unroll
                for (int k = 0; k < 4; k++) y[k] = j + 32 * k + lane < ds ? __ldg(adj + os + j + 32 * k + lane) : 0;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (j + 32 * k < ds) visit(j + 32 * k + lane < ds, y[k]);
            }
        }
        if (d >= 64) d = 0;
        const int incl = pgd_warp_incl_scan(d);
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        const int64_t first = o - (incl - d);   // slot = first + flattened index
        for (int b = 0; b < total; b += 64) {
            int32_t y[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int it = b + 32 * k + lane;
                int own = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, incl, own + step - 1) <= it) own += step;
                const int64_t f = __shfl_sync(0xffffffffu, first, own & 31);
                y[k] = it < total ? __ldg(adj + f + it) : 0;
            }
#pragma unroll
            for (int k = 0; k < 2; k++)
                if (b + 32 * k < total) visit(b + 32 * k + lane < total, y[k]);
        }
    }
}

// Where the cluster starts: at the beginning (na 0), or where the whole device
// left off: vertices alive, a frontier of nf vertices in f0 not yet peeled.
struct CoreStart {
    int level, removed;
    unsigned int na, nf;
};

// f and b: two buffers each of the frontier's short and long rows; a0, a1:
// vertices alive.  A level scan moves every alive vertex of count <= level to the
// frontier and the others to the other alive list; a peel round takes one off the
// count of the frontier's neighbours.
__global__ void __cluster_dims__(kCoreBlocks, 1, 1) __launch_bounds__(kCoreThreads, 1)
k_core_cluster(const int64_t *off, const int32_t *adj, const int32_t *deg, int n, int32_t *cur, int32_t *core,
               int32_t *f0, int32_t *f1, int32_t *b0, int32_t *b1, int32_t *a0, int32_t *a1, CoreShared *S,
               int max_degree, CoreStart at) {
    const int lane = threadIdx.x & 31;
    const int rank = (int)pgd_cl::cluster_rank();
    constexpr int kAll = kCoreBlocks * kCoreThreads;
    const int t = rank * kCoreThreads + (int)threadIdx.x, w = t >> 5;
    const int t0 = t - lane;
    if (at.na == 0)
        for (int v = t; v < n; v += kAll) {
            cur[v] = deg[v];
            core[v] = -1;
            a0[v] = v;
        }
    if (t == 0) {
        for (int i = 0; i < 3; i++) S->slot[i] = CoreSlot{0, 0, 0, INT_MAX};
        S->max_core = 0;
        S->failed = 0;
    }
    pgd_cl::cluster_sync();
    int level = at.level, removed = at.removed;
    unsigned na = at.na ? at.na : (unsigned)n, nf = at.nf, nb = 0;
    long long step = 0;
    const long long max_steps = 2ll * n + max_degree + 8;   // every step removes a vertex or raises the level
    int32_t *ain = a0, *aout = a1, *fin = f0, *fout = f1, *bin = b0, *bout = b1;
    auto next_slot = [&]() -> CoreSlot * {   // this step's slot; the one after it is cleared
        CoreSlot *s = &S->slot[step % 3];
        if (t == 0) S->slot[(step + 1) % 3] = CoreSlot{0, 0, 0, INT_MAX};
        step++;
        return s;
    };
    while ((removed < n || nf > 0) && step < max_steps) {
        if (nf == 0) {   // no frontier left over: a level scan
            CoreSlot *s = next_slot();
            int low = INT_MAX;
            for (unsigned i0 = (unsigned)t0; i0 < na; i0 += kAll) {
                const unsigned i = i0 + lane;
                bool leaves = false, stays = false;
                int32_t v = 0;
                int d = 0;
                if (i < na) {
                    v = __ldcg(ain + i);
                    if (__ldcg(core + v) == -1) {
                        const int c = __ldcg(cur + v);
                        leaves = c <= level;
                        stays = !leaves;
                        if (leaves) {
                            __stcg(core + v, level);
                            d = deg[v];
                        } else {
                            low = min(low, c);
                        }
                    }
                }
                core_append(leaves && d < kCoreLong, v, fin, &s->front, lane);
                core_append(leaves && d >= kCoreLong, v, bin, &s->lng, lane);
                core_append(stays, v, aout, &s->alive, lane);
            }
            low = __reduce_min_sync(0xffffffffu, low);
            if (lane == 0 && low != INT_MAX) atomicMin(&s->min_rest, low);
            pgd_cl::cluster_sync();
            nf = __ldcg(&s->front);
            nb = __ldcg(&s->lng);
            na = __ldcg(&s->alive);
            int32_t *x = ain;
            ain = aout;
            aout = x;
            if (nf + nb == 0) {
                level = max(level + 1, __ldcg(&s->min_rest));   // nobody at this level: on to the smallest count
                continue;
            }
            removed += (int)(nf + nb);
        }
        while (nf + nb > 0 && step < max_steps) {
            CoreSlot *s = next_slot();
            // one off the count of neighbour y; it leaves when that drops to the level
            auto visit = [&](bool act, int32_t y) {
                bool leaves = false;
                int d = 0;
                if (act && __ldcg(core + y) == -1 && atomicSub(cur + y, 1) == level + 1) {
                    __stcg(core + y, level);
                    leaves = true;
                    d = deg[y];
                }
                if (__any_sync(0xffffffffu, leaves)) {
                    core_append(leaves && d < kCoreLong, y, fout, &s->front, lane);
                    core_append(leaves && d >= kCoreLong, y, bout, &s->lng, lane);
                }
            };
            core_rows(adj, nf, w, kAll / 32, [&](unsigned i) { return __ldcg(fin + i); },
                      [&](int32_t v, int64_t &o, int &d) {
                          o = off[v];
                          d = deg[v];
                      },
                      visit);
            // a long row is shared by all warps, by a block's where there is one for
            // each block, or taken by one warp where there are plenty (the chains of
            // loads then run side by side: G(3000, 0.5) 2.6 -> 0.57 ms with eight blocks)
            const int share = nb >= (unsigned)(kAll / 32) ? 32 : nb >= (unsigned)kCoreBlocks ? kCoreThreads : kAll;
            for (unsigned i = (unsigned)(t / share); i < nb; i += (unsigned)(kAll / share)) {
                const int32_t v = __ldcg(bin + i);
                const int64_t o = off[v], e = o + deg[v];
                for (int64_t j = o + t0 % share; j < e; j += share)
                    visit(j + lane < e, j + lane < e ? __ldg(adj + j + lane) : 0);
            }
            pgd_cl::cluster_sync();
            nf = __ldcg(&s->front);
            nb = __ldcg(&s->lng);
            removed += (int)(nf + nb);
            int32_t *x = fin;
            fin = fout;
            fout = x;
            x = bin;
            bin = bout;
            bout = x;
        }
        level++;
    }
    // the value the reference prints leaves the last vertex out
    int top = 0;
    for (int v = t; v < n - 1; v += kAll) top = max(top, __ldcg(core + v));
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0 && top > 0) atomicMax(&S->max_core, top);
    if (t == 0 && removed < n) S->failed = 1;
}

// Small graphs: one block with every count (16 bits), a bit per vertex removed and
// the row offsets in shared memory.  The bound is the chain of removals, one L2
// latency (the row) and some shared-memory operations per link, so the warps of a level never wait for each other: each takes its part
// of the vertices of count <= level, then whatever a removal has pushed onto the
// level's queue, until nothing is queued or in work.  A vertex belongs to the warp
// that sets its bit.  What finds the queue full is left to another turn of the same
// level.
// Up to 2^20 entries and about 32,000 vertices, microseconds of the call against
// the cluster's: R-MAT 12 261 / 695, R-MAT 14 656 / 1197 (1239 for eight blocks),
// R-MAT 15 1148 / 1496, G(1000, 0.5) 176 / 313, a 20,000-vertex BA graph 349 / 350,
// a path of 20,000 7.9 / 33 ms.  Without the offsets in shared memory (R-MAT 16 with
// 5 edges per vertex 1357 / 1270, a geometric graph of 60,000 987 / 498) and for
// more entries (G(1500, 0.9) 421 / 168) the cluster is the faster one.
constexpr int kCoreSmallBytes = 196 * 1024;
constexpr int64_t kCoreSmallEntries = 1ll << 20;
constexpr int kCoreQueue = 4096;
constexpr int kCoreQueueRoom = kCoreQueue - kCoreThreads;   // every warp may add 32 after it has seen room
constexpr int kCoreSpins = 1 << 26;                         // turns without work after which a warp gives up

static size_t core_small_bytes(int64_t n) {
    return (size_t)((n + 63) / 64) * 64 * 2 + (size_t)((n + 63) / 64) * 8 + ((size_t)n + 1) * 4;
}

__global__ void __launch_bounds__(kCoreThreads, 1)
k_core_block(const int64_t *off, const int32_t *adj, const int32_t *deg, int n, int32_t *core, CoreShared *S) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    constexpr int kWarps = kCoreThreads / 32;
    __shared__ int32_t s_queue[kCoreQueue];          // vertex + 1, 0 until written
    __shared__ int32_t s_mine[kWarps][64];           // a warp's vertices of one group
    __shared__ unsigned int s_head, s_tail, s_done;  // entries taken, reserved, worked off
    __shared__ unsigned int s_scanned;               // warps through with their part
    __shared__ int s_removed, s_low, s_again, s_fail, s_max;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int groups = (n + 63) / 64;       // 64 vertices: 32 words of counts, 2 of bits
    uint32_t *cur = s_dyn, *gone = s_dyn + 32 * groups, *s_off = gone + 2 * groups;
    for (int i = threadIdx.x; i <= n; i += kCoreThreads) s_off[i] = (uint32_t)off[i];
    auto row = [&](int32_t v, int64_t &o, int &d) {
        o = s_off[v];
        d = (int)(s_off[v + 1] - s_off[v]);
    };
    for (int i = threadIdx.x; i < 32 * groups; i += kCoreThreads) {
        const uint32_t lo = 2 * i < n ? (uint32_t)deg[2 * i] : 0, hi = 2 * i + 1 < n ? (uint32_t)deg[2 * i + 1] : 0;
        cur[i] = lo | hi << 16;
    }
    for (int i = threadIdx.x; i < 2 * groups; i += kCoreThreads)
        gone[i] = 32 * i + 32 <= n ? 0u : (32 * i >= n ? 0xffffffffu : 0xffffffffu << (n - 32 * i));
    for (int i = threadIdx.x; i < kCoreQueue; i += kCoreThreads) s_queue[i] = 0;
    if (threadIdx.x == 0) {
        s_head = s_tail = s_done = s_scanned = 0;
        s_removed = s_again = s_fail = s_max = 0;
        s_low = INT_MAX;
    }
    __syncthreads();
    volatile unsigned int *head = &s_head, *tail = &s_tail, *done = &s_done, *scanned = &s_scanned;
    volatile int *fail = &s_fail;
    volatile int32_t *queue = s_queue;
    int level = 0, before = 0;
    while (true) {
        int taken = 0;                      // vertices this warp has removed in this turn
        auto visit = [&](bool act, int32_t y) {
            bool in = false;
            if (act && !((gone[y >> 5] >> (y & 31)) & 1u)) {
                const int sh = (y & 1) << 4;
                // at most deg(y) take one off: the half never borrows
                in = (int)((atomicSub(cur + (y >> 1), 1u << sh) >> sh) & 0xffffu) == level + 1;
            }
            if (!__any_sync(0xffffffffu, in)) return;
            const bool room = __shfl_sync(0xffffffffu, (int)(*tail <= (unsigned)kCoreQueueRoom), 0);
            if (!room) {
                if (lane == 0) s_again = 1;
                return;
            }
            // a part of this level still ahead may have taken it already
            if (in) in = !((atomicOr(gone + (y >> 5), 1u << (y & 31)) >> (y & 31)) & 1u);
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (!m) return;
            unsigned at = 0;
            if (lane == 0) at = atomicAdd(&s_tail, (unsigned)__popc(m));
            at = __shfl_sync(0xffffffffu, at, 0) + (unsigned)__popc(m & ((1u << lane) - 1));
            if (in) {
                queue[at] = y + 1;
                core[y] = level;
            }
            taken += __popc(m);
        };
        auto one_row = [&](int32_t v) {     // the same v in all lanes
            int64_t o;
            int d;
            row(v, o, d);
            for (int j = 0; j < d; j += 128) {
                int32_t y[4];
#pragma unroll
                for (int k = 0; k < 4; k++) y[k] = j + 32 * k + lane < d ? __ldg(adj + o + j + 32 * k + lane) : 0;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (j + 32 * k < d) visit(j + 32 * k + lane < d, y[k]);
            }
        };
        // this warp's part: every vertex left of count <= level
        int low = INT_MAX;
        for (int g = wid; g < groups; g += kWarps) {
            const uint32_t out = gone[2 * g + (lane >> 4)];
            if (__all_sync(0xffffffffu, out == 0xffffffffu)) continue;
            const uint32_t c2 = cur[32 * g + lane];
            const int b = 2 * (lane & 15), ca = (int)(c2 & 0xffffu), cb = (int)(c2 >> 16);
            const bool ha = !((out >> b) & 1u), hb = !((out >> b) & 2u);
            bool ia = ha && ca <= level, ib = hb && cb <= level;
            if (ha && !ia) low = min(low, ca);
            if (hb && !ib) low = min(low, cb);
            if (!__any_sync(0xffffffffu, ia || ib)) continue;
            if (ia || ib) {
                const uint32_t had = atomicOr(gone + 2 * g + (lane >> 4), (ia ? 1u << b : 0u) | (ib ? 2u << b : 0u));
                ia = ia && !((had >> b) & 1u);
                ib = ib && !((had >> b) & 2u);
            }
            const unsigned ma = __ballot_sync(0xffffffffu, ia), mb = __ballot_sync(0xffffffffu, ib);
            const unsigned below = (1u << lane) - 1;
            const int32_t v = 64 * g + 2 * lane;
            if (ia) {
                s_mine[wid][__popc(ma & below)] = v;
                core[v] = level;
            }
            if (ib) {
                s_mine[wid][__popc(ma) + __popc(mb & below)] = v + 1;
                core[v + 1] = level;
            }
            __syncwarp();
            const unsigned nf = (unsigned)(__popc(ma) + __popc(mb));
            taken += (int)nf;
            if (nf == 1) one_row(s_mine[wid][0]);
            else core_rows(adj, nf, 0, 1, [&](unsigned i) { return s_mine[wid][i]; }, row, visit);
            __syncwarp();
        }
        low = __reduce_min_sync(0xffffffffu, low);
        if (lane == 0) {
            if (low != INT_MAX) atomicMin(&s_low, low);
            __threadfence_block();
            atomicAdd(&s_scanned, 1u);
        }
        // then what is queued
        int spins = 0;
        while (true) {
            unsigned h = 0;
            int take = 0;                   // -1: nothing queued or in work
            if (lane == 0) {
                const bool all = *scanned == (unsigned)kWarps;
                const unsigned over = *done;   // before the tail: equal means that nothing was left
                h = *head;
                const unsigned t = *tail;
                if (h < t) {
                    const int want = (int)min(32u, max(1u, (t - h) / kWarps));
                    if (atomicCAS(&s_head, h, h + (unsigned)want) == h) take = want;
                } else if (all && over == t) {
                    take = -1;
                } else {
                    if (++spins > kCoreSpins) s_fail = 1;
                    if (*fail) take = -1;
                    __nanosleep(20);
                }
            }
            take = __shfl_sync(0xffffffffu, take, 0);
            h = __shfl_sync(0xffffffffu, h, 0);
            if (take < 0) break;
            if (take == 0) continue;
            int32_t v = 0;
            if (lane < take)
                for (int i = 0; i < kCoreSpins && (v = queue[h + lane]) == 0; i++) __nanosleep(20);   // being written
            if (__any_sync(0xffffffffu, lane < take && v == 0)) {
                if (lane == 0) s_fail = 1;
                break;
            }
            if (lane < take) queue[h + lane] = 0;
            if (take == 1) one_row(__shfl_sync(0xffffffffu, v, 0) - 1);
            else core_rows(adj, (unsigned)take, 0, 1, [&](unsigned) { return v - 1; }, row, visit);   // entry i: lane i
            __syncwarp();
            if (lane == 0) {
                __threadfence_block();
                atomicAdd(&s_done, (unsigned)take);
            }
        }
        if (lane == 0 && taken) atomicAdd(&s_removed, taken);
        __syncthreads();
        const int removed = s_removed, lowest = s_low;
        const bool again = s_again != 0, failed = s_fail != 0;
        __syncthreads();
        if (threadIdx.x == 0) {
            s_head = s_tail = s_done = s_scanned = 0;
            s_low = INT_MAX;
            s_again = 0;
        }
        __syncthreads();
        if (removed >= n || failed) break;
        if (!again) level = removed == before ? max(level + 1, lowest) : level + 1;
        before = removed;
    }
    int top = 0;
    for (int v = threadIdx.x; v < n - 1; v += kCoreThreads) top = max(top, core[v]);
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0 && top > 0) atomicMax(&s_max, top);
    __syncthreads();
    if (threadIdx.x == 0) {
        S->max_core = s_max;
        S->failed = s_fail;
    }
}

}  // namespace

cudaError_t pgd_build_limits() {
    constexpr cudaFuncAttribute kDyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
    constexpr int kSort = 2 * (int)kSmallPairs * 8;
    cudaError_t e = cudaFuncSetAttribute(k_core_block, kDyn, kCoreSmallBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_core_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_small_build, kDyn, kSort);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_small_edges, kDyn, kSort);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_small_order, kDyn, kSort);
    return e;
}

// Waits for a peeling by one block or the cluster, whose work array it frees.
// *launched false: the device has no room for the cluster, nothing was done.
static pgd_status cores_result(pgd_graph *g, void *work, const CoreShared *S, bool *launched) {
    pgd_ctx *ctx = g->ctx;
    cudaError_t e = cudaGetLastError();
    *launched = e != cudaErrorLaunchOutOfResources && e != cudaErrorInvalidClusterSize;
    if (e == cudaSuccess) e = pgd_fetch(ctx, 0, S, sizeof(CoreShared));
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    pgd_tmp_free(ctx, work);
    if (!*launched) return PGD_OK;
    if (e != cudaSuccess) return pgd_cuda_fail(ctx, e, "k-core peeling");
    const CoreShared h = pgd_pinned<CoreShared>(ctx, 0);
    if (h.failed) return pgd_fail(ctx, PGD_EINVAL, "k-core peeling did not converge");
    g->max_core = h.max_core;
    g->has_cores = true;
    return PGD_OK;
}

// A light graph, by one block or the cluster.
static pgd_status cores_light(pgd_graph *g, bool *launched) {
    pgd_ctx *ctx = g->ctx;
    const int64_t n = g->n;
    int32_t *work = nullptr;
    pgd_status st;
    const size_t lists = (7 * (size_t)n * sizeof(int32_t) + 15) & ~(size_t)15;
    if ((st = pgd_tmp_alloc(ctx, (void **)&work, lists + sizeof(CoreShared)))) return st;
    CoreShared *S = (CoreShared *)((uint8_t *)work + lists);
    if (g->max_degree < 65536 && 2 * g->m <= kCoreSmallEntries && core_small_bytes(n) <= (size_t)kCoreSmallBytes)
        PGD_LAUNCH(ctx, k_core_block, 1, kCoreThreads, core_small_bytes(n), g->off, g->adj, g->deg, (int)n, g->core, S);
    else
        PGD_LAUNCH(ctx, k_core_cluster, kCoreBlocks, kCoreThreads, 0, g->off, g->adj, g->deg, (int)n, work, g->core,
               work + n, work + 2 * n, work + 3 * n, work + 4 * n, work + 5 * n, work + 6 * n, S, g->max_degree,
               CoreStart{0, 0, 0, 0});
    return cores_result(g, work, S, launched);
}

// Other graphs: on the whole device, until their steps are narrow.
// Device-driven peeling: the state machine below replaces a host loop with
// one round trip per level and per peel round.  Each step is a work kernel
// (a level scan or a peel round, chosen from the state) and a one-thread
// control kernel that applies the transition; a block of kCoreSteps steps is
// captured once as a CUDA graph and replayed until the control kernel
// reports that every vertex has a core number or the steps are narrow.  A level scan reads only the
// vertices still alive at the previous scan (a compacted list, rewritten by
// each scan), so the scans shrink as the peeling goes inward.
namespace {

struct CoreState {
    int level, mode, sel, done, failed, min_rest;
    unsigned int cnt[2];          // frontier sizes of buffers 0 and 1
    long long removed, steps, max_steps;
    long long scanned;            // vertices that the scans have read
    int asel;                     // alive list read by the next scan
    unsigned int acnt[2];         // alive list sizes
};

constexpr int kCoreSteps = 64;
enum { kCoreScan = 0, kCorePeel = 1 };

__global__ void k_core_work(const int64_t *off, const int32_t *adj, int32_t *cur, int32_t *core, int64_t n,
                            int32_t *f0, int32_t *f1, int32_t *a0, int32_t *a1, CoreState *st) {
    if (st->done) return;
    const int mode = st->mode, level = st->level, sel = st->sel;
    int32_t *fin = sel ? f1 : f0, *fout = sel ? f0 : f1;
    if (mode == kCoreScan) {
        // every alive vertex with cur <= level leaves now; the others are
        // kept in the next alive list, and the smallest cur among them lets
        // the control kernel skip empty levels
        const int asel = st->asel;
        const int32_t *ain = asel ? a1 : a0;
        int32_t *aout = asel ? a0 : a1;
        const unsigned int na = st->acnt[asel];
        int local_min = INT_MAX;
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < na; i += (int64_t)gridDim.x * blockDim.x) {
            const int32_t v = ain[i];
            if (core[v] != -1) continue;
            const int c = cur[v];
            if (c <= level) {
                core[v] = level;
                fin[atomicAdd(&st->cnt[sel], 1u)] = v;
            } else {
                local_min = min(local_min, c);
                aout[atomicAdd(&st->acnt[asel ^ 1], 1u)] = v;
            }
        }
        for (int o = 16; o > 0; o >>= 1) local_min = min(local_min, __shfl_xor_sync(0xffffffffu, local_min, o));
        if ((threadIdx.x & 31) == 0 && local_min != INT_MAX) atomicMin(&st->min_rest, local_min);
    } else {
        // remove the frontier: each alive neighbour loses one; the one whose
        // count drops to `level` joins the next frontier (one warp per vertex)
        const int lane = threadIdx.x & 31;
        const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
        const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
        const unsigned int fsize = st->cnt[sel];
        for (int64_t f = w; f < fsize; f += nw) {
            const int32_t v = fin[f];
            for (int64_t j = off[v] + lane; j < off[v + 1]; j += 32) {
                const int32_t x = adj[j];
                if (core[x] != -1) continue;
                const int old = atomicSub(&cur[x], 1);
                if (old == level + 1) {
                    core[x] = level;
                    fout[atomicAdd(&st->cnt[sel ^ 1], 1u)] = x;
                }
            }
        }
    }
}

__global__ void k_core_ctrl(CoreState *st, int64_t n) {
    if (st->done) return;
    const int sel = st->sel;
    if (st->mode == kCoreScan) {
        // the scan's survivors are the next alive list
        st->scanned += st->acnt[st->asel];
        st->asel ^= 1;
        st->acnt[st->asel ^ 1] = 0;
        const unsigned int f = st->cnt[sel];
        if (f == 0) {
            // nobody at this level: jump to the smallest remaining count
            st->level = max(st->level + 1, st->min_rest);
            st->min_rest = INT_MAX;
        } else {
            st->removed += f;
            st->mode = kCorePeel;
            st->cnt[sel ^ 1] = 0;
        }
    } else {
        const unsigned int nf = st->cnt[sel ^ 1];
        st->removed += nf;
        if (nf == 0) {
            st->level += 1;
            st->mode = kCoreScan;
            st->cnt[sel] = 0;
            st->min_rest = INT_MAX;
        } else {
            st->sel = sel ^ 1;
            st->cnt[sel] = 0;   // the buffer written next
        }
    }
    st->steps += 1;
    if (st->removed >= n) st->done = 1;
    else if (st->steps >= st->max_steps) {
        st->done = 1;
        st->failed = 1;
    }
}

}  // namespace

pgd_status pgd_dev_cores(pgd_graph *g) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    pgd_status st;
    int64_t n = g->n;
    if (!g->core) {
        if ((st = pgd_graph_alloc(g, (void **)&g->core, (n + 1) * sizeof(int32_t)))) return st;
    }
    if (n == 0) { g->has_cores = true; g->max_core = 0; return PGD_OK; }
    if (pgd_core_light(n, 2 * g->m)) {
        bool launched = false;
        const pgd_status st = cores_light(g, &launched);
        if (launched || st) return st;
    }
    int32_t *cur = nullptr, *fa = nullptr, *fb = nullptr, *aa = nullptr, *ab = nullptr;
    CoreState *d_st = nullptr;
    if ((st = pgd_tmp_alloc(ctx, (void **)&cur, n * sizeof(int32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&fa, n * sizeof(int32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&fb, n * sizeof(int32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&aa, n * sizeof(int32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&ab, n * sizeof(int32_t)))) return st;
    if ((st = pgd_tmp_alloc(ctx, (void **)&d_st, sizeof(CoreState)))) return st;
    auto release = [&]() {
        pgd_tmp_free(ctx, cur);
        pgd_tmp_free(ctx, fa);
        pgd_tmp_free(ctx, fb);
        pgd_tmp_free(ctx, aa);
        pgd_tmp_free(ctx, ab);
        pgd_tmp_free(ctx, d_st);
    };
    PGD_LAUNCH(ctx, k_core_init, grid_for(n), kThreads, 0, g->deg, n, cur, g->core, aa);
    // every step removes a vertex or raises the level (at most max_degree + 1
    // levels), so 2 (n + max_degree) + 4 steps always suffice
    CoreState h{};
    h.min_rest = INT_MAX;
    h.max_steps = 2 * (n + (long long)g->max_degree) + 4;
    h.asel = 0;
    h.acnt[0] = (unsigned int)n;   // every vertex alive at the first scan
    h.acnt[1] = 0;
    PGD_CUDA(ctx, cudaMemcpyAsync(d_st, &h, sizeof(h), cudaMemcpyHostToDevice, s));
    const int work_grid = grid_for(32 * (int64_t)ctx->num_sms * 64);
    // capture kCoreSteps steps once, replay until done
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        for (int i = 0; i < kCoreSteps; i++) {
            k_core_work<<<work_grid, kThreads, 0, s>>>(g->off, g->adj, cur, g->core, n, fa, fb, aa, ab, d_st);
            k_core_ctrl<<<1, 1, 0, s>>>(d_st, n);
        }
        e = cudaStreamEndCapture(s, &graph);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    if (e != cudaSuccess) {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        release();
        return pgd_cuda_fail(ctx, e, "k-core step graph");
    }
    bool narrow = false, room = true;   // room: the device takes the cluster
    while (!h.done && !narrow) {
        const CoreState was = h;
        e = cudaGraphLaunch(exec, s);
        if (e == cudaSuccess) e = pgd_fetch(ctx, 0, d_st, sizeof(h));
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) break;
        h = pgd_pinned<CoreState>(ctx, 0);
        ctx->launches += 2 * kCoreSteps;
        narrow = room && !h.done &&
                 pgd_core_narrow(n, 2 * g->m, kCoreSteps, h.scanned - was.scanned, h.removed - was.removed);
        if (!narrow) continue;
        // the steps are narrow: the rest in the cluster, from the state between two steps
        int32_t *work = nullptr;
        const size_t lists = (2 * (size_t)n * sizeof(int32_t) + 15) & ~(size_t)15;
        if (pgd_tmp_alloc(ctx, (void **)&work, lists + sizeof(CoreShared))) {
            room = narrow = false;
            continue;
        }
        CoreShared *S = (CoreShared *)((uint8_t *)work + lists);
        const bool peel = h.mode == kCorePeel;
        PGD_LAUNCH(ctx, k_core_cluster, kCoreBlocks, kCoreThreads, 0, g->off, g->adj, g->deg, (int)n, cur, g->core,
                   h.sel ? fb : fa, h.sel ? fa : fb, work, work + n, h.asel ? ab : aa, h.asel ? aa : ab, S,
                   g->max_degree, CoreStart{h.level, (int)h.removed, h.acnt[h.asel], peel ? h.cnt[h.sel] : 0u});
        st = cores_result(g, work, S, &room);
        narrow = room;
    }
    cudaGraphExecDestroy(exec);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
        release();
        return pgd_cuda_fail(ctx, e, "k-core peeling");
    }
    if (narrow) {
        release();
        return st;
    }
    int *d_mc = (int *)d_st;
    if (h.failed) {
        release();
        return pgd_fail(ctx, PGD_EINVAL, "k-core peeling did not converge");
    }
    PGD_CUDA(ctx, cudaMemsetAsync(d_mc, 0, sizeof(int), s));
    if (n > 1) PGD_LAUNCH(ctx, k_max_core, grid_for(n - 1), kThreads, 0, g->core, n - 1, d_mc);
    int mc = 0;
    PGD_CUDA(ctx, cudaMemcpyAsync(&mc, d_mc, sizeof(int), cudaMemcpyDeviceToHost, s));
    PGD_CUDA(ctx, cudaStreamSynchronize(s));
    release();
    PGD_CUDA(ctx, cudaGetLastError());
    g->max_core = mc;
    g->has_cores = true;
    return PGD_OK;
}

pgd_status pgd_dev_assortativity(pgd_graph *g, double *r) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    pgd_status st;
    int64_t m = g->m;
    int blocks = grid_for(m, kThreads, 4 * ctx->num_sms);
    double *partial = nullptr;
    if ((st = pgd_tmp_alloc(ctx, (void **)&partial, 3 * blocks * sizeof(double)))) return st;
    PGD_LAUNCH(ctx, k_assort_partial, blocks, kThreads, 0, g->ev, g->eu, g->deg, m, partial);
    double *h = (double *)malloc(3 * blocks * sizeof(double));
    PGD_CUDA(ctx, cudaMemcpyAsync(h, partial, 3 * blocks * sizeof(double), cudaMemcpyDeviceToHost, s));
    PGD_CUDA(ctx, cudaStreamSynchronize(s));
    pgd_tmp_free(ctx, partial);
    double mu = 0, jd = 0, psi = 0;
    for (int b = 0; b < blocks; b++) { mu += h[3 * b]; jd += h[3 * b + 1]; psi += h[3 * b + 2]; }
    free(h);
    double dm = (double)m;
    double tau = (jd / dm) * (jd / dm);
    double rr = ((mu / dm) - tau) / ((psi / dm) - tau);
    // The reference's isnan() guard is compiled out by -ffast-math
    // (graphlet_core.cpp:1054), so a NaN stays NaN; the range check cannot
    // fire on NaN either.
    if (rr < -1 || rr > 1.0) rr = 1;
    if (m == 0) rr = 0.0;
    *r = rr;
    return PGD_OK;
}

// Orders every edge (d_ids == null, count == m) or the sample d_ids[0..count)
// (device array of edge ids in [0, m)); E_ordered gets count entries.
static pgd_status sort_edges_impl(pgd_graph *g, int kind, int s2l, const int32_t *d_ids, int64_t count) {
    pgd_ctx *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    pgd_status st;
    int64_t m = g->m;
    if (!g->order) {
        if ((st = pgd_graph_alloc(g, (void **)&g->order, (m + 1) * sizeof(int32_t)))) return st;
    }
    g->sorted = false;
    g->has_micro = false;
    g->norder = count;
    if (count == 0) { g->sorted = true; return PGD_OK; }
    uint64_t *vsum = nullptr;
    if (kind == PGD_ORD_DEG_VOL) {
        vsum = g->vol2;
        if (!g->has_vol2) {
            PGD_LAUNCH(ctx, k_neigh_sum, grid_for(g->n * 32), kThreads, 0, g->off, g->adj, g->deg, nullptr, g->n, 0, vsum);
            g->has_vol2 = true;
        }
    } else if (kind == PGD_ORD_KCORE_VOL || kind == PGD_ORD_KCORE_DEG_VOL) {
        if ((st = pgd_tmp_alloc(ctx, (void **)&vsum, g->n * sizeof(uint64_t)))) return st;
        PGD_LAUNCH(ctx, k_neigh_sum, grid_for(g->n * 32), kThreads, 0, g->off, g->adj, g->deg, g->core, g->n,
                                                              kind == PGD_ORD_KCORE_VOL ? 1 : 2, vsum);
    }
    // bits of the keys: all 32 where they may be negative (volumes and products
    // wrap as the reference's ints do)
    const uint64_t d2 = 2 * (uint64_t)g->max_degree, c2 = 2 * (uint64_t)g->max_core;
    uint64_t top = UINT64_MAX;   // largest key, where it is known
    switch (kind) {
    case PGD_ORD_DEG: top = d2; break;
    case PGD_ORD_KCORE: top = c2; break;
    case PGD_ORD_KCORE_DEG: top = d2 * c2; break;
    case PGD_ORD_DEG_U: top = d2 / 2; break;
    case PGD_ORD_DEG_VOL:
    case PGD_ORD_KCORE_VOL:
    case PGD_ORD_KCORE_DEG_VOL: break;
    default: top = (uint64_t)count; break;
    }
    const bool small = top < 0x80000000ull;
    const int kb = small ? std::max(1, pgd_bit_length(top)) : 32;
    const uint32_t flip = small ? 0u : 0x80000000u;
    size_t tb = 0;
    void *tmp = nullptr;
    if (!d_ids && count <= kSmallPairs) {
        const int P = pgd_small_words(count);
        PGD_LAUNCH(ctx, k_small_order, 1, kSmallThreads, P * sizeof(uint64_t), g->ev, g->eu, g->deg, g->core, vsum,
                   (int)count, kind, s2l, P, g->order);
    } else if (!d_ids) {
        uint32_t *keys = nullptr, *keys2 = nullptr;
        int32_t *ids = nullptr;
        if (s2l) cub::DeviceRadixSort::SortPairs(nullptr, tb, keys, keys2, ids, g->order, count, 0, kb, s);
        else cub::DeviceRadixSort::SortPairsDescending(nullptr, tb, keys, keys2, ids, g->order, count, 0, kb, s);
        const size_t cb = count * sizeof(uint32_t);
        pgd_pieces P;
        P.add(cb); P.add(cb); P.add(cb); P.add(tb);
        void *work = nullptr;
        if ((st = pgd_tmp_alloc(ctx, &work, P.bytes))) return st;
        P.base = (uint8_t *)work;
        keys = P.take<uint32_t>(cb);
        keys2 = P.take<uint32_t>(cb);
        ids = P.take<int32_t>(cb);
        tmp = P.take<void>(tb);
        PGD_LAUNCH(ctx, k_edge_keys, grid_for(count), kThreads, 0, g->ev, g->eu, g->deg, g->core, vsum, count, kind,
                   flip, keys, ids);
        if (s2l) cub::DeviceRadixSort::SortPairs(tmp, tb, keys, keys2, ids, g->order, count, 0, kb, s);
        else cub::DeviceRadixSort::SortPairsDescending(tmp, tb, keys, keys2, ids, g->order, count, 0, kb, s);
        pgd_tmp_free(ctx, work);
    } else {
        uint64_t *keys = nullptr, *keys2 = nullptr;
        if ((st = pgd_tmp_alloc(ctx, (void **)&keys, count * sizeof(uint64_t)))) return st;
        if ((st = pgd_tmp_alloc(ctx, (void **)&keys2, count * sizeof(uint64_t)))) return st;
        const int idb = std::max(1, pgd_bit_length((uint64_t)m));
        PGD_LAUNCH(ctx, k_sample_keys, grid_for(count), kThreads, 0, g->ev, g->eu, g->deg, g->core, vsum, d_ids, count,
                   kind, s2l, flip, idb, keys);
        if (s2l) cub::DeviceRadixSort::SortKeys(nullptr, tb, keys, keys2, count, 0, kb + idb, s);
        else cub::DeviceRadixSort::SortKeysDescending(nullptr, tb, keys, keys2, count, 0, kb + idb, s);
        if ((st = pgd_tmp_alloc(ctx, &tmp, tb))) return st;
        if (s2l) cub::DeviceRadixSort::SortKeys(tmp, tb, keys, keys2, count, 0, kb + idb, s);
        else cub::DeviceRadixSort::SortKeysDescending(tmp, tb, keys, keys2, count, 0, kb + idb, s);
        pgd_tmp_free(ctx, tmp);
        PGD_LAUNCH(ctx, k_keys_to_ids, grid_for(count), kThreads, 0, keys2, count, s2l, idb, g->order);
        pgd_tmp_free(ctx, keys);
        pgd_tmp_free(ctx, keys2);
    }
    if (vsum && vsum != g->vol2) pgd_tmp_free(ctx, vsum);
    PGD_CUDA(ctx, cudaGetLastError());
    g->sorted = true;
    return PGD_OK;
}

pgd_status pgd_dev_sort_edges(pgd_graph *g, int kind, int s2l) { return sort_edges_impl(g, kind, s2l, nullptr, g->m); }

pgd_status pgd_dev_sort_edges_sample(pgd_graph *g, int kind, int s2l, const int64_t *h_ids, int64_t k) {
    pgd_ctx *ctx = g->ctx;
    pgd_status st;
    if (k < 0 || k > g->m) return pgd_fail(ctx, PGD_EINVAL, "sample size must be between 0 and m");
    for (int64_t i = 0; i < k; i++)
        if (h_ids[i] < 0 || h_ids[i] >= g->m) return pgd_fail(ctx, PGD_EINVAL, "sampled edge id out of range");
    std::vector<int32_t> ids32((size_t)k + 1);
    for (int64_t i = 0; i < k; i++) ids32[(size_t)i] = (int32_t)h_ids[i];
    int32_t *d_ids = nullptr;
    if ((st = pgd_tmp_alloc(ctx, (void **)&d_ids, (k + 1) * sizeof(int32_t)))) return st;
    cudaError_t e = cudaMemcpyAsync(d_ids, ids32.data(), k * sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);   // ids32 is a host temporary
    if (e != cudaSuccess) {
        pgd_tmp_free(ctx, d_ids);
        return pgd_cuda_fail(ctx, e, "copy of the sampled edge ids");
    }
    st = sort_edges_impl(g, kind, s2l, d_ids, k);
    pgd_tmp_free(ctx, d_ids);
    return st;
}

// ---------------------------------------------------------------------------
// Row ids of the per-edge output (the writer's id+1 convention,
// graphlet_core.cpp:1694-1701): row e is edge order[e].

__global__ void k_micro_ids(const int32_t *ev, const int32_t *eu, const int32_t *order, int64_t m, int64_t *src1,
                            int64_t *dst1) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t id = order[e];
        if (src1) src1[e] = (int64_t)ev[id] + 1;
        if (dst1) dst1[e] = (int64_t)eu[id] + 1;
    }
}

// The per-edge rows and their ids written straight into host memory that the
// device can address (page-locked and mapped): one pass of every SM over the
// host link, 16-byte stores.  Any of the three outputs may be null.
__global__ void k_micro_out(const uint4 *micro, const int32_t *ev, const int32_t *eu, const int32_t *order,
                            int64_t m, uint4 *cols, int64_t *src1, int64_t *dst1) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (cols)   // a row is 8 x 8 bytes = 4 x 16 bytes
        for (int64_t i = t0; i < m * (PGD_NMICRO / 2); i += stride) cols[i] = micro[i];
    if (src1 || dst1)
        for (int64_t e = t0; e < m; e += stride) {
            const int32_t id = order[e];
            if (src1) src1[e] = (int64_t)ev[id] + 1;
            if (dst1) dst1[e] = (int64_t)eu[id] + 1;
        }
}

pgd_status pgd_dev_micro_out(pgd_graph *g, uint64_t *cols, int64_t *src1, int64_t *dst1) {
    pgd_ctx *ctx = g->ctx;
    if (g->norder > 0)
        PGD_LAUNCH(ctx, k_micro_out, ctx->num_sms * 8, kThreads, 0, (const uint4 *)g->micro, g->ev, g->eu, g->order,
                   g->norder, (uint4 *)cols, src1, dst1);
    PGD_CUDA(ctx, cudaGetLastError());
    return PGD_OK;
}

pgd_status pgd_dev_micro_ids(pgd_graph *g, int64_t *d_src1, int64_t *d_dst1) {
    pgd_ctx *ctx = g->ctx;
    if (g->norder > 0)
        PGD_LAUNCH(ctx, k_micro_ids, grid_for(g->norder), kThreads, 0, g->ev, g->eu, g->order, g->norder, d_src1, d_dst1);
    PGD_CUDA(ctx, cudaGetLastError());
    return PGD_OK;
}
