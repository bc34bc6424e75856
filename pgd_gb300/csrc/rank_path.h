// rank_path.h -- decomposition of graphs in degree-rank order (rank_path.cu):
// what decompose.cu needs to build the rank-ordered graph and to run it.
#pragma once

#include "pgd_internal.h"

// The rank-ordered copy of a graph and its work lists, all in device memory.
// Ranks are positions in (degree descending, id descending); vertices whose
// degree is masked to 0 (members of a batch that another path decomposes)
// come last and have no rows.
struct pgd_rank_graph {
    int64_t n = 0;        // vertices
    int64_t nnz = 0;      // entries of radj
    uint32_t *roff = nullptr;    // n + 1: row offsets by rank
    int32_t *rup = nullptr;      // n: entries of the row that are ranked above it (its first ones)
    int32_t *radj = nullptr;     // nnz: ranks, ascending in each row
    uint32_t *wcode = nullptr;   // nnz: bit address of the entry's counter
    uint32_t *tw = nullptr;      // nnz: slot of the reversed edge (slots take all 32 bits: up to 2^31 - 1 edges)
    uint32_t *eslot = nullptr;   // per edge id: slot of the edge in the row of its lower-ranked end (all ones: none)
    uint32_t *bend = nullptr;    // n: first entry of the row whose vertex has degree 1
    uint32_t *bpos = nullptr;    // (nranges - 1) x n2: first entry of the row at or beyond an inner range
                                 // boundary (null: searched when needed)
    int32_t *lists = nullptr;    // work lists by class, n entries each
    unsigned long long *hbase = nullptr;   // n2: place of the vertex's triangles among all pairs of all N+
    int64_t pairs = 0;           // those pairs
    int2 *items = nullptr;       // {u, first range | one past the last range << 16}
    void *meta = nullptr;        // device-side sizes (RankMeta)
    int32_t n2 = 0;              // vertices of degree >= 2
    int32_t nranges = 0;
    int32_t max_up = 0;          // largest rup
    uint32_t nitems = 0;
    int64_t words = 0;           // 32-bit words of all counters
    uint32_t nlist[8] = {0};
    void *held[12] = {nullptr};  // the allocations above
    size_t held_bytes[12] = {0};
    int nheld = 0;
};

// What the closing pass writes to: the per-edge rows, and the sums of the
// graph (or of each graph of a batch).
struct pgd_rank_out {
    const int32_t *ev, *eu, *deg, *order;
    int64_t npos;
    long long n, m;
    uint64_t *micro;              // npos x 8, or null
    unsigned long long *sums;     // PGD_NSUMS, or PGD_NSUMS per graph of a batch
    const int32_t *egraph;        // batch: graph of each position, else null
    const long long *gnm;         // batch: n and m of each graph
    const uint8_t *gdense;        // batch: graphs that another path decomposes, or null
};

// Builds R, owned by g, from g's CSR and edge arrays.  vmask, with vgraph,
// marks the members of a batch that are left out; nnz is the number of entries
// that remain.
pgd_status pgd_rank_build(pgd_graph *g, int64_t nnz, const int32_t *vgraph, const uint8_t *vmask, pgd_rank_graph *R);
void pgd_rank_free(pgd_graph *g, pgd_rank_graph *R);
// Counts every edge and closes the positions of out.  Records tri0/tri1 around
// the triangle and 4-clique passes and cyc0/cyc1 around the 4-cycle pass.
pgd_status pgd_rank_decompose(pgd_ctx *ctx, const pgd_rank_graph &R, const pgd_rank_out &out);
