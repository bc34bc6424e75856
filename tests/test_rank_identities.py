"""CPU check of the counts rank_path.cu forms: t and k4 credited from each
vertex's up-neighbourhood, 4-cycles from the wedges below their highest-ranked
vertex, and c4 = C4 - D + 2 t + 2 k4, against the oracle's per-edge rows."""
import itertools

import numpy as np
import pytest

import oracle_lib as ol
import pgd_gb300 as pgd


def rank_counts(src, dst):
    """Per edge {(lo, hi): (t, k4, c4)} by the passes of rank_path.cu."""
    edges = {(min(a, b), max(a, b)) for a, b in zip(src.tolist(), dst.tolist()) if a != b}
    n = 1 + max(max(e) for e in edges)
    deg = np.zeros(n, int)
    for a, b in edges:
        deg[a] += 1
        deg[b] += 1
    order = sorted(range(n), key=lambda v: (-deg[v], -v))
    rank = {v: i for i, v in enumerate(order)}
    nb = [[] for _ in range(n)]
    key = {}
    for a, b in edges:
        x, y = rank[a], rank[b]
        nb[x].append(y)
        nb[y].append(x)
        key[(min(x, y), max(x, y))] = (a, b)
    nb = [sorted(r) for r in nb]
    at = lambda x, y: (min(x, y), max(x, y))  # noqa: E731
    t, k4, D, cyc = ({e: 0 for e in key} for _ in range(4))
    tri = []
    for a in range(n):
        up = [x for x in nb[a] if x < a]
        ups = set(up)
        for x in up:
            for y in nb[x]:
                if y < x and y in ups:
                    tri.append((a, x, y))
                    for e in (at(a, x), at(a, y), at(x, y)):
                        t[e] += 1
    adj = [set(r) for r in nb]
    for a, x, y in tri:
        e = [at(a, x), at(a, y), at(x, y)]
        for i in range(3):
            D[e[i]] += t[e[(i + 1) % 3]] + t[e[(i + 2) % 3]]
        ups = {z for z in nb[a] if z < a}
        c = len(ups & adj[x] & adj[y])   # 4-cliques {a, x, y, z}, a the lowest
        k4[e[2]] += c
    # edges (a, x): each 4-clique {a, x, y, z} is met from its three upper edges
    for a in range(n):
        up = [z for z in nb[a] if z < a]
        for x in up:
            s = sum(len(set(up) & adj[x] & adj[y]) for y in up if y in adj[x])
            k4[at(a, x)] += s // 2
    for u in range(n):
        cnt = {}
        low = [v for v in nb[u] if v > u]
        for v in low:
            for w in nb[v]:
                if w > u:
                    cnt[w] = cnt.get(w, 0) + 1
        for v in low:
            for w in nb[v]:
                if w > u:
                    assert cnt[w] <= deg[order[w]]   # fits the counter of w's degree
                    cyc[at(u, v)] += cnt[w] - 1
                    cyc[at(v, w)] += cnt[w] - 1
    return {key[e]: (t[e], k4[e], cyc[e] - D[e] + 2 * t[e] + 2 * k4[e]) for e in key}


@pytest.mark.parametrize("kind", ["er", "rmat", "ba", "rgg", "k5"])
def test_passes_give_the_oracles_counts(kind):
    if kind == "er":
        src, dst = pgd.erdos_renyi(34, 0.5, seed=1)
    elif kind == "rmat":
        src, dst = pgd.rmat(6, 6, seed=2)
    elif kind == "ba":
        src, dst = pgd.barabasi_albert(60, 4, seed=3)
    elif kind == "rgg":
        src, dst = pgd.rgg3d(90, 0.3, seed=4)
    else:
        src, dst = (np.array(v, np.int32) for v in zip(*itertools.combinations(range(5), 2)))
    got = rank_counts(src, dst)
    o = ol.OracleGraph.from_pairs(src, dst, dedup=True).run(order="natural", micro=True)
    a, b, cols = o.micro()
    assert len(cols) == len(got)
    for x, y, row in zip(a.tolist(), b.tolist(), cols.tolist()):
        assert got[(min(x, y) - 1, max(x, y) - 1)] == (row[0], row[2], row[5])
