"""Samples on both sides of the share up to which they are decomposed edge by edge,
and small ones in every layout of the edge-by-edge kernels' shared memory: the rows
are the whole graph's.  All counts are exact."""
import numpy as np
import pytest

import pgd_gb300 as pgd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p", [(600, 0.9), (1000, 0.5), (1500, 0.3)])
def test_dense_samples(ctx, n, p):
    src, dst = pgd.erdos_renyi(n, p, seed=n)
    g = ctx.graph_from_edges(src, dst, dedup=True)
    g.sort_edges("natural")
    r = g.decompose(micro=True)
    full = {(a, b): tuple(c) for a, b, c in zip(*[v.tolist() for v in g.micro()])}
    rng = np.random.default_rng(n)
    for share in (1 / 2048, 1 / 512, 1 / 128, 1 / 32, 1 / 8, 1 / 3, 1):
        ids = np.sort(rng.choice(g.m, max(1, int(g.m * share)), replace=False))
        g.sort_edges_sample(ids, "deg")
        s = g.decompose(micro=True)
        a, b, cols = g.micro()
        rows = [full[e] for e in zip(a.tolist(), b.tolist())]
        assert rows == [tuple(c) for c in cols.tolist()]
        assert int(s.sums[0]) == sum(c[0] for c in rows) and int(s.sums[3]) == sum(c[2] for c in rows)
    assert (s.sums == r.sums).all()
    g.destroy()


@pytest.mark.parametrize("case", ["16-bit counters in global memory", "32-bit counters in global memory",
                                  "bitmap split", "bitmap of many vertices"])
def test_small_samples_by_layout(case):
    """k_hub keeps its histogram (16-bit counters where the largest degree is below
    65536) in shared memory where it fits, and the bitmap of N(p) in the rest."""
    c = pgd.Context()
    n_min = 0
    if case == "bitmap of many vertices":
        src, dst = pgd.rmat(14, 16, seed=12)
        n_min = 2000000
    else:
        c.set_thresholds(2, 2)
        if case == "32-bit counters in global memory":
            src, dst = pgd.barabasi_albert(70000, 2, seed=13)
            leaves = np.arange(70000, dtype=np.int32)
            src, dst = np.concatenate([src, leaves]), np.concatenate([dst, np.full(70000, 70000, np.int32)])
        else:
            src, dst = pgd.barabasi_albert(120000 if case.startswith("16") else 78000, 6, seed=11)
    g = c.graph_from_edges(src, dst, n_min=n_min)
    g.sort_edges("natural")
    g.decompose(micro=True)
    full = {(a, b): tuple(v) for a, b, v in zip(*[x.tolist() for x in g.micro()])}
    ids = np.arange(3, g.m, 4096, dtype=np.int64)[: g.m // 2048 - 1]
    g.sort_edges_sample(ids, "deg")
    r = g.decompose(micro=True)
    a, b, cols = g.micro()
    rows = [full[e] for e in zip(a.tolist(), b.tolist())]
    assert len(rows) == len(ids) and rows == [tuple(v) for v in cols.tolist()]
    assert int(r.sums[0]) == sum(v[0] for v in rows) and int(r.sums[4]) == sum(v[5] for v in rows)
    g.destroy()
    c.close()
