"""The rank-ordered passes (rank_path.cu) at the edges of their work classes:
neighbourhood sizes around the warp / block / global-table limits, wedge counts
around the warp / block / counter-array limits, every counter width, and both
sides of the sample-size rule.  Complete and complete bipartite graphs have
closed forms; the rest is compared with the oracle.  All counts are exact, so
every comparison is for equality."""
import numpy as np
import pytest

import oracle_lib as ol
import pgd_gb300 as pgd

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = pgd.Context(device=0)
    yield c
    c.close()


def rows_of(ctx, src, dst, order="deg"):
    g = ctx.graph_from_edges(src, dst, dedup=True)
    g.sort_edges(order)
    r = g.decompose(micro=True)
    rows = g.micro()
    g.destroy()
    return r, rows


@pytest.mark.parametrize("n", [3, 4, 32, 33, 34, 35, 257, 258, 513, 514, 1025, 1026])
def test_complete_graph(ctx, n):
    a, b = np.triu_indices(n, 1)
    r, (_, _, cols) = rows_of(ctx, a.astype(np.int32), b.astype(np.int32))
    t = n - 2
    k4 = t * (t - 1) // 2
    assert r.m == n * (n - 1) // 2
    assert (cols[:, 0] == t).all() and (cols[:, 2] == k4).all()
    assert (cols[:, 3] == 0).all() and (cols[:, 5] == 0).all()
    assert int(r.totals[6]) == n * (n - 1) * (n - 2) * (n - 3) // 24


# degrees on both sides of the counter widths (4, 16, 256, 65536) and wedge
# counts on both sides of 512 and 4096
@pytest.mark.parametrize("a,b", [(2, 2), (2, 3), (3, 4), (4, 16), (15, 17), (16, 32), (16, 33), (64, 65), (32, 129),
                                 (255, 257), (300, 700), (2, 65535), (2, 65537), (3, 70000)])
def test_complete_bipartite_graph(ctx, a, b):
    src = np.repeat(np.arange(a), b).astype(np.int32)
    dst = (a + np.tile(np.arange(b), a)).astype(np.int32)
    r, (_, _, cols) = rows_of(ctx, src, dst)
    assert (cols[:, 0] == 0).all() and (cols[:, 2] == 0).all()
    assert (cols[:, 5] == (a - 1) * (b - 1)).all()
    assert int(r.totals[9]) == a * (a - 1) // 2 * (b * (b - 1) // 2)


@pytest.mark.parametrize("kind,order", [("er", "deg"), ("rmat", "kcore"), ("ba", "natural"), ("rgg", "deg_vol"),
                                        ("star+clique", "deg")])
def test_random_graphs_match_the_oracle(ctx, kind, order):
    if kind == "er":
        src, dst = pgd.erdos_renyi(420, 0.7, seed=3)
    elif kind == "rmat":
        src, dst = pgd.rmat(11, 14, seed=4)
    elif kind == "ba":
        src, dst = pgd.barabasi_albert(3000, 7, seed=5)
    elif kind == "rgg":
        src, dst = pgd.rgg3d(5000, 0.09, seed=6)
    else:   # a hub over a clique: one vertex with many wedges of low-degree ends
        a, b = np.triu_indices(40, 1)
        src = np.concatenate([a, np.zeros(3000, int), np.arange(40, 3039)]).astype(np.int32)
        dst = np.concatenate([b, np.arange(40, 3040), np.arange(41, 3040)]).astype(np.int32)
    r, (x, y, cols) = rows_of(ctx, src, dst, order)
    o = ol.OracleGraph.from_pairs(src, dst, dedup=True).run(order=order, micro=True)
    ox, oy, ocols = o.micro()
    assert (r.totals == o.totals()).all()
    assert (x == ox).all() and (y == oy).all() and (cols == ocols).all()


@pytest.mark.parametrize("share", [0.0003, 0.0006, 0.005, 0.014, 0.017, 0.5])
def test_sample_rows_equal_the_full_run(ctx, share):
    """Samples below and above the share of edges from which the passes over
    the whole graph are taken give the same rows."""
    src, dst = pgd.rmat(12, 10, seed=8)
    g = ctx.graph_from_edges(src, dst, dedup=True)
    g.sort_edges("natural")
    g.decompose(micro=True)
    full = {(a, b): tuple(c) for a, b, c in zip(*[v.tolist() for v in g.micro()])}
    rng = np.random.default_rng(1)
    ids = np.sort(rng.choice(g.m, max(1, int(g.m * share)), replace=False))
    g.sort_edges_sample(ids, "deg")
    r = g.decompose(micro=True)
    s, d, c = g.micro()
    assert len(c) == len(ids)
    assert all(full[(a, b)] == tuple(v) for a, b, v in zip(s.tolist(), d.tolist(), c.tolist()))
    assert int(r.sums[0]) == sum(full[(a, b)][0] for a, b in zip(s.tolist(), d.tolist()))
    g.destroy()
