"""Dense batch graphs at the edges of the tensor-core tiles of k4 (64 columns per
stage, 128 edges and 256 rows per tile, the number of stages that fits, degree
1088): every count equals the one of the passes for a single graph.  All counts
are exact."""
import numpy as np
import pytest

import pgd_gb300 as pgd

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = pgd.Context(device=0)
    yield c
    c.close()


def complete(n):
    a, b = np.triu_indices(n, 1)
    return a.astype(np.int32), b.astype(np.int32)


def single(c, src, dst):
    g = c.graph_from_edges(src, dst, dedup=True)
    g.sort_edges("deg")
    r = g.decompose(micro=False)
    g.destroy()
    return r


@pytest.mark.parametrize("sizes", [(65, 66, 128, 129, 130), (193, 257, 258, 321), (513, 514, 769), (1025, 1088),
                                   (1089, 1090)])
def test_complete_graphs(ctx, sizes):
    for n, r in zip(sizes, ctx.decompose_pairs_batch([complete(n) for n in sizes])):
        t = n - 2
        m = n * (n - 1) // 2
        assert r.n == n and r.m == m
        assert int(r.sums[0]) == m * t and int(r.sums[3]) == m * (t * (t - 1) // 2) and int(r.sums[4]) == 0


def test_random_graphs_equal_the_single_graph_passes(ctx):
    graphs = [pgd.erdos_renyi(n, p, seed=n) for n, p in ((70, 0.95), (300, 0.45), (515, 0.5), (700, 0.4), (1030, 0.26),
                                                         (2048, 0.5), (2048, 0.1), (1500, 0.7))]
    for (src, dst), r in zip(graphs, ctx.decompose_pairs_batch(graphs)):
        w = single(ctx, src, dst)
        assert r.m == w.m and (r.sums == w.sums).all() and (r.totals == w.totals).all()
