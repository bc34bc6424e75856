"""A graph that was decomposed takes a new neighbour order: its edge ids change,
and the next decomposition (whole graph or sample) gives the counts of the new
ids.  All counts are exact, so every comparison is for equality."""
import numpy as np
import pytest

import oracle_lib as ol
import pgd_gb300 as pgd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", ["one block per stage", "grid-wide stages"])
def test_counts_follow_a_new_neighbour_order(ctx, pairs):
    src, dst = pgd.rmat(7, 10, seed=3) if pairs == "one block per stage" else pgd.rmat(11, 8, seed=3)
    g = ctx.graph_from_edges(src, dst, dedup=True)
    rng = np.random.default_rng(5)
    ids = []
    for neigh, s2l, order in [("deg", False, "deg"), ("kcore", False, "kcore"), ("natural", False, "deg_vol"),
                              ("deg", True, "natural"), ("deg", False, "kcore_deg")]:
        g.preprocess(neigh, s2l=s2l)
        g.sort_edges(order)
        r = g.decompose(micro=True)
        got = g.micro()
        o = ol.OracleGraph.from_pairs(src, dst, dedup=True).run(neigh=neigh, s2l_neigh=s2l, order=order, micro=True)
        assert (r.totals == o.totals()).all()
        for a, b in zip(got, o.micro()):
            assert (a == b).all()
        ids.append(g.edges(with_order=False)[0])
        # a sample under the same ids: its rows are the whole graph's
        rows = {(a, b): tuple(c) for a, b, c in zip(*[v.tolist() for v in got])}
        pick = np.sort(rng.choice(g.m, g.m // 3, replace=False))
        g.sort_edges_sample(pick, order)
        g.decompose(micro=True)
        s, d, c = g.micro()
        assert len(c) == len(pick)
        assert all(rows[(a, b)] == tuple(v) for a, b, v in zip(s.tolist(), d.tolist(), c.tolist()))
    assert any((x != ids[0]).any() for x in ids[1:])   # the ids did change
    g.destroy()
