"""Samples of dense graphs on both sides of the share up to which they are
decomposed edge by edge: the rows are the whole graph's.  All counts are exact."""
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
