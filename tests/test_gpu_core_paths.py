"""k-core numbers on both sides of the weight (row entries and three quarters of
the vertices, 6 million) up to which one cluster peels a graph, and beyond it
where the whole device hands the rest over to the cluster, with a frontier and
without one; and the largest vertex ids.  All values are exact."""
import numpy as np
import pytest

import oracle_lib as ol
import pgd_gb300 as pgd

pytestmark = pytest.mark.gpu


def grid(w):
    i = np.arange(w * w, dtype=np.int32).reshape(w, w)
    return np.r_[i[:, :-1].ravel(), i[:-1].ravel()], np.r_[i[:, 1:].ravel(), i[1:].ravel()]


def random_pairs(n, k):
    p = np.random.default_rng(n + k).integers(0, n, (2, k), dtype=np.int32)
    p[0, -1], p[1, -1] = 0, n - 1
    return p[0], p[1]


@pytest.mark.parametrize("kind", ["below the line", "above the line", "isolated vertices", "grid", "rmat", "dense"])
def test_core_numbers_by_weight(ctx, kind):
    src, dst = {"below the line": lambda: random_pairs(262144, 5 << 19),
                "above the line": lambda: random_pairs(262144, 6 << 19),
                "isolated vertices": lambda: random_pairs(9000000, 200000),
                "grid": lambda: grid(1500),                                 # over a thousand narrow steps
                "rmat": lambda: pgd.rmat(18, 16, seed=2),                   # hundreds of levels
                "dense": lambda: pgd.erdos_renyi(3600, 0.7, seed=3)}[kind]()  # thousands of possible levels
    g = ctx.graph_from_edges(src, dst, dedup=True)
    top, core = g.compute_cores(), g.kcore()
    g.destroy()
    o = ol.OracleGraph.from_pairs(src, dst, dedup=True)
    o.prepare(order="kcore")
    assert (np.asarray(core) == np.asarray(o.kcore())).all()
    assert top == int(np.asarray(core)[1:-1].max())


def test_largest_vertex_ids():
    """Vertex 2^31 - 1, among 2^31: about 90 GB of arrays by vertex."""
    import torch

    if torch.cuda.mem_get_info()[0] < 160 << 30:
        pytest.skip("needs 160 GB of free device memory")
    last = 2 ** 31 - 1
    src, dst = np.random.default_rng(1).integers(0, last + 1, (2, 400000)).astype(np.int32)
    src[:3], dst[:3] = [last, last - 1, last], [last - 1, last - 2, last - 2]   # a triangle at the end
    c = pgd.Context()
    g = c.graph_from_edges(src, dst, dedup=True)
    want = np.unique(np.stack([np.minimum(src, dst), np.maximum(src, dst)])[:, src != dst], axis=1)
    assert g.n == last + 1 and g.m == want.shape[1]
    assert g.compute_cores() == 2
    ev, eu, _ = g.preprocess("natural").edges(with_order=False)
    got = np.unique(np.stack([np.minimum(ev, eu), np.maximum(ev, eu)]), axis=1)
    assert (got == want).all()
    g.destroy()
    c.close()


@pytest.mark.parametrize("k", [3, 3000])
def test_more_vertices_than_ids_are_refused(ctx, k):
    """n_min beyond 2^31: the k-core and the ranks would number vertices past 32 bits."""
    p = np.arange(k, dtype=np.int32)
    held = ctx.resident_bytes
    with pytest.raises(pgd.PGDError) as e:
        ctx.graph_from_edges(p, p + 1, n_min=2 ** 31 + 1)
    assert e.value.status == 1 and ctx.resident_bytes == held   # PGD_EINVAL
