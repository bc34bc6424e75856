"""Both sides of the sizes up to which a graph is built, ordered and ranked by one
block per stage (2,048 pairs, 8,192 vertices) and of the row entries (2^20) up to
which one block peels the k-core: every count and the edge order equal the
oracle's, and what is refused is refused on either side."""
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


def compare(ctx, src, dst, order="deg", neigh="deg", s2l=False):
    g = ctx.graph_from_edges(src, dst, dedup=True)
    g.preprocess(neigh)
    g.sort_edges(order, s2l=s2l)
    r = g.decompose(micro=True)
    got = g.micro()
    info = g.info()
    g.destroy()
    o = ol.OracleGraph.from_pairs(src, dst, dedup=True).run(order=order, neigh=neigh, s2l=s2l, micro=True)
    assert (r.totals == o.totals()).all()
    for a, b in zip(got, o.micro()):
        assert (a == b).all()
    return info


def with_repeats(n, k, seed):
    """k pairs below n: repeated and reversed ones, self loops, the last id used."""
    rng = np.random.default_rng(seed)
    p = rng.integers(0, n, (k, 2)).astype(np.int32)
    p[: k // 8] = p[k // 8 : 2 * (k // 8)][:, ::-1]
    p[k // 2 : k // 2 + 3, 1] = p[k // 2 : k // 2 + 3, 0]
    p[-1] = (0, n - 1)
    return np.ascontiguousarray(p[:, 0]), np.ascontiguousarray(p[:, 1])


@pytest.mark.parametrize("n,k", [(2, 9), (40, 33), (90, 2047), (120, 2048), (120, 2049), (8192, 2048), (8193, 2048),
                                 (8192, 2049)])
@pytest.mark.parametrize("order,neigh,s2l", [("deg", "deg", False), ("kcore", "natural", True),
                                             ("natural", "kcore", False), ("deg_vol", "deg", True)])
def test_around_the_one_block_sizes(ctx, n, k, order, neigh, s2l):
    info = compare(ctx, *with_repeats(n, k, n + k), order=order, neigh=neigh, s2l=s2l)
    assert info.self_loops >= 3 and info.duplicates >= 1


@pytest.mark.parametrize("n", [63, 64, 65])   # 1,953, 2,016 and 2,080 edges
def test_small_complete_graph(ctx, n):
    a, b = np.triu_indices(n, 1)
    compare(ctx, a.astype(np.int32), b.astype(np.int32))


@pytest.mark.parametrize("k", [2048, 2049])
def test_refusals_are_the_same_on_both_sides(ctx, k):
    a = np.arange(k, dtype=np.int32) % 64
    b = 64 + np.arange(k, dtype=np.int32) // 64
    with pytest.raises(pgd.PGDError):
        ctx.graph_from_edges(np.append(a[1:], a[1]), np.append(b[1:], b[1]), dedup=False)
    with pytest.raises(pgd.PGDError):
        ctx.graph_from_edges(np.append(a[1:], -1).astype(np.int32), b, dedup=True)


@pytest.mark.parametrize("n", [1024, 1025])   # 1,047,552 and 1,049,600 entries
def test_core_numbers_around_the_one_block_size(ctx, n):
    a, b = np.triu_indices(n, 1)
    tail = np.arange(1, 60, dtype=np.int64)   # a path hung on the clique
    src, dst = np.r_[a, n - 2 + tail].astype(np.int32), np.r_[b, n - 1 + tail].astype(np.int32)
    if n == 1024:
        src, dst = src[200:], dst[200:]       # below the line with the path
    g = ctx.graph_from_edges(src, dst, dedup=True)
    core = g.kcore()
    g.destroy()
    o = ol.OracleGraph.from_pairs(src, dst, dedup=True)
    o.prepare(order="kcore")
    assert (np.asarray(core) == np.asarray(o.kcore())).all()


@pytest.mark.parametrize("kind", ["path", "star", "ladder", "matching", "ba"])
def test_core_numbers_by_chain_and_width(ctx, kind):
    """One link per step, one step of every vertex, and more vertices than the
    one block's queue and its 32,000 or so vertices hold."""
    p = np.arange(9000, dtype=np.int32)
    src, dst = {"path": (p[:-1], p[1:]), "star": (np.zeros(8999, np.int32), p[1:]),
                "ladder": (np.r_[p[:-1], p[:-100]], np.r_[p[1:], p[100:]]),
                "matching": (2 * p[:8000], 2 * p[:8000] + 1), "ba": pgd.barabasi_albert(40000, 3, seed=1)}[kind]
    g = ctx.graph_from_edges(src, dst, dedup=True)
    core = g.kcore()
    g.destroy()
    o = ol.OracleGraph.from_pairs(src, dst, dedup=True)
    o.prepare(order="kcore")
    assert (np.asarray(core) == np.asarray(o.kcore())).all()
