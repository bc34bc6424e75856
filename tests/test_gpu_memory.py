"""Memory that a decomposition can do without: the triangles kept between the
passes and the table of range positions of the 4-cycle pass.  Where the budget
has no room for them the counts are the same, and every class of the passes that
list the triangles again is run.  All counts are exact."""
import ctypes

import numpy as np
import pytest

import pgd_gb300 as pgd

pytestmark = pytest.mark.gpu

MB = 1 << 20


def decomposed(budget, src, dst, micro=True):
    """Counts, rows and resident bytes of a graph in a context of `budget` bytes."""
    c = pgd.Context(hbm_budget=budget)
    g = c.graph_from_edges(src, dst, dedup=True)
    g.sort_edges("deg")
    r = g.decompose(micro=micro)
    rows = g.micro() if micro else None
    held = g.resident_bytes
    g.destroy()
    c.close()
    return r, rows, held


def complete(n):
    a, b = np.triu_indices(n, 1)
    return a.astype(np.int32), b.astype(np.int32)


@pytest.mark.parametrize("room", [1, 1200])
@pytest.mark.parametrize("kind", ["complete", "dense", "rmat", "geometric"])
def test_triangles_found_again(kind, room):
    """Triangles of more than 256 MB in a context without room for them: with a list
    per block, and without any."""
    src, dst = {"complete": lambda: complete(1100), "dense": lambda: pgd.erdos_renyi(1300, 0.9, seed=1),
                "rmat": lambda: pgd.rmat(17, 16, seed=2), "geometric": lambda: pgd.rgg3d(20000, 0.17, seed=3)}[kind]()
    r, rows, held = decomposed(0, src, dst)
    w, wrows, _ = decomposed(held + room * MB, src, dst)
    assert (r.sums == w.sums).all() and (r.totals == w.totals).all()
    for a, b in zip(rows, wrows):
        assert (a == b).all()
    if kind == "complete":
        t = 1098
        assert (wrows[2][:, 0] == t).all() and (wrows[2][:, 2] == t * (t - 1) // 2).all()
        assert (wrows[2][:, 5] == 0).all()


def test_range_positions_searched():
    """A budget that holds everything but the table of range positions."""
    src, dst = pgd.rmat(14, 16, seed=4)
    r, _, held = decomposed(0, src, dst, micro=False)
    n2 = int((np.bincount(np.concatenate(pgd_edges(src, dst))) >= 2).sum())
    w, _, small = decomposed(held - 15 * 4 * n2 // 2, src, dst, micro=False)   # half of at least 15 positions a vertex
    assert small < held
    assert (r.sums == w.sums).all() and (r.totals == w.totals).all()


def pgd_edges(src, dst):
    lo, hi = np.minimum(src, dst), np.maximum(src, dst)
    return np.unique(np.stack([lo, hi])[:, lo != hi], axis=1)


class Pool:
    """The device's default memory pool, as the CUDA runtime reports it."""

    def __init__(self):
        self.rt = ctypes.CDLL("libcudart.so.13")
        self.pool = ctypes.c_void_p()
        assert self.rt.cudaDeviceGetDefaultMemPool(ctypes.byref(self.pool), 0) == 0

    def restart(self):
        assert self.rt.cudaMemPoolSetAttribute(self.pool, 8, ctypes.byref(ctypes.c_uint64(0))) == 0   # UsedMemHigh

    def used(self):
        v = ctypes.c_uint64()
        assert self.rt.cudaMemPoolGetAttribute(self.pool, 7, ctypes.byref(v)) == 0   # UsedMemCurrent
        return v.value

    def high(self):
        v = ctypes.c_uint64()
        assert self.rt.cudaMemPoolGetAttribute(self.pool, 8, ctypes.byref(v)) == 0
        return v.value


def test_a_small_budget_bounds_the_lists():
    """1.8 GB of triangles of a complete graph: not where 100 MB are asked for."""
    src, dst = complete(1100)
    p = Pool()
    before = p.used()   # graphs that other tests still hold
    p.restart()
    decomposed(100 * MB, src, dst, micro=False)
    assert p.high() - before < 700 * MB   # 256 MB of lists, the graph, 16 bytes per entry, sort buffers


def test_small_graphs_hold_little():
    """A program may keep thousands of them: 96 vertices and 239 edges in less than
    the 28,532 bytes of the edge-by-edge structures."""
    _, _, held = decomposed(0, *pgd.erdos_renyi(96, 0.06, seed=1), micro=False)
    assert held < 28532


def test_either_path_makes_room_for_the_other():
    """A budget that holds the structures of whole graphs or those of small samples,
    as it held the one set that served both."""
    src, dst = pgd.rmat(14, 16, seed=5)
    big = pgd.Context()
    g = big.graph_from_edges(src, dst, dedup=True)
    g.sort_edges("deg")
    ids = np.arange(7, g.m, g.m // 60, dtype=np.int64)     # below 1/2048 of the edges
    assert len(ids) < g.m // 2048
    g.sort_edges_sample(ids, "natural", s2l=True)
    part = g.decompose(micro=True)
    part_rows, held = g.micro(), g.resident_bytes          # structures of small samples alone
    g.sort_edges("deg")
    whole = g.decompose(micro=True)
    assert g.resident_bytes > held                         # both
    g.destroy()
    big.close()
    c = pgd.Context(hbm_budget=held + MB)
    g = c.graph_from_edges(src, dst, dedup=True)
    for _ in range(2):
        g.sort_edges("deg")
        assert (g.decompose(micro=True).sums == whole.sums).all()
        g.sort_edges_sample(ids, "natural", s2l=True)
        assert (g.decompose(micro=True).sums == part.sums).all()
        for a, b in zip(g.micro(), part_rows):
            assert (a == b).all()
        assert g.resident_bytes <= held + MB
    g.destroy()
    assert c.resident_bytes == 0
    c.close()


@pytest.mark.parametrize("workers,budget", [(1, 400), (2, 800)])
def test_a_servers_budget_bounds_what_its_requests_take(workers, budget):
    """3 GB of triangles in each request, estimated at 180 MB."""
    graphs = [pgd.erdos_renyi(2100, 0.5, seed=i) for i in range(4)]
    want = [decomposed(0, *g, micro=False)[0].totals for g in graphs]
    p = Pool()
    before = p.used()
    p.restart()
    sv = pgd.Server(workers=workers, hbm_budget=budget * MB)
    tickets = [sv.submit(*g) for g in graphs]
    for t, w in zip(tickets, want):
        st, r = sv.wait(t, 120000)
        assert st == 0 and (r.totals == w).all()
    assert sv.stats()["peak_bytes"] <= budget * MB
    sv.close()
    assert p.high() - before <= budget * MB
