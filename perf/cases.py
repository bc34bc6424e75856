"""The calls that users of this library make, as cases to be timed.

Each case is one whole call sequence through the public Python binding, over the
shapes of the repository's own configurations, tests and benchmarks: one small
graph per call, the small dense configuration, the power-law, mesh-like and
preferential-attachment graphs of the large ones, a graph file, a sample of the
edges and batches of many graphs.  A case is a dict of plain values:

  kind   what is called (see run)
  graph  "rmat" (scale, ef), "rgg" (n, mean degree deg), "ba" (n, attach),
         "er" (n, p); batches: "uneven" or "proteins" (count)

Inputs come from the seed alone.  Host inputs are numpy arrays, because that
is what the entry points take; result rows of the resident cases go to
page-locked buffers that a program keeps.
"""
import concurrent.futures as cf
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import pgd_gb300 as pgd

_ctx = None


def _context():
    """One context per process, as a program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = pgd.Context(device=0)
    return _ctx


def listed():
    return [
        # one small sparse graph per call, global counts: latency and launches
        {"name": "call-er96", "kind": "call", "graph": "er", "n": 96, "p": 0.06},
        # the small dense configuration, host pairs in, per-edge rows out
        {"name": "rows-er250-dense", "kind": "rows", "graph": "er", "n": 250, "p": 0.9, "order": "deg"},
        # a mid-size social graph end to end in k-core order, per-edge rows out
        {"name": "rows-rmat16", "kind": "rows", "graph": "rmat", "scale": 16, "ef": 16, "order": "kcore"},
        # a graph file through the reader, global counts (the command line's work)
        {"name": "file-rmat14", "kind": "file", "graph": "rmat", "scale": 14, "ef": 16, "order": "kcore"},
        # the headline: a resident power-law graph, k-core order, per-edge rows
        {"name": "resident-rmat20", "kind": "resident", "graph": "rmat", "scale": 20, "ef": 16, "order": "kcore"},
        # a resident mesh-like graph: even degrees, many triangles
        {"name": "resident-rgg20", "kind": "resident", "graph": "rgg", "n": 1 << 20, "deg": 24.0, "order": "kcore"},
        # a resident sparse social graph: hubs, few triangles
        {"name": "resident-ba-200k", "kind": "resident", "graph": "ba", "n": 200003, "attach": 8, "order": "deg"},
        # one tenth of the edges of a resident graph (the sampled edge order)
        {"name": "sample-rmat17", "kind": "sample", "graph": "rmat", "scale": 17, "ef": 16, "order": "deg",
         "share": 0.1},
        # the batched configuration: uneven graphs, half of them dense
        {"name": "batch-uneven256", "kind": "batch", "graph": "uneven", "count": 256},
        # many small sparse graphs (graph-classification data sets): one call
        {"name": "batch-proteins1178", "kind": "batch", "graph": "proteins", "count": 1178},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "rows", "file", "resident", "resident", "sample", "batch", "batch"])
    if kind == "batch":
        graph = rng.choice(["uneven", "proteins"])
        return {"kind": kind, "graph": graph, "count": _log_int(rng, 1, 320 if graph == "uneven" else 1500)}
    if kind == "call":
        n = _log_int(rng, 12, 3000)
        return {"kind": kind, "graph": "er", "n": n, "p": round(min(0.9, rng.uniform(2.0, 12.0) / n), 6)}
    c = {"kind": kind, "order": rng.choice(["deg", "kcore", "natural", "kcore_deg", "deg_vol"])}
    if kind == "sample":
        c["share"] = round(math.exp(rng.uniform(math.log(0.002), math.log(0.6))), 4)
    graph = rng.choice(["rmat", "rmat", "rgg", "ba", "er"])
    big = kind == "resident"
    if graph == "rmat":
        c.update(graph=graph, scale=rng.randint(10, 19 if big else 16), ef=_log_int(rng, 4, 24))
    elif graph == "rgg":
        c.update(graph=graph, n=_log_int(rng, 1000, 900000 if big else 60000), deg=round(rng.uniform(6.0, 40.0), 2))
    elif graph == "ba":
        c.update(graph=graph, n=_log_int(rng, 1000, 400000 if big else 60000), attach=rng.randint(2, 12))
    else:
        c.update(graph=graph, n=_log_int(rng, 100, 1500), p=round(rng.uniform(0.05, 0.9), 3))
    return c


def _radius(case):
    return (3.0 * case["deg"] / (4.0 * math.pi * case["n"])) ** (1.0 / 3.0)


def _pairs(case, seed):
    graph = case["graph"]
    if graph == "rmat":
        return pgd.rmat(case["scale"], case["ef"], seed=seed)
    if graph == "rgg":
        return pgd.rgg3d(case["n"], _radius(case), seed=seed)
    if graph == "ba":
        return pgd.barabasi_albert(case["n"], case["attach"], seed=seed)
    return pgd.erdos_renyi(case["n"], case["p"], seed=seed)


def _distinct(case):
    """Distinct edges of a case with per-edge rows: below what any seed gives
    (R-MAT draws an edge more than once, more often on small vertex sets)."""
    pairs, n = _edges(case)
    if case["graph"] == "rmat":
        return int(pairs * (0.93 - 0.03 * (20 - case["scale"]) - 0.008 * max(0, case["ef"] - 16)))
    if case["graph"] == "ba":
        return int(pairs) - case["attach"] * case["attach"]
    inside = 0.99 - 1.15 * _radius(case) if case["graph"] == "rgg" else 1.0   # points near the cube's faces
    return int(pairs * inside - 5.0 * math.sqrt(pairs))


def _simple(case, seed):
    """The case's graph as _distinct(case) distinct pairs in random order and
    direction, so that every seed has as many per-edge rows."""
    src, dst = (torch.from_numpy(x).cuda().long() for x in _pairs(case, seed))
    lo, hi = torch.minimum(src, dst), torch.maximum(src, dst)
    key = torch.unique((lo << 32 | hi)[lo != hi])
    m = _distinct(case)
    if len(key) < m:
        raise ValueError("%d distinct edges, %d wanted: %r" % (len(key), m, case))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    at = torch.randperm(len(key), generator=gen, device="cuda")[:m]
    lo, hi, flip = key[at] >> 32, key[at] & 0xffffffff, (at & 1).bool()
    return (torch.where(flip, hi, lo).int().cpu().numpy(), torch.where(flip, lo, hi).int().cpu().numpy())


def _many(case, seed):
    """The graphs of a batch: a list of (src, dst)."""
    rng = np.random.default_rng([seed, case["count"]])
    jobs = []
    for i in range(case["count"]):
        s = int(rng.integers(1, 1 << 30))
        if case["graph"] == "uneven":        # n ~ U[16, 2048]; half G(n, p), half preferential attachment
            n = int(rng.integers(16, 2049))
            jobs.append((pgd.erdos_renyi, n, float(rng.uniform(0.01, 0.5)), s) if i % 2 == 0
                        else (pgd.barabasi_albert, n, int(rng.integers(2, 9)), s))
        else:                                # geometric contact graphs, mean degree about 5
            n = max(30, min(3000, int(np.exp(rng.normal(math.log(240.0), 0.55)))))
            jobs.append((pgd.rgg3d, n, (3.0 * 5.5 / (4.0 * math.pi * n)) ** (1.0 / 3.0), s))
    with cf.ThreadPoolExecutor(os.cpu_count() or 4) as ex:
        return list(ex.map(lambda j: j[0](j[1], j[2], seed=j[3]), jobs))


def _pinned(a):
    return torch.from_numpy(a).pin_memory().numpy()


class _File:
    """A graph file on disk, removed with the state."""

    def __init__(self, src, dst):
        a, b = np.minimum(src, dst).astype(np.int64), np.maximum(src, dst).astype(np.int64)
        key = np.unique((a << 32 | b)[a != b])
        ids = np.stack([key & 0xffffffff, key >> 32], 1) + 1     # 1-based, the larger id first
        n = int(ids.max()) if len(ids) else 1
        self.dir = tempfile.mkdtemp(prefix="pgd_case_")
        self.path = os.path.join(self.dir, "graph.mtx")
        with open(self.path, "w") as f:
            f.write("%%%%MatrixMarket matrix coordinate pattern symmetric\n%d %d %d\n" % (n, n, len(ids)))
            f.write("%d %d\n" * len(ids) % tuple(ids.ravel().tolist()))

    def __del__(self):
        shutil.rmtree(self.dir, ignore_errors=True)


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "ctx": _context(), "order": case.get("order", "deg")}
    if kind == "batch":
        off, src, dst = pgd.concat_pairs(_many(case, seed))
        state.update(off=off, src=_pinned(src), dst=_pinned(dst))
        return state
    src, dst = _pairs(case, seed) if kind in ("call", "file") else _simple(case, seed)
    if kind in ("call", "rows"):
        state.update(src=src, dst=dst)
    elif kind == "file":
        state.update(file=_File(src, dst))
    else:
        g = state["ctx"].graph_from_edges(src, dst, dedup=True)
        g.preprocess("deg")
        if "kcore" in state["order"]:
            g.compute_cores()
        rows = g.m
        if kind == "sample":
            rng = np.random.default_rng(seed)
            rows = max(1, int(g.m * case["share"]))
            state["ids"] = np.sort(rng.choice(g.m, rows, replace=False)).astype(np.int64)
        buf = torch.empty((max(1, rows), pgd.NMICRO), dtype=torch.int64, pin_memory=True)
        state.update(g=g, rows=buf.numpy().view(np.uint64))
    return state


def _signed(a):
    return np.ascontiguousarray(a).view(np.int64)


def run(state):
    kind, ctx, order = state["kind"], state["ctx"], state["order"]
    if kind == "call":            # one graph, global counts
        g = ctx.graph_from_edges(state["src"], state["dst"])
        r = g.decompose(micro=False)
        g.destroy()
        return {"totals": _signed(r.totals), "sums": _signed(r.sums)}
    if kind == "rows":            # host pairs -> per-edge rows on the host
        g = ctx.graph_from_edges(state["src"], state["dst"], dedup=True)
        g.preprocess("deg")
        k = g.compute_cores()
        g.sort_edges(order)
        r = g.decompose(micro=True)
        src, dst, cols = g.micro()
        g.destroy()
        return {"totals": _signed(r.totals), "sums": _signed(r.sums), "max_core": k, "src": src, "dst": dst,
                "cols": _signed(cols)}
    if kind == "file":            # file -> global counts, as the command line does it
        g = ctx.graph_from_file(state["file"].path)
        g.preprocess("deg")
        k = g.compute_cores()
        g.sort_edges(order)
        r = g.decompose(micro=False)
        g.destroy()
        return {"totals": _signed(r.totals), "sums": _signed(r.sums), "max_core": k}
    if kind in ("resident", "sample"):   # order + decomposition of a graph on the device, rows to the host
        g = state["g"]
        if kind == "sample":
            g.sort_edges_sample(state["ids"], order)
        else:
            g.sort_edges(order)
        r = g.decompose(micro=True)
        cols = g.micro(ids=False, out=state["rows"])
        return {"totals": _signed(r.totals), "sums": _signed(r.sums), "cols": _signed(cols)}
    res = ctx.decompose_pairs_batch_flat(state["off"], state["src"], state["dst"])
    return {"totals": _signed(np.stack([r.totals for r in res])), "sums": _signed(np.stack([r.sums for r in res]))}


def exact(case, seed):
    """Every output is a whole number: compared as it is, bit for bit."""
    return None


def _edges(case):
    """Expected pairs and vertices of a case's input."""
    graph = case["graph"]
    if graph == "rmat":
        return case["ef"] * float(1 << case["scale"]), float(1 << case["scale"])
    if graph == "rgg":
        return 0.5 * case["deg"] * case["n"], float(case["n"])
    if graph == "ba":
        return float(case["attach"] * case["n"]), float(case["n"])
    if graph == "er":
        return 0.5 * case["p"] * case["n"] * (case["n"] - 1), float(case["n"])
    k = case["count"]
    if graph == "uneven":
        return k * (0.5 * 0.255 * 0.5 * 1.40e6 + 0.5 * 5.0 * 1032), k * 1032.0
    return k * 2.4 * 280.0, k * 280.0


def work(case):
    """Bytes a pass cannot do without: its input read once (host pairs, the
    file, or the resident CSR) and its results written once.  The counting
    itself is integer work, so no floating-point operations."""
    pairs, n = _edges(case)
    kind = case["kind"]
    row = 8 * pgd.NMICRO
    counts = 8 * (pgd.NTOTALS + pgd.NSUMS)
    if kind == "rows":
        b = 8 * pairs + (row + 16) * pairs
    elif kind == "file":
        b = 13 * pairs
    elif kind == "resident":
        b = 8 * pairs + 8 * n + row * pairs
    elif kind == "sample":
        b = 8 * pairs + 8 * n + (row + 8) * pairs * case["share"]
    else:
        b = 8 * pairs
    if kind == "batch":
        counts *= case["count"]
    return {"bytes": b + counts, "flops": 0.0}
