"""Counts: a result of its own, whose fields a program may replace (no GPU)."""
import ctypes
import pickle

import numpy as np

import pgd_gb300 as pgd


def filled(k):
    out = (pgd.pgd_counts * k)()
    for i, c in enumerate(out):
        c.totals[:] = [100 * i + j for j in range(pgd.NTOTALS)]
        c.sums[:] = [1000 * i + j for j in range(pgd.NSUMS)]
        c.n, c.m, c.kernel_ms, c.hub_ms, c.tri_ms = i, 2 * i, 0.5 * i, 0.25, 0.125
    return out


def check(r, i):
    assert r.totals.tolist() == [100 * i + j for j in range(pgd.NTOTALS)]
    assert r.sums.tolist() == [1000 * i + j for j in range(pgd.NSUMS)]
    assert r.totals.dtype == r.sums.dtype == np.uint64
    assert (r.n, r.m, r.kernel_ms, r.hub_ms, r.tri_ms) == (i, 2 * i, 0.5 * i, 0.25, 0.125)
    assert type(r.n) is int and type(r.m) is int and type(r.kernel_ms) is float


def test_fields_can_be_replaced_and_added():
    for r in (pgd.Counts(filled(1)[0]), pgd._counts_list(filled(3))[2]):
        i = 0 if r.n == 0 else 2
        check(r, i)
        r.totals = r.totals + np.uint64(1)
        r.sums += np.uint64(2)
        r.n, r.m, r.kernel_ms, r.note = 7, 8, 9.5, "kept"
        assert r.totals[1] == 100 * i + 2 and r.sums[3] == 1000 * i + 5
        assert (r.n, r.m, r.kernel_ms, r.note) == (7, 8, 9.5, "kept")
        assert r.as_dict()[pgd.TOTAL_NAMES[1]] == 100 * i + 2
        assert pickle.loads(pickle.dumps(r)).totals[1] == 100 * i + 2


def test_a_result_does_not_follow_its_source():
    out = filled(2)
    r = pgd.Counts(out[1])
    ctypes.memset(out, 0, ctypes.sizeof(out))
    check(r, 1)


def test_results_of_a_batch():
    res = pgd._counts_list(filled(5))
    for i, r in enumerate(res):
        check(r, i)
    res[1].totals[0] = 9
    check(res[2], 2)
    assert pgd._counts_list((pgd.pgd_counts * 0)()) == []
