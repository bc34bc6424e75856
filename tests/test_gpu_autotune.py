"""The autotuner times candidates that differ in the work they do, and leaves alone
what no batch reads."""
import pytest

import pgd_gb300 as pgd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own", [None, (128, 40, 700)])
def test_sparse_graphs_leave_the_thresholds(own):
    """No graph takes the matrix kernels: one candidate, nothing to choose."""
    c = pgd.Context()
    if own:
        c.set_thresholds(*own)
    before, degree = c.thresholds(), c.tensor_min_degree()
    graphs = [c.graph_from_edges(*pgd.barabasi_albert(600 + 50 * i, 3, seed=i)) for i in range(6)]
    c.decompose_batch(graphs)
    launches = c.kernel_launches
    c.decompose_batch(graphs)
    once = c.kernel_launches - launches
    a, h, d, ms = c.autotune(graphs, reps=2)
    assert (a, h, d) == c.thresholds() == before and c.tensor_min_degree() == degree and ms > 0
    assert c.kernel_launches - launches - once == 2 * once
    c.close()


def test_hub_thresholds_are_not_tuned_on_a_batch():
    c = pgd.Context()
    c.set_thresholds(100, 50)
    graphs = [c.graph_from_edges(*pgd.erdos_renyi(n, 0.5, seed=n)) for n in (100, 200, 300, 1100)]
    a, h, d, _ = c.autotune(graphs, reps=1)
    assert (a, h) == (100, 50) == c.thresholds()[:2] and d in (0, 256, 1024, 2048)
    c.close()
