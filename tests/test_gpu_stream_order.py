"""Pairs in page-locked memory that the caller's stream is still filling are read
in the order of that stream, by graphs of either size."""
import numpy as np
import pytest

import pgd_gb300 as pgd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [300, 2048, 2049])
def test_pairs_filled_on_the_callers_stream(k):
    import torch

    p = np.random.default_rng(k).integers(0, 150, (2, k)).astype(np.int32)
    src, dst = (torch.full((k,), x, dtype=torch.int32).pin_memory() for x in (3, 4))   # other pairs until then
    d_src, d_dst = (torch.from_numpy(x).cuda() for x in p)
    s = torch.cuda.Stream()
    c = pgd.Context(stream=s.cuda_stream)
    want = c.graph_from_edges(*p, dedup=True)
    s.wait_stream(torch.cuda.current_stream())
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(100000000)          # some 50 ms
        src.copy_(d_src, non_blocking=True)
        dst.copy_(d_dst, non_blocking=True)
    g = c.graph_from_edges(src.numpy(), dst.numpy(), dedup=True)
    assert (g.n, g.m) == (want.n, want.m) and (g.decompose().totals == want.decompose().totals).all()
    g.destroy()
    want.destroy()
    c.close()
