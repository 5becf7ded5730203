"""The most edges a call accepts: positions near 2^31 in the first pass."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_last_edges_of_the_range(tchll):
    """2^31 - 1 times the edge (0, 1) of one triangle.  (About 60 GB of device
    memory for the edges and the workspace.)"""
    import torch
    from triangle_counting_hll_b200 import _lib, core
    n = 2**31 - 1
    rp, ci = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, 2, 3, 3], [1, 2, 2]))
    u = torch.zeros(n, dtype=torch.int32, device="cuda")
    v = torch.ones(n, dtype=torch.int32, device="cuda")
    try:
        res, _ = core.exact_count_tensors(rp, ci, u, v)
        r = _lib.read_count_result(res)
        assert (r.status, r.exact, r.n_exact) == (0, n, n)
    finally:
        del u, v
        _lib.workspace.clear()
        torch.cuda.empty_cache()
