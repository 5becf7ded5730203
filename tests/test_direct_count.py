"""Small graphs are counted from their edges as given, in one launch: edge
counts around its chunk sizes and its limit, against the regrouped path
(pairs=2) and the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(oracle, m, seed=3):
    """An R-MAT CSR and exactly m of its edges (repeated when it has fewer)."""
    u, v = oracle.gen_rmat(12, 16, 0.57, 0.19, 0.19, seed)
    g = oracle.csr_build(u, v)
    pick = np.sort(np.random.default_rng(seed).integers(0, g["n_edges"], m))
    return g, g["edge_u"][pick].copy(), g["edge_v"][pick].copy()


@pytest.mark.parametrize("m", [1, 7, 8, 9, 31, 33, 98303, 98304, 196608, (1 << 19), (1 << 19) + 1])
def test_edge_counts(tchll, oracle, m):
    import torch
    from triangle_counting_hll_b200 import core
    g, eu, ev = _graph(oracle, m)
    rp, ci, u, v = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g["row_ptr"], g["col_idx"], eu, ev))
    deg = (rp[1:] - rp[:-1]).contiguous()
    slot, n_rows = core.sketch_slots(rp, 16)
    rows = core.build_sketches_compact_tensors(rp, ci, slot, n_rows, 9)
    got = []
    base = core.get_count_tuning()
    try:
        for pairs in (1, 2):
            core.set_count_tuning(**dict(base, pairs=pairs))
            res, _ = core.exact_count_tensors(rp, ci, u, v)
            hres, _ = core.hybrid_count_compact_tensors(rp, ci, u, v, deg, rows, slot, 9, 20, split_kernels=True)
            total, r = core.hybrid_from_result(hres)
            got.append((core.exact_from_result(res), total, r.n_approx, r.n_exact, r.n_fallback, r.n_clamped))
    finally:
        core.set_count_tuning(**base)
    assert got[0] == got[1]
    assert got[0][0] == oracle.exact_count(g["row_ptr"], g["col_idx"], eu, ev)
    assert got[0][2] + got[0][3] == m


@pytest.mark.parametrize("pairs", [1, 2])
@pytest.mark.parametrize("at", [0, 1, 4, 5, -1])
def test_neighbour_ids_are_checked_without_long_lists(tchll, pairs, at):
    """A neighbour id outside the graph is refused whatever the path."""
    import torch
    from triangle_counting_hll_b200 import core
    iu, iv = np.triu_indices(6, 1)
    g = core.csr_from_edges(iu.astype(np.int32), iv.astype(np.int32))
    col = g.col_idx.clone()
    col[at] = g.n_nodes
    base = core.get_count_tuning()
    try:
        core.set_count_tuning(**dict(base, pairs=pairs))
        res, _ = core.exact_count_tensors(g.row_ptr, col, g.edge_u, g.edge_v)
        with pytest.raises(ValueError, match="neighbour id"):
            core.exact_from_result(res)
    finally:
        core.set_count_tuning(**base)
