"""Batches with graphs around and above the size from which many CTAs number a
graph's core, at odd places between small ones."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _path_and_core(n, k, seed):
    """Exactly n vertices: a path, and k of them joined by a dense random graph."""
    import torch
    rng = np.random.default_rng(seed)
    at = np.sort(rng.permutation(n)[:k]).astype(np.int32)
    iu, iv = np.triu_indices(k, 1)
    keep = rng.random(len(iu)) < 0.8
    u = np.concatenate([np.arange(n - 1), at[iu[keep]]]).astype(np.int32)
    v = np.concatenate([np.arange(1, n), at[iv[keep]]]).astype(np.int32)
    return torch.from_numpy(u).cuda(), torch.from_numpy(v).cuda(), n


@pytest.mark.parametrize("sizes", [(32767, 32768, 32769), (5, 40000, 3, 4096, 8192, 70001, 2), (33000, 33000, 33000),
                                   (100, 61440, 100)])
def test_sizes(tchll, sizes):
    from triangle_counting_hll_b200 import batch, core
    graphs = [_path_and_core(n, min(n, 400) if n > 100 else 2, i) for i, n in enumerate(sizes)]
    graphs.append((*core.gen_rmat(10, 8, seed=3), 1 << 10))
    b = batch.GraphBatch.from_edge_lists(graphs)
    assert np.diff(b.vbase.cpu().numpy())[:len(sizes)].tolist() == list(sizes)
    csrs = [core.csr_from_edges(u, v) for u, v, _ in graphs]
    want = batch.plain_exact_counts(csrs)
    base = core.get_count_tuning()
    try:
        for tuning in ({}, {"hub": 64}, {"hub": 128, "packed": False}):
            core.set_count_tuning(**dict(base, **tuning))
            assert np.array_equal(b.exact_counts(), want), tuning
            totals, stats = b.hybrid_counts(120, 120, 8)
            plain, pstats = batch.plain_hybrid_counts(csrs, batch.plain_sketches(csrs, 120, 8), 120, 8)
            assert np.array_equal(totals, plain), tuning
            assert all(np.array_equal(stats[k], pstats[k]) for k in stats)
    finally:
        core.set_count_tuning(**base)


def test_skewed_graphs(tchll):
    from triangle_counting_hll_b200 import batch, core
    graphs = []
    for i, scale in enumerate((10, 16, 11, 17, 16, 12)):
        graphs.append((*core.gen_rmat(scale, 16, seed=i), 1 << scale))
    b = batch.GraphBatch.from_edge_lists(graphs)
    csrs = [core.csr_from_edges(u, v) for u, v, _ in graphs]
    assert np.array_equal(b.exact_counts(), batch.plain_exact_counts(csrs))


@pytest.mark.parametrize("shift", [0, 1, 8])
def test_register_rows_at_any_byte(tchll, shift):
    """Register rows that do not start on 16 bytes: the same result blocks, and
    the pairs of long lists still go by the hub kernels."""
    import torch
    from triangle_counting_hll_b200 import _lib, batch, core
    graphs = [(*core.gen_rmat(s, 16, seed=s), 1 << s) for s in (9, 13, 14)]
    b = batch.GraphBatch.from_edge_lists(graphs)
    rows, slot = b.sketches(100, 8)
    buf = torch.empty(rows.numel() + shift, dtype=torch.uint8, device="cuda")
    buf[shift:] = rows
    blocks = []
    core.set_phase_timing(True)
    try:
        for r in (rows, buf[shift:]):
            res = torch.zeros(3 * _lib.RESULT_BYTES, dtype=torch.uint8, device="cuda")
            b.hybrid_launch(res, r, slot, 8, 100)
            assert core.phase_times()["hub"] is not None
            blocks.append(res.cpu())
    finally:
        core.set_phase_timing(False)
    assert torch.equal(blocks[0], blocks[1])
    assert batch.hybrid_from_results(blocks[0], 3)[1]["n_approx"].sum() > 0
