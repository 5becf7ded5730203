"""Pairs of lists of middling length are grouped by table side and counted
with a warp's hash table: at the lengths where they start and end, with more
pairs of one side than a segment holds, in batches and without hub kernels."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(rng, n, lens):
    row_ptr = np.zeros(n + 1, dtype=np.int32)
    row_ptr[1:len(lens) + 1] = np.cumsum(lens)
    row_ptr[len(lens) + 1:] = row_ptr[len(lens)]
    return row_ptr, np.concatenate([np.sort(rng.permutation(n)[:d]) for d in lens]).astype(np.int32)


@pytest.mark.parametrize("hub", [0, 64, 128, 300])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("per_side", [1, 255, 256, 257, 700])
def test_lengths_and_segments(tchll, oracle, hub, offset, per_side):
    """Each of 30 table sides with per_side probe sides of every length."""
    import torch
    from triangle_counting_hll_b200 import core
    rng = np.random.default_rng(per_side + offset)
    n = 600
    tables = [31, 32, 33, 34, 63, 64, 65, 127, 128, 129, 299, 300, 301, 512, 513] * 2
    probes = [0, 1, 15, 16, 17, 18, 31, 32, 33, 40]
    row_ptr, col = _csr(rng, n, tables + probes * 5)
    eu = np.repeat(np.arange(len(tables)), per_side).astype(np.int32)
    ev = (len(tables) + rng.integers(0, 5 * len(probes), len(eu))).astype(np.int32)
    flip = rng.random(len(eu)) < 0.5  # either end may be the table side
    eu, ev = np.where(flip, ev, eu).astype(np.int32), np.where(flip, eu, ev).astype(np.int32)
    order = rng.permutation(len(eu))
    eu, ev = eu[order].copy(), ev[order].copy()
    buf = torch.zeros(len(col) + offset, dtype=torch.int32, device="cuda")
    buf[offset:] = torch.from_numpy(col).cuda()
    rp, u, v = (torch.from_numpy(a).cuda() for a in (row_ptr, eu, ev))
    base = core.get_count_tuning()
    try:
        core.set_count_tuning(**dict(base, pairs=2, hub=hub))
        res, _ = core.exact_count_tensors(rp, buf[offset:], u, v)
        assert core.exact_from_result(res) == oracle.exact_count(row_ptr, col, eu, ev)
        from triangle_counting_hll_b200 import _lib
        assert _lib.read_count_result(res).n_exact == len(eu)
    finally:
        core.set_count_tuning(**base)


def test_even_graphs_alone_and_in_a_batch(tchll):
    """Graphs whose lists are all about 50 long, beside short-listed ones."""
    import torch
    from triangle_counting_hll_b200 import batch, core
    graphs = []
    for i in range(12):
        n, m = (1500, 75000) if i % 3 else (2000, 4000)
        graphs.append((*core.gen_er(n, m, seed=i), n))
    b = batch.GraphBatch.from_edge_lists(graphs)
    csrs = [core.csr_from_edges(u, v) for u, v, _ in graphs]
    base = core.get_count_tuning()
    try:
        got = {}
        for hub in (0, 64, 128):
            core.set_count_tuning(**dict(base, hub=hub))
            got[hub] = b.exact_counts()
            totals, stats = b.hybrid_counts(40, 40, 10)
            want, wstats = batch.plain_hybrid_counts(csrs, batch.plain_sketches(csrs, 40, 10), 40, 10)
            assert np.array_equal(totals, want)
            assert all(np.array_equal(stats[k], wstats[k]) for k in stats)
        for pairs in (1, 2, 0):
            core.set_count_tuning(**dict(base, pairs=pairs))
            assert all(np.array_equal(got[h], batch.plain_exact_counts(csrs)) for h in got)
    finally:
        core.set_count_tuning(**base)


@pytest.mark.parametrize("shuffled", [False, True])
def test_given_edges_in_any_order(tchll, oracle, shuffled):
    import torch
    from triangle_counting_hll_b200 import core
    u, v = oracle.gen_er(20000, 1000000, 5) if hasattr(oracle, "gen_er") else (None, None)
    if u is None:
        du, dv = core.gen_er(20000, 1000000, seed=5)
        u, v = du.cpu().numpy(), dv.cpu().numpy()
    g = oracle.csr_build(u, v)
    eu, ev = g["edge_u"], g["edge_v"]
    if shuffled:
        order = np.random.default_rng(1).permutation(len(eu))
        eu, ev = eu[order].copy(), ev[order].copy()
    rp, ci, du, dv = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g["row_ptr"], g["col_idx"], eu, ev))
    res, _ = core.exact_count_tensors(rp, ci, du, dv)
    assert core.exact_from_result(res) == oracle.exact_count(g["row_ptr"], g["col_idx"], eu, ev, nthreads=0)
