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


def _random_csr(rng, lens, n):
    row_ptr = np.zeros(n + 1, dtype=np.int32)
    row_ptr[1:] = np.cumsum(lens)
    col = np.concatenate([np.sort(rng.permutation(n)[:d]) for d in lens] or [[]]).astype(np.int32)
    return row_ptr, col


# list lengths around 16-byte quads and the short / hub line, starts at every
# alignment, an array that does or does not end in a whole quad
@pytest.mark.parametrize("pairs,offset", [(1, 0), (2, 0), (1, 1), (2, 1)])
@pytest.mark.parametrize("tail", [0, 1, 2, 3])
def test_searched_lists(tchll, oracle, pairs, offset, tail):
    import torch
    from triangle_counting_hll_b200 import core
    rng = np.random.default_rng(11 + tail)
    n = 900
    lens = rng.choice([0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33, 63, 64, 65, 127, 128, 129], n)
    lens[-1] = 6
    lens[-1] += (tail - lens.sum()) % 4
    row_ptr, col = _random_csr(rng, lens, n)
    assert len(col) % 4 == tail
    eu, ev = (rng.integers(0, n, 40001).astype(np.int32) for _ in range(2))
    eu[:7], ev[:7] = n - 1, rng.integers(0, n, 7)
    ref = oracle.exact_count(row_ptr, col, eu, ev)
    buf = torch.zeros(len(col) + offset, dtype=torch.int32, device="cuda")  # offset: not 16-byte aligned
    buf[offset:] = torch.from_numpy(col).cuda()
    base = core.get_count_tuning()
    try:
        core.set_count_tuning(**dict(base, pairs=pairs))
        res, _ = core.exact_count_tensors(torch.from_numpy(row_ptr).cuda(), buf[offset:], torch.from_numpy(eu).cuda(),
                                          torch.from_numpy(ev).cuda())
        assert core.exact_from_result(res) == ref
    finally:
        core.set_count_tuning(**base)


def test_batch_mixes_graphs_with_and_without_long_lists(tchll, oracle):
    """Only the graphs with hub pairs get lists and their own core numbering;
    counts and totals equal one graph at a time."""
    import torch
    from triangle_counting_hll_b200 import batch, core
    graphs = []
    for i in range(60):
        if i % 5 == 2:  # a clique inside an R-MAT graph: lists past the hub line
            u, v = core.gen_rmat(10, 8, seed=i)
            iu, iv = np.triu_indices(150 + i, 1)
            u = torch.cat([u, torch.from_numpy(iu.astype(np.int32)).cuda()])
            v = torch.cat([v, torch.from_numpy(iv.astype(np.int32)).cuda()])
            graphs.append((u, v, 1 << 10))
        else:
            graphs.append((*core.gen_er(37 + 11 * i, 200 + 30 * i, seed=i), 37 + 11 * i))
    b = batch.GraphBatch.from_edge_lists(graphs)
    csrs = [core.csr_from_edges(u, v) for u, v, _ in graphs]
    assert np.array_equal(b.exact_counts(), batch.plain_exact_counts(csrs))
    totals, stats = b.hybrid_counts(64, 64, 10)
    want, wstats = batch.plain_hybrid_counts(csrs, batch.plain_sketches(csrs, 64, 10), 64, 10)
    assert np.array_equal(totals, want)
    assert all(np.array_equal(stats[k], wstats[k]) for k in stats)


@pytest.mark.parametrize("length", [1 << 25, (1 << 25) + 1])
def test_lists_longer_than_a_warp_adds_up(tchll, length):
    """Vertex 0 is joined to all others, vertex 1 to all after it: the pair
    (0, 1) closes one triangle for every member of the shorter list."""
    import torch
    from triangle_counting_hll_b200 import core
    n = length + 2
    row_ptr = torch.full((n + 1,), 2 * length + 1, dtype=torch.int32, device="cuda")
    row_ptr[0] = 0
    row_ptr[1] = length + 1
    col = torch.cat([torch.arange(1, n, dtype=torch.int32, device="cuda"),
                     torch.arange(2, n, dtype=torch.int32, device="cuda")])
    u = torch.tensor([0, 0, 0], dtype=torch.int32, device="cuda")
    v = torch.tensor([1, 2, 1], dtype=torch.int32, device="cuda")
    res, _ = core.exact_count_tensors(row_ptr, col, u, v)
    assert core.exact_from_result(res) == 2 * length
