"""The small CSR build (hash table, row sort) against the CPU oracle: id spaces
dense and sparse, duplicates, self-loops, both row-sort forms and the largest
size, and one raw edge past it (the sort pipeline)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(oracle, u, v):
    import torch
    from triangle_counting_hll_b200 import core
    u, v = np.ascontiguousarray(u, dtype=np.int32), np.ascontiguousarray(v, dtype=np.int32)
    og = oracle.csr_build(u, v)
    g, und = core.csr_from_edges(torch.from_numpy(u).cuda(), torch.from_numpy(v).cuda(), undirected=True)
    assert (g.n_nodes, g.n_edges) == (og["n_nodes"], og["n_edges"])
    for name in ("row_ptr", "col_idx", "degrees", "edge_u", "edge_v"):
        assert np.array_equal(getattr(g, name).cpu().numpy(), og[name]), name
    assert np.array_equal(g.node_ids.cpu().numpy().astype(np.int64), og["node_ids"])
    want = og["degrees"].astype(np.int64) + np.bincount(og["col_idx"], minlength=og["n_nodes"])
    assert np.array_equal(und.cpu().numpy(), want)


@pytest.mark.parametrize("n_raw", [1, 2, 3, 511, 1025, 30000])
@pytest.mark.parametrize("spread", [1, 1000])
def test_dense_and_sparse_ids(tchll, oracle, n_raw, spread):
    rng = np.random.default_rng(n_raw + spread)
    ids = rng.integers(0, max(2, n_raw // 3), (2, n_raw)) * spread + (spread > 1) * 5
    if n_raw > 2:
        ids[1, 0] = ids[0, 0]              # a self-loop
        ids[:, 1] = ids[::-1, 2]           # a pair twice, reversed
        if spread > 1:
            ids[0, 2] = ids[1, 1] = 2**31 - 1  # the largest id
    _check(oracle, ids[0], ids[1])


def test_only_self_loops(tchll):
    import torch
    from triangle_counting_hll_b200 import core
    u = torch.arange(7, dtype=torch.int32, device="cuda")
    g = core.csr_from_edges(u, u)
    assert (g.n_nodes, g.n_edges) == (0, 0) and g.row_ptr.cpu().tolist() == [0]


@pytest.mark.parametrize("n", [64, 65, 66, 129, 300, 2047])
def test_row_lengths(tchll, oracle, n):
    """A clique: forward lists of every length up to n - 1."""
    iu, iv = np.triu_indices(n, 1)
    order = np.random.default_rng(n).permutation(len(iu))
    _check(oracle, iv[order], iu[order])


@pytest.mark.parametrize("extra", [0, 1])
def test_largest_size(tchll, oracle, extra):
    u, v = oracle.gen_rmat(17, 16, 0.57, 0.19, 0.19, 9)
    assert len(u) == 1 << 21
    _check(oracle, np.concatenate([u, u[:extra]]), np.concatenate([v, v[:extra]]))
