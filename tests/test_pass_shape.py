"""The first pass's launch shape: any number of blocks per SM, for aligned and
unaligned neighbour arrays in either order, gives the same counts."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [0, 1])
def test_blocks_per_sm(tchll, first):
    import torch
    from triangle_counting_hll_b200 import batch, core
    g = core.csr_from_edges(*core.gen_rmat(16, 16, seed=4))
    buf = torch.zeros(g.n_edges + 1, dtype=torch.int32, device="cuda")
    buf[1:] = g.col_idx
    cols = [g.col_idx, buf[1:]]
    graphs = [(*core.gen_er(2000, 9000, seed=i), 2000) for i in range(40)]
    b = batch.GraphBatch.from_edge_lists(graphs)
    base = core.get_count_tuning()
    got, batches = set(), set()
    try:
        for blocks in (0, 1, 3, 32, 0):
            core.set_count_tuning(**dict(base, blocks_per_sm=blocks))
            for col in (cols[first], cols[1 - first]):
                got.add(core.exact_from_result(core.exact_count_tensors(g.row_ptr, col, g.edge_u, g.edge_v)[0]))
            batches.add(tuple(b.exact_counts().tolist()))
    finally:
        core.set_count_tuning(**base)
    assert len(got) == 1 and len(batches) == 1
