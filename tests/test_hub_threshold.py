"""The hub threshold in effect: what was asked for, or by the graph."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _near(n, d):
    """Every vertex joined to d of its next 4 d ones: lists evenly about d long."""
    import torch
    from triangle_counting_hll_b200 import core
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    u = torch.arange(n, device="cuda").repeat_interleave(d)
    v = (u + torch.randint(1, 4 * d, (n * d,), generator=gen, device="cuda")) % n
    return core.csr_from_edges(u.to(torch.int32), v.to(torch.int32))


def _rmat(scale, ef):
    from triangle_counting_hll_b200 import core
    return core.csr_from_edges(*core.gen_rmat(scale, ef, seed=1))


# few vertices; few edges; skewed; evenly long lists; more edges than the automatic 64 is for
@pytest.mark.parametrize("graph,want", [(lambda: _near(100_000, 60), 64), (lambda: _rmat(19, 8), 64),
                                        (lambda: _rmat(20, 16), 64), (lambda: _near(200_000, 60), 128),
                                        (lambda: _rmat(21, 16), 128)])
def test_automatic(tchll, graph, want):
    from triangle_counting_hll_b200 import core
    g = graph()
    args = (g.row_ptr, g.col_idx, g.edge_u, g.edge_v)
    base = core.get_count_tuning()
    assert base["hub"] == -1
    assert core.hub_threshold(*args) == want
    part = (g.edge_u[:100_000].contiguous(), g.edge_v[:100_000].contiguous())
    assert core.hub_threshold(g.row_ptr, g.col_idx, *part) == 128  # its workspace holds no lists
    counts = {core.exact_from_result(core.exact_count_tensors(*args)[0])}
    try:
        for hub in (0, 64, 128, 200):
            core.set_count_tuning(**dict(base, hub=hub))
            assert core.get_count_tuning()["hub"] == hub
            assert core.hub_threshold(*args) == hub
            counts.add(core.exact_from_result(core.exact_count_tensors(*args)[0]))
    finally:
        core.set_count_tuning(**base)
    assert core.get_count_tuning()["hub"] == -1
    assert len(counts) == 1
    with pytest.raises(ValueError):
        core.set_count_tuning(hub=-2)


def test_batches_of_large_and_small_graphs(tchll):
    """A batch takes 64 only where every graph's core surely fits; the counts
    are those of one graph at a time."""
    import torch
    from triangle_counting_hll_b200 import batch, core
    lists = [(*core.gen_rmat(12, 32, seed=i), 1 << 12) for i in range(8)]
    lists.append((*core.gen_er(140_000, 4_200_000, seed=3), 140_000))
    for graphs in (lists[:8], lists, lists[8:]):
        b = batch.GraphBatch.from_edge_lists(graphs)
        csrs = [core.csr_from_edges(u, v) for u, v, _ in graphs]
        want = batch.plain_exact_counts(csrs)
        assert np.array_equal(b.exact_counts(), want)
        totals, stats = b.hybrid_counts(64, 64, 8)
        plain, pstats = batch.plain_hybrid_counts(csrs, batch.plain_sketches(csrs, 64, 8), 64, 8)
        assert np.array_equal(totals, plain)
        assert all(np.array_equal(stats[k], pstats[k]) for k in stats)
        del b, csrs
        torch.cuda.empty_cache()
