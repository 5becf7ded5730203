"""Which way a graph is counted: as given in one launch, or with its long-list
pairs regrouped for the hub kernels.  The graph decides, not the edges asked
for; the phases of the call tell which way it went."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(name):
    """Edges by name; the lists of each stay on one side of the lines."""
    import torch
    from triangle_counting_hll_b200 import core

    def clique(k, step=1):
        iu, iv = np.triu_indices(k, 1)
        return (torch.from_numpy((x * step).astype(np.int32)).cuda() for x in (iu, iv))

    def pendants(k, n):
        ids = torch.arange(n, dtype=torch.int32, device="cuda")
        return ids + k, ids % k

    def joined(*parts):
        return core.csr_from_edges(torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts]))

    if name == "small":                    # every list fits a warp's table
        return core.csr_from_edges(*core.gen_rmat(12, 16, seed=1))
    if name == "rmat":
        return core.csr_from_edges(*core.gen_rmat(17, 16, seed=1))
    if name == "clique with pendants":     # few edges, a mean below 128, lists of 699
        return joined(tuple(clique(700)), pendants(700, 2000))
    if name == "lattice":                  # no long list
        return core.csr_from_edges(*core.gen_lattice(400, 400, seed=1))
    return joined(core.gen_lattice(900, 900, seed=1), tuple(clique(400, step=601)))  # "dense core in a lattice"


def _phases(core, run):
    core.set_phase_timing(True)
    try:
        run()
        return core.phase_times()
    finally:
        core.set_phase_timing(False)


@pytest.mark.parametrize("name,regrouped", [("small", False), ("rmat", True), ("clique with pendants", True),
                                            ("lattice", True), ("dense core in a lattice", True)])
def test_exact_and_hybrid(tchll, oracle, name, regrouped):
    from triangle_counting_hll_b200 import core
    g = _graph(name)
    n = (lambda t: t.cpu().numpy())
    want = oracle.exact_count(n(g.row_ptr), n(g.col_idx), n(g.edge_u), n(g.edge_v), nthreads=0)
    got = []
    ph = _phases(core, lambda: got.append(core.exact_from_result(
        core.exact_count_tensors(g.row_ptr, g.col_idx, g.edge_u, g.edge_v)[0])))
    assert got == [want]
    assert (ph["pairs"] is not None, ph["hub"] is not None) == (regrouped, regrouped)
    slot, rows_n = core.sketch_slots(g.row_ptr, 1 << 30)  # no sketch: every edge exact
    rows = core.build_sketches_compact_tensors(g.row_ptr, g.col_idx, slot, rows_n, 8)
    hyb = []
    ph = _phases(core, lambda: hyb.append(core.hybrid_from_result(
        core.hybrid_count_compact_tensors(g.row_ptr, g.col_idx, g.edge_u, g.edge_v, g.degrees, rows, slot, 8, 16,
                                          split_kernels=True)[0])))
    assert hyb[0][0] == want and hyb[0][1].n_exact == g.n_edges
    assert (ph["pairs"] is not None, ph["hub"] is not None) == (regrouped, regrouped)


@pytest.mark.parametrize("part", [1, 1000, 100_000])
def test_part_of_the_edges(tchll, oracle, part):
    """A rank's shard of a graph takes the graph's way."""
    from triangle_counting_hll_b200 import core
    g = _graph("rmat")
    u, v = g.edge_u[-part:].contiguous(), g.edge_v[-part:].contiguous()
    n = (lambda t: t.cpu().numpy())
    want = oracle.exact_count(n(g.row_ptr), n(g.col_idx), n(u), n(v), nthreads=0)
    got = []
    ph = _phases(core, lambda: got.append(core.exact_from_result(
        core.exact_count_tensors(g.row_ptr, g.col_idx, u, v)[0])))
    assert got == [want] and ph["pairs"] is not None and ph["hub"] is not None


@pytest.mark.parametrize("name", ["lattice", "dense core in a lattice"])
@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("offset", [0, 1])
def test_sparse_graphs_check_every_id(tchll, name, packed, offset):
    import torch
    from triangle_counting_hll_b200 import core
    g = _graph(name)
    base = core.get_count_tuning()
    try:
        core.set_count_tuning(**dict(base, packed=packed))
        want = core.exact_from_result(core.exact_count_tensors(g.row_ptr, g.col_idx, g.edge_u, g.edge_v)[0])
        for at in (None, 0, g.n_edges // 2, -1):
            buf = torch.zeros(g.n_edges + offset, dtype=torch.int32, device="cuda")
            buf[offset:] = g.col_idx
            col = buf[offset:]
            if at is not None:
                col[at] = g.n_nodes
            res, _ = core.exact_count_tensors(g.row_ptr, col, g.edge_u, g.edge_v)
            if at is None:
                assert core.exact_from_result(res) == want
            else:
                with pytest.raises(ValueError, match="neighbour id"):
                    core.exact_from_result(res)
    finally:
        core.set_count_tuning(**base)


@pytest.mark.parametrize("name", ["small", "lattice", "dense core in a lattice"])
def test_from_host_memory(tchll, name):
    """The arrays arrive while the count runs: the ids are checked once they have."""
    from triangle_counting_hll_b200 import core
    g = _graph(name)
    want = core.exact_from_result(core.exact_count_tensors(g.row_ptr, g.col_idx, g.edge_u, g.edge_v)[0])
    host = [t.cpu().pin_memory() for t in (g.row_ptr, g.col_idx, g.edge_u, g.edge_v)]
    for _ in range(3):
        assert core.exact_from_result(core.exact_count_host(*host)) == want
