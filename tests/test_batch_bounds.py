"""Batches whose graph table or row pointers are malformed at a graph's bounds
are refused, never followed: the graph and those behind it report a bad row,
the graphs before it keep their counts."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAD_ROW = 2


def _counts(L, core, g, row_ptr, vbase, hybrid):
    """Status and exact part of every graph of the table."""
    import torch
    from triangle_counting_hll_b200 import _lib, batch
    n = vbase.numel() - 1
    nb = C.c_size_t(0)
    assert L.tchll_batch_workspace_bytes(g.n_nodes, g.n_edges, n, C.byref(nb)) == 0
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    res = torch.full((n * _lib.RESULT_BYTES,), 0xAB, dtype=torch.uint8, device="cuda")
    st = _lib.stream_handle(g.device)
    csr = (row_ptr.data_ptr(), g.n_nodes, g.col_idx.data_ptr(), g.n_edges, g.edge_u.data_ptr(), g.edge_v.data_ptr(),
           g.n_edges)
    if hybrid:
        slot = torch.full((g.n_nodes,), -1, dtype=torch.int64, device="cuda")
        rc = L.tchll_batch_hybrid_count(*csr, g.degrees.data_ptr(), None, 0, slot.data_ptr(), 10, 16,
                                        vbase.data_ptr(), n, res.data_ptr(), ws.data_ptr(), nb.value, st)
    else:
        rc = L.tchll_batch_exact_count(*csr, vbase.data_ptr(), n, res.data_ptr(), ws.data_ptr(), nb.value, st)
    assert rc == 0, _lib.last_error()
    r = batch._results(res, n)
    return r["status"].tolist(), r["exact"].tolist()


@pytest.mark.parametrize("hybrid", [False, True])
def test_bounds(tchll, oracle, hybrid):
    import torch
    from triangle_counting_hll_b200 import _lib, batch, core
    L = _lib.load()
    iu, iv = (torch.from_numpy(x.astype(np.int32)).cuda() for x in np.triu_indices(90, 1))
    b = batch.GraphBatch.from_edge_lists([(iu, iv, 90)] * 6)
    g, n, vb = b.csr, b.n_graphs, b.vbase
    want = 90 * 89 * 88 // 6
    big = 2**31 - 1

    def changed(t, at, value):
        t = t.clone()
        t[at] = value
        return t

    bound = int(vb[3])  # row pointer between graphs 2 and 3
    for value in (big, g.n_edges + 1, -1, -big, 0):
        # (the check of all rows reports to the first graph's block)
        status, exact = _counts(L, core, g, changed(g.row_ptr, bound, value), vb, hybrid)
        assert exact[:2] == [want, want] and exact[2:] == [0, 0, 0, 0], value
        assert all(s & BAD_ROW for s in status[2:]) and status[1] == 0, value
    for value in (big, -1, g.n_nodes + 1, 0):  # the table itself
        status, exact = _counts(L, core, g, g.row_ptr, changed(vb, 3, value), hybrid)
        assert status[:2] == [0, 0] and exact[:2] == [want, want]
        assert all(s & BAD_ROW for s in status[2:]), value
    # a table that runs over the whole graph again and again
    again = torch.tensor([0, g.n_nodes] * 500, dtype=torch.int32, device="cuda")
    status, exact = _counts(L, core, g, g.row_ptr, again, hybrid)
    assert status[0] == 0 and exact[0] == 6 * want and all(s & BAD_ROW for s in status[1:])
    status, exact = _counts(L, core, g, g.row_ptr, vb, hybrid)
    assert status == [0] * n and exact == [want] * n
