"""Graphs without a long list whose neighbour array starts on any word: every
id is checked whatever the start, and the count is the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(tail):
    """Lists of at most 40 members, at least as many edges as members (the
    workspace then holds the lists); the neighbour array's length is tail modulo 4."""
    rng = np.random.default_rng(23 + tail)
    n = 700
    lens = rng.integers(0, 41, n)
    lens[-1] = 5
    lens[-1] += (tail - lens.sum()) % 4
    row_ptr = np.zeros(n + 1, dtype=np.int32)
    row_ptr[1:] = np.cumsum(lens)
    col = np.concatenate([np.sort(rng.permutation(n)[:d]) for d in lens]).astype(np.int32)
    eu, ev = (rng.integers(0, n, 20001).astype(np.int32) for _ in range(2))
    return n, row_ptr, col, eu, ev


def _shifted(col, offset):
    import torch
    buf = torch.zeros(len(col) + offset, dtype=torch.int32, device="cuda")
    buf[offset:] = torch.from_numpy(col).cuda()
    return buf[offset:]


# the regrouped path (pairs=2), with packed lists and with 32-bit ones
@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("tail", [0, 3])
def test_counts_and_checked_ids(tchll, oracle, packed, offset, tail):
    import torch
    from triangle_counting_hll_b200 import core
    n, row_ptr, col, eu, ev = _graph(tail)
    rp, u, v = (torch.from_numpy(a).cuda() for a in (row_ptr, eu, ev))
    base = core.get_count_tuning()
    try:
        core.set_count_tuning(**dict(base, pairs=2, packed=packed))
        res, _ = core.exact_count_tensors(rp, _shifted(col, offset), u, v)
        assert core.exact_from_result(res) == oracle.exact_count(row_ptr, col, eu, ev)
        for at in (0, 1, 2, 3, 4, len(col) // 2, -5, -4, -3, -2, -1):
            wrong = col.copy()
            wrong[at] = n
            res, _ = core.exact_count_tensors(rp, _shifted(wrong, offset), u, v)
            with pytest.raises(ValueError, match="neighbour id"):
                core.exact_from_result(res)
    finally:
        core.set_count_tuning(**base)
