"""The hub kernels' packed lists (bitmap prefix + 16-bit keys) at the sizes
where their layout changes, against the CPU oracle on hand-built CSRs."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(rng, n, lens, skew):
    """n rows, the first len(lens) with sorted distinct members of [0, n); a
    higher skew concentrates the members on few vertices."""
    rows = []
    for d in lens:
        got = np.zeros(0, dtype=np.int64)
        while len(got) < d:
            got = np.unique(np.concatenate([got, (n * rng.random(2 * d + 8) ** skew).astype(np.int64)]))
        rows.append(np.sort(rng.permutation(got)[:d]))
    perm = rng.permutation(n)  # popular members anywhere in the id space
    rows = [np.sort(perm[r]) for r in rows]
    row_ptr = np.zeros(n + 1, dtype=np.int32)
    row_ptr[1:len(rows) + 1] = np.cumsum([len(r) for r in rows])
    row_ptr[len(rows) + 1:] = row_ptr[len(rows)]
    return row_ptr, np.concatenate(rows).astype(np.int32)


def _gpu(row_ptr, col, eu, ev, **tuning):
    """The count with the edges regrouped, which small graphs do not choose
    by themselves (pairs=2)."""
    import torch
    from triangle_counting_hll_b200 import core
    from triangle_counting_hll_b200.gpu_hybrid import gpu_exact_triangle_count
    base = core.get_count_tuning()
    try:
        core.set_count_tuning(**dict(base, pairs=2, **tuning))
        return gpu_exact_triangle_count(*(torch.from_numpy(a).cuda() for a in (row_ptr, col, eu, ev)))[0]
    finally:
        core.set_count_tuning(**base)


# core sizes: one bitmap word, one plane, two planes, beyond the packed lists
@pytest.mark.parametrize("n,hubs,skew", [(700, 60, 1.0), (5000, 120, 3.0), (70000, 150, 6.0), (110000, 320, 1.0),
                                         (170000, 420, 1.0)])
def test_list_forms(tchll, oracle, n, hubs, skew):
    rng = np.random.default_rng(n)
    edge = [0, 1, 7, 8, 9, 31, 32, 33, 63, 127, 128, 129, 130, 255, 257]
    long = [x for x in (1000, 1023, 1024, 1025, 1200) if x < n]
    lens = edge * 3 + [int(x) for x in rng.integers(129, min(n // 2, 900), hubs)] + long
    row_ptr, col = _csr(rng, n, lens, skew)
    eu, ev = (rng.integers(0, len(lens), 60000).astype(np.int32) for _ in range(2))
    ref = oracle.exact_count(row_ptr, col, eu, ev)
    for tuning in ({}, {"packed": False}, {"packed": False, "bitmap_lg": 0}, {"overlap": 0}, {"overlap": 2}):
        assert _gpu(row_ptr, col, eu, ev, **tuning) == ref, tuning


def test_repeated_members_stay_keys(tchll):
    """A probe list that repeats a member counts it once per mention, as
    the key lists do; a bitmap would count it once."""
    rng = np.random.default_rng(5)
    n = 4000
    x = np.sort(rng.permutation(n)[:600])
    y = np.sort(np.concatenate([x[:100], x[:40], rng.permutation(n)[:60]]))
    row_ptr = np.zeros(n + 1, dtype=np.int32)
    row_ptr[1], row_ptr[2:] = len(x), len(x) + len(y)
    col = np.concatenate([x, y]).astype(np.int32)
    eu, ev = np.zeros(300, dtype=np.int32), np.ones(300, dtype=np.int32)
    assert _gpu(row_ptr, col, eu, ev) == 300 * int(np.isin(y, x).sum())
