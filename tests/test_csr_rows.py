"""The small CSR build where it has many short rows, popular ids and repeated
edges, against the CPU oracle (all arrays equal)."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_csr_small import _check

pytestmark = pytest.mark.gpu


# below and above the row count from which a warp takes 32 rows at a time
@pytest.mark.parametrize("n", [132_000, 133_500, 400_000])
@pytest.mark.parametrize("spread", [1, 3001])
def test_many_short_rows_and_some_long(tchll, oracle, n, spread):
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, n), rng.integers(0, n, n)
    parts_u, parts_v = [u, np.arange(n - 1)], [v, np.arange(1, n)]  # every id occurs
    for k, at in ((6, 50), (40, 1000), (80, 7777), (300, 90_000)):  # rows of every sorted form
        iu, iv = np.triu_indices(k, 1)
        parts_u.append(iu * 3 + at)
        parts_v.append(iv * 3 + at)
    u, v = np.concatenate(parts_u) * spread, np.concatenate(parts_v) * spread
    order = rng.permutation(len(u))
    assert len(u) < 1 << 21
    _check(oracle, u[order], v[order])
