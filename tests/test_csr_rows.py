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


# one id in every edge, first or last or all over; one pair; few pairs, often
@pytest.mark.parametrize("kind", ["star", "star of the last", "star among others", "one pair", "few pairs"])
@pytest.mark.parametrize("n_raw", [33, 5000, 300_000])
def test_popular_ids_and_repeated_edges(tchll, oracle, kind, n_raw):
    rng = np.random.default_rng(n_raw)
    at = np.arange(n_raw)
    u, v = {"star": (0 * at, at + 1), "star of the last": (at, 0 * at + n_raw + 7),
            "star among others": (np.where(at % 2, 3, rng.integers(0, n_raw, n_raw)), rng.integers(0, n_raw, n_raw)),
            "one pair": (0 * at + 4, 0 * at + 2), "few pairs": (at % 5, at % 3)}[kind]
    order = rng.permutation(n_raw)
    for o in (at, order):
        _check(oracle, u[o], v[o])
        _check(oracle, v[o] * 5000 % (2**31 - 1), u[o] * 5000 % (2**31 - 1))


# few ids in many edges, on both sides of the line, with and without unused ids
@pytest.mark.parametrize("n_raw", [(1 << 17), (1 << 17) + 1, 200_000])
@pytest.mark.parametrize("ids", [512, 513, 700, 900])
@pytest.mark.parametrize("step", [1, 7, 100_000])
def test_dense_lists(tchll, oracle, n_raw, ids, step):
    rng = np.random.default_rng(ids + n_raw)
    u, v = rng.integers(0, ids, n_raw) * step, rng.integers(0, ids, n_raw) * step
    _check(oracle, u, v)
