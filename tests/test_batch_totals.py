"""Batched hybrid totals from result blocks: rounded once, like Python's
integers, below and above 64 bits (host arithmetic only)."""
from __future__ import annotations

import numpy as np
import torch

from triangle_counting_hll_b200 import batch


def test_totals_round_once():
    rng = np.random.default_rng(0)
    top = np.iinfo(np.uint64).max
    cases = [(0, 0, 0), (0, 1, 0), (2**31 - 1, 2**63 - 1, 0), (2**31 - 1, 2**63, 0), (2**31, 0, 0), (2**40, top, 0),
             (5, top, 3), (2**31 - 1, 2**53 + 1, 0), (0, 2**62 + 2**8 + 1, 0), (1, 2**60 - 1, 2**20)]
    cases += [(int(rng.integers(0, 1 << 36)), int(rng.integers(0, top, dtype=np.uint64)), int(rng.integers(0, 3)))
              for _ in range(400)]
    raw = np.zeros((len(cases), 8), dtype=np.uint64)
    for i, c in enumerate(cases):
        raw[i, :3] = c
    totals, _ = batch.hybrid_from_results(torch.from_numpy(raw.view(np.uint8).reshape(-1)), len(cases))
    want = [((e << 32) + ((h << 64) | lo)) / 4294967296 for e, lo, h in cases]
    assert totals.tolist() == want
