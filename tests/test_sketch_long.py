"""Sketches of long lists, which a whole CTA hashes, beside short ones, against
the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [4, 10, 12, 13])
def test_around_the_line(tchll, oracle, p):
    import torch
    from triangle_counting_hll_b200 import core
    rng = np.random.default_rng(p)
    lens = np.concatenate([rng.choice([0, 5, 200, 4096, 16383, 16384, 16385, 40000], 60), np.zeros(700, dtype=np.int64)])
    lens = lens[rng.permutation(len(lens))]
    n = len(lens)
    row_ptr = np.zeros(n + 1, dtype=np.int32)
    row_ptr[1:] = np.cumsum(lens)
    col = np.concatenate([np.sort(rng.permutation(50000)[:d]) for d in lens]).astype(np.int32)
    slot, rows = oracle.build_sketches_compact(row_ptr.astype(np.int64), col.astype(np.int64), 16, p)
    rp, ci = torch.from_numpy(row_ptr).cuda(), torch.from_numpy(col).cuda()
    gslot, n_rows = core.sketch_slots(rp, 16)
    got = core.build_sketches_compact_tensors(rp, ci, gslot, n_rows, p)
    assert np.array_equal(got.cpu().numpy(), np.asarray(rows, dtype=np.uint8).reshape(-1)[: n_rows << p])
    regs, has = tchll.alloc_sketch_arrays_device(n, p)
    tchll.build_sketches_kernel[(n + 255) // 256, 256](rp, ci, n, 16, p, regs, has)
    assert np.array_equal(regs.cpu().numpy().reshape(n, -1)[slot >= 0].reshape(-1), got.cpu().numpy())
