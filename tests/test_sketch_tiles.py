"""Sketch build at the edges of its tiles (groups of 8 of 256 vertices) and
of its two forms (a warp per vertex up to p = 12, a CTA above), and the byte
clearing under it, against the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 9, 255, 256, 257, 2049])
@pytest.mark.parametrize("p", [4, 12, 13])
def test_tiles(tchll, oracle, n, p):
    import torch
    from triangle_counting_hll_b200 import core
    rng = np.random.default_rng(n * 17 + p)
    lens = rng.choice([0, 1, 15, 16, 17, 127, 129, 700], n)
    row_ptr = np.zeros(n + 1, dtype=np.int32)
    row_ptr[1:] = np.cumsum(lens)
    col = np.concatenate([np.sort(rng.permutation(5000)[:d]) for d in lens] or [[]]).astype(np.int32)
    slot, rows = oracle.build_sketches_compact(row_ptr.astype(np.int64), col.astype(np.int64), 16, p)
    rp, ci = torch.from_numpy(row_ptr).cuda(), torch.from_numpy(col).cuda()
    regs, has = tchll.alloc_sketch_arrays_device(n, p)
    assert not regs.any() and not has.any()
    tchll.build_sketches_kernel[(n + 255) // 256, 256](rp, ci, n, 16, p, regs, has)
    assert np.array_equal(has.cpu().numpy() == 1, slot >= 0)
    dense = np.zeros((n, 1 << p), dtype=np.uint8)
    dense[slot >= 0] = np.asarray(rows, dtype=np.uint8).reshape(-1, 1 << p)[: int((slot >= 0).sum())]
    assert np.array_equal(regs.cpu().numpy().reshape(n, -1), dense)
    gslot, n_rows = core.sketch_slots(rp, 16)
    got = core.build_sketches_compact_tensors(rp, ci, gslot, n_rows, p)
    assert np.array_equal(got.cpu().numpy(), dense[slot >= 0].reshape(-1))


@pytest.mark.parametrize("at,n", [(0, 0), (1, 5), (3, 13), (15, 1), (16, 16), (5, 4099), (0, (4 << 20) + 3)])
def test_clearing(tchll, at, n):
    import torch
    from triangle_counting_hll_b200 import _lib
    t = torch.full((n + at + 40,), 7, dtype=torch.uint8, device="cuda")
    part = t[at:at + n]
    _lib.check(_lib.load().tchll_zero_bytes(_lib.ptr(part), n, _lib.stream_handle()))
    want = torch.full_like(t, 7)
    want[at:at + n] = 0
    assert torch.equal(t, want)
