"""Reading a result block back belongs to the device that the block is on,
whatever device is current (library, devices and streams faked: no GPU)."""
from __future__ import annotations

import contextlib
import ctypes as C
import types

import pytest
import torch

from triangle_counting_hll_b200 import _lib, core


class FakeCuda:
    """Two devices with one default stream each, and the calls in order."""

    def __init__(self, monkeypatch, current):
        self.current, self.log = current, []
        monkeypatch.setattr(torch.cuda, "current_device", lambda: self.current)
        monkeypatch.setattr(torch.cuda, "device", self.device)
        monkeypatch.setattr(_lib, "_raw_stream", lambda idx: 0)
        monkeypatch.setattr(_lib, "load", lambda: self)

    @contextlib.contextmanager
    def device(self, dev):
        before, self.current = self.current, torch.device(dev).index
        self.log.append(("current", self.current))
        try:
            yield
        finally:
            self.current = before
            self.log.append(("current", before))

    def tchll_fetch(self, dst, src, n, stream):
        self.log.append(("fetch", self.current, src, n, stream))
        return 0


def _block(index):
    return types.SimpleNamespace(device=torch.device("cuda", index), data_ptr=lambda: 4096)


@pytest.mark.parametrize("read", [_lib.read_count_result, core.exact_from_result, core.hybrid_from_result])
def test_other_device(monkeypatch, read):
    cuda = FakeCuda(monkeypatch, current=0)
    read(_block(1))
    assert cuda.log == [("current", 1), ("fetch", 1, 4096, _lib.RESULT_BYTES, 0), ("current", 0)]


def test_current_device_is_left_alone(monkeypatch):
    cuda = FakeCuda(monkeypatch, current=1)
    got = C.c_int64(0)
    _lib.fetch(got, _block(1), 8)
    assert cuda.log == [("fetch", 1, 4096, 8, 0)]


def test_block_on_the_host(monkeypatch):
    monkeypatch.setattr(_lib, "load", lambda: pytest.fail("no library call for a block on the host"))
    r = _lib.CountResult()
    r.exact, r.n_exact = 12345678901, 77
    t = torch.frombuffer(bytearray(bytes(r)), dtype=torch.uint8)
    assert core.exact_from_result(t) == 12345678901
    assert _lib.read_count_result(t).n_exact == 77


def test_device_is_put_back_after_an_error(monkeypatch):
    cuda = FakeCuda(monkeypatch, current=0)
    monkeypatch.setattr(cuda, "tchll_fetch", lambda *a: 999, raising=False)
    monkeypatch.setattr(_lib, "last_error", lambda: "failed")
    with pytest.raises(_lib.TchllError):
        _lib.read_count_result(_block(1))
    assert cuda.current == 0


@pytest.mark.parametrize("device,index", [(None, 0), (1, 1), (torch.device("cuda"), 0), (torch.device("cuda", 1), 1),
                                          ("cuda:1", 1), ("cuda", 0)])
def test_stream_of_a_device_however_named(monkeypatch, device, index):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(_lib, "_raw_stream", lambda idx: 1000 + idx)
    assert _lib.stream_handle(device) == 1000 + index
