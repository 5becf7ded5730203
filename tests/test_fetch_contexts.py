"""tchll_fetch where contexts come and go, and from several threads at once:
its pinned pages belong to the context that they were made in.  In a child
process without torch, through the driver's own calls."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, sys, threading
cu, lib = C.CDLL("libcuda.so.1"), C.CDLL(sys.argv[1])
lib.tchll_fetch.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_void_p]

def ok(rc):
    assert rc == 0, rc

ok(cu.cuInit(0))
dev = C.c_int()
ok(cu.cuDeviceGet(C.byref(dev), 0))

def context():
    ctx = C.c_void_p()
    ok(cu.cuCtxCreate_v2(C.byref(ctx), 0, dev))
    return ctx

def fetch(byte, n):
    p = C.c_void_p()
    ok(cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(n)))
    ok(cu.cuMemsetD8_v2(p, C.c_ubyte(byte), C.c_size_t(n)))
    out = (C.c_ubyte * n)()
    ok(lib.tchll_fetch(out, p, n, None))
    assert bytes(out) == bytes([byte]) * n
    ok(cu.cuMemFree_v2(p))

byte = 1
for _ in range(6):  # one after the other
    ctx = context()
    for n in (64, 4096, 4097):
        fetch(byte, n)
    byte = byte % 250 + 1
    ok(cu.cuCtxDestroy_v2(ctx))
a, b = context(), context()
for ctx in (a, b, a, b, b):  # two alive at a time
    ok(cu.cuCtxSetCurrent(ctx))
    fetch(byte, 64)
    byte += 1
ok(cu.cuCtxDestroy_v2(a))
ok(cu.cuCtxSetCurrent(b))
fetch(byte, 64)
bad = []

def many(k):
    try:
        ok(cu.cuCtxSetCurrent(b))
        for i in range(200):
            fetch((k * 31 + i) % 256, 16 + k)
    except BaseException as e:
        bad.append(e)

threads = [threading.Thread(target=many, args=(k,)) for k in range(8)]
[t.start() for t in threads]
[t.join() for t in threads]
assert not bad, bad
print("fetched")
"""


def test_contexts_and_threads(tchll):
    from triangle_counting_hll_b200 import _lib
    r = subprocess.run([sys.executable, "-c", CHILD, _lib.LIB_PATH], capture_output=True, text=True, timeout=240,
                       env=dict(os.environ))
    assert r.returncode == 0 and "fetched" in r.stdout, (r.returncode, r.stdout, r.stderr[-2000:])
