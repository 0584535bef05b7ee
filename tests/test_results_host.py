"""The engine's result arrays: memory is used again only when neither an array nor a view of it is left, is bounded, and is given back.  Against a library that counts."""
import ctypes as C
import gc
import importlib
import threading

import numpy as np
import pytest

engine = importlib.import_module("aws-k8s-ansible-provisioner_b200.engine")


class Lib:
    def __init__(self):
        self.held = {}

    def b2_host_alloc(self, size, out):
        buf = (C.c_char * size)()
        out._obj.value = C.addressof(buf)
        self.held[out._obj.value] = buf
        return 0

    def b2_host_free(self, p):
        del self.held[p]


def addr(a):
    return a.ctypes.data


def test_memory_is_reused_only_when_nobody_holds_a_view():
    lib = Lib()
    r = engine._Results(lib, 3000)
    a, c = r.array(2, 100), r.array(1, 10)
    assert {addr(a), addr(c)} == set(lib.held)
    a[:] = 1.0
    at, row = addr(a), a[1][::2]
    del a
    gc.collect()
    b = r.array(2, 100)
    assert addr(b) != at and (row == 1.0).all()
    del row
    gc.collect()
    assert addr(r.array(2, 100)) == at and len(lib.held) == 2


@pytest.mark.parametrize("first", [0, 1 << 16, 1 << 40])
def test_blocks_are_bounded_and_given_back(first):
    lib = Lib()
    r = engine._Results(lib, first)
    held = [r.array(3, 70000) for _ in range(9)]
    kept = {addr(a) for a in held[:r.BLOCKS]}
    assert len(lib.held) == (2 if first == 1 << 16 else 0) and len({addr(a) for a in held}) == 9 and all(a.shape == (3, 70000) and a.flags.writeable for a in held)
    assert r.array(0, 10).shape == (0, 10) and r.blocks == r.BLOCKS
    for a in held:
        a[:] = 1.0
    del a
    held.clear()
    gc.collect()
    again = [r.array(3, 70000) for _ in range(2)]
    assert {addr(a) for a in again} == kept
    small = r.array(1, 1)
    r.close()
    assert (again[0].sum(), again[1].sum()) == (210000.0, 210000.0)
    again.clear()
    del small
    gc.collect()
    assert not r.free and not r.back and r.array(1, 1).shape == (1, 1)
    next_one = engine._Results(lib, first)   # (the closed engine's page-locked blocks serve the next one)
    assert len(lib.held) == (2 if first == 1 << 16 else 0)
    next_one.close()
    engine._page_locked.trim(0)
    assert not lib.held


def test_threads():
    lib = Lib()
    r = engine._Results(lib, 4096)

    def work(k):
        for i in range(200):
            a = r.array(1, 64)
            a[:] = k * 1000 + i
            assert (a == k * 1000 + i).all()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert len(lib.held) == 2 and r.blocks <= r.BLOCKS
