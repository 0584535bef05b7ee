"""The engine's result arrays: memory is used again only when neither an array nor a view of it is left, is bounded, is ordinary memory, and is given back."""
import concurrent.futures
import gc
import importlib
import threading

import numpy as np
import pytest

engine = importlib.import_module("aws-k8s-ansible-provisioner_b200.engine")


def addr(a):
    return a.ctypes.data


def test_memory_is_reused_only_when_nobody_holds_a_view():
    r = engine._Results()
    a, c = r.array(2, 100), r.array(1, 10)
    assert addr(a) != addr(c)
    a[:] = 1.0
    at, row = addr(a), a[1][::2]
    del a
    gc.collect()
    b = r.array(2, 100)
    assert addr(b) != at and (row == 1.0).all()
    del row
    gc.collect()
    assert addr(r.array(2, 100)) == at and r.blocks == 3


@pytest.mark.parametrize("rows", [1, 3, 200])
def test_blocks_are_bounded_and_given_back(rows):
    r = engine._Results()
    held = [r.array(rows, 70000) for _ in range(9)]
    kept = {addr(a) for a in held[:min(r.BLOCKS, r.LIMIT // (rows * 70000 * 4))]}
    assert len({addr(a) for a in held}) == 9 and all(a.shape == (rows, 70000) and a.flags.writeable for a in held)
    assert r.array(0, 10).shape == (0, 10) and r.blocks == len(kept) and r.bytes <= r.LIMIT
    for a in held:
        a[:] = 1.0
    del a
    held.clear()
    gc.collect()
    again = [r.array(rows, 70000) for _ in range(len(kept))]
    assert {addr(a) for a in again} == kept
    one = r.array(1, 1)
    r.close()
    assert all((a == 1.0).all() for a in again)   # (what is lent stays as it is)
    again.clear()
    del one
    gc.collect()
    assert not r.free and not r.back and r.array(1, 1).shape == (1, 1)


def test_later_sizes_take_the_place_of_idle_ones():
    r = engine._Results()
    large = r.BLOCKS * 1000
    held = [r.array(1, 500) for _ in range(r.BLOCKS)]
    addrs = {addr(a) for a in held}
    fresh = r.array(1, large)   # (every block is lent)
    assert r.blocks == r.BLOCKS and r.bytes == r.BLOCKS * 2000
    del held
    gc.collect()
    a = r.array(1, large)
    at = addr(a)
    assert r.blocks == r.BLOCKS and r.bytes == (r.BLOCKS - 1) * 2000 + large * 4 and len(r.free) == r.BLOCKS - 1
    del a
    gc.collect()
    few = r.array(1, 500)   # a small result does not take the large block
    assert addr(few) in addrs
    b = r.array(1, large)
    assert addr(b) == at
    del b
    gc.collect()
    most = r.array(1, (r.LIMIT - 2000) // 4)   # makes room for itself as far as idle blocks go
    assert r.bytes == r.LIMIT and r.blocks == 2 and not r.free
    beyond = r.array(1, r.LIMIT // 4 + 1)
    assert beyond.shape == (1, r.LIMIT // 4 + 1) and r.bytes == r.LIMIT
    del fresh, few, most


def hold_and_compare(r, threads=6, turns=200):
    """Every thread makes a result, fills it and holds it until all of them have one: the addresses of those that are held together, turn by turn; raises what a thread raises."""
    meet, held = threading.Barrier(threads, timeout=60), [[None] * threads for _ in range(turns)]

    def work(k):
        try:
            for i in range(turns):
                a = r.array(1, 64)
                a[:] = k * 1000 + i
                held[i][k] = addr(a)
                meet.wait()
                assert (a == k * 1000 + i).all()
                meet.wait()   # (nobody makes the next one before all have looked)
                del a
        except BaseException:
            meet.abort()
            raise

    with concurrent.futures.ThreadPoolExecutor(threads) as pool:
        for done in [pool.submit(work, k) for k in range(threads)]:
            done.result()
    return held


def test_threads():
    r = engine._Results()
    assert all(len(set(addrs)) == len(addrs) for addrs in hold_and_compare(r))
    assert r.blocks <= r.BLOCKS and len(r.free) + len(r.back) == r.blocks


def test_threads_see_memory_that_is_lent_twice():
    """The check above on a pool that gives everybody the same memory."""

    class Wrong(engine._Results):
        one = np.zeros((1, 64), dtype=np.float32)

        def array(self, rows, cols):
            return self.one

    with pytest.raises((AssertionError, threading.BrokenBarrierError)):
        hold_and_compare(Wrong())


class Lib:
    """Stands for the library where an engine is closed."""

    def b2_engine_free(self, h):
        pass


def test_the_collector_may_close_engines_anywhere():
    """Engines in reference cycles are closed by the collector, which runs at any allocation: while another engine makes or gives back results, in the same thread too."""

    def work():
        for i in range(3000):
            gc.set_threshold(3 + i % 97, 1, 1)
            e = engine.Engine.__new__(engine.Engine)
            e.lib, e.h, e.me, e._results = Lib(), 1, e, engine._Results()
            held = [e._results.array(1, 64) for _ in range(3)]
            del held
            other = engine._Results()
            other.array(1, 64)
            other.close()

    old = gc.get_threshold()
    t = threading.Thread(target=work, daemon=True)
    try:
        t.start()
        t.join(60)
    finally:
        gc.set_threshold(*old)
    assert not t.is_alive()
