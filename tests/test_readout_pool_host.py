"""The readouts' pool of page-locked blocks without a GPU: the library's two calls that lock and unlock are stood in for, and
arrays end where the pool is at its least convenient."""
import gc
import threading
import types

import numpy as np
import pytest

import vexfluid as vf


class Calls(types.SimpleNamespace):
    """The stand-in: what is locked, by address."""

    def __init__(self):
        super().__init__(locked={}, rc=vf.VF_OK)

    def vf_host_register(self, address, size):
        if self.rc == vf.VF_OK:
            assert address not in self.locked
            self.locked[address] = size
        return self.rc

    def vf_host_unregister(self, address):
        del self.locked[address]
        return vf.VF_OK


@pytest.fixture
def calls(monkeypatch):
    c = Calls()
    monkeypatch.setattr(vf, "lib", lambda: c)
    monkeypatch.setattr(vf, "_POOL", vf._PinnedPool())
    yield c
    gc.collect()
    pool = vf._POOL
    assert pool.locked == sum(c.locked.values()) <= pool.LIMIT and set(pool.blocks) == set(c.locked)


def finishes(work, seconds=60):
    """Runs work on a thread of its own; False where it never returns."""
    done = []
    t = threading.Thread(target=lambda: done.append(work()), daemon=True)
    t.start()
    t.join(seconds)
    return bool(done)


def test_arrays_that_end_in_a_collection_inside_the_pool(calls):
    """Readouts caught in reference cycles, so that the collector ends them, which it may while the pool is at work."""
    class Frame:
        pass

    def work():
        old = gc.get_threshold()
        gc.set_threshold(1, 1, 1)
        try:
            for k in range(3000):
                f = Frame()
                f.me, f.a = f, vf._out(20000 + 9000 * (k % 3))
                f.a[0] = k
                vf._POOL.owns(0)
        finally:
            gc.set_threshold(*old)
        return True

    assert finishes(work)


def test_a_finaliser_that_reads_out_itself(calls):
    """... and one that takes an array of its own there, as an object does that saves a last frame when it ends."""
    last = []

    class Frame:
        def __del__(self):
            last[:] = [vf._out(30000)]
            last[0][:] = 7

    def work():
        old = gc.get_threshold()
        gc.set_threshold(1, 1, 1)
        try:
            for k in range(2000):
                f = Frame()
                f.me, f.a = f, vf._out(20000)
                f.a[:] = k
                assert (f.a == k).all()
        finally:
            gc.set_threshold(*old)
        return True

    assert finishes(work)
    last.clear()


def test_threads_end_each_others_arrays(calls):
    def work(k, out):
        for j in range(2000):
            a = vf._out(17000 + k)
            a[:] = k
            out.append(a)
            if j % 7 == 0:
                out.clear()
        return True

    shared, ok = [], []
    threads = [threading.Thread(target=lambda k=k: ok.append(work(k, shared)), daemon=True) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert len(ok) == 4
    shared.clear()


def test_idle_blocks_past_the_bound_are_unlocked(calls):
    pool = vf._POOL
    held = [vf._out(1 << 20) for _ in range(60)]                 # 4 MB each, 192 MB the limit
    assert sum(calls.locked.values()) == pool.LIMIT == pool.locked
    del held
    gc.collect()
    assert sum(calls.locked.values()) == pool.IDLE == pool.locked
