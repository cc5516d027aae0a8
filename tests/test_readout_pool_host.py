"""The readouts' pool of page-locked blocks without a GPU: the library's two calls that lock and unlock are stood in for, and
arrays end where the pool is at its least convenient."""
import gc
import os
import signal
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
    assert pool.locked == sum(c.locked.values()) <= pool.LIMIT
    assert {a: q.size for a, q in pool.slabs.items()} == c.locked and pool.idle <= pool.IDLE


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


def in_child(work):
    """The value of work() in a forked child, which ends there."""
    r, w = os.pipe()
    pid = os.fork()
    if pid == 0:
        code = 1
        signal.alarm(30)              # ends a child that hangs
        try:
            os.write(w, repr(work()).encode())
            code = 0
        finally:
            os._exit(code)
    os.close(w)
    with os.fdopen(r, "rb") as f:
        said = f.read().decode()
    assert os.waitpid(pid, 0)[1] == 0
    return said


def test_a_child_keeps_the_frame_it_was_forked_with(calls):
    """The parent goes on reading out: the child's array is a copy, as any other array of it is."""
    a = vf._out(20000)
    a[:] = 1
    go, out = os.pipe(), os.pipe()
    pid = os.fork()
    if pid == 0:
        signal.alarm(30)
        try:
            os.read(go[0], 1)
            os.write(out[1], repr((float(a[0]), float(a[-1]))).encode())
        finally:
            os._exit(0)
    a[:] = 7                        # what the next readout into its block would do
    os.write(go[1], b"x")
    os.close(out[1])
    with os.fdopen(out[0], "rb") as f:
        assert f.read() == b"(1.0, 1.0)"
    os.waitpid(pid, 0)


def test_a_childs_writes_stay_in_the_child(calls):
    a = vf._out(20000)
    a[:] = 3

    def child():
        a[:] = 99
        return float(a[0])

    assert in_child(child) == "99.0" and (a == 3).all()


def test_a_child_has_none_of_the_parents_blocks(calls):
    """Neither to use again nor to unlock: its arrays that end there are let go."""
    a, b = vf._out(20000), vf._out(1 << 20)
    del b
    gc.collect()
    vf._POOL.settle()
    assert vf._POOL.idle > 0 and len(vf._POOL.slabs) == 2

    def child():
        nonlocal a
        calls.rc = vf.VF_EINVAL                        # CUDA does not work in a forked child
        before = dict(calls.locked)
        del a
        gc.collect()
        q = vf._out(20000)
        q[:] = 5
        return before == calls.locked, vf._POOL.locked, vf._POOL.idle, vf._POOL.owns(q.ctypes.data), float(q.sum())

    assert in_child(child) == repr((True, 0, 0, False, 100000.0))


def test_a_block_from_before_a_fork_is_not_read_into_again(calls):
    """A page shared with a child moves when it is written to, which a device that goes on writing to it need not notice."""
    a = vf._out(20000)
    at = a.ctypes.data
    assert in_child(lambda: 1) == "1"
    del a
    gc.collect()
    assert vf._POOL.locked == 0 and not vf._POOL.owns(at)


def test_a_fork_while_another_thread_is_at_work_on_the_pool(calls):
    stop = threading.Event()

    def work():
        while not stop.is_set():
            vf._out(20000)

    threads = [threading.Thread(target=work, daemon=True) for _ in range(2)]
    for t in threads:
        t.start()
    try:
        for _ in range(20):
            calls_ok = in_child(lambda: (setattr(calls, "rc", vf.VF_EINVAL), vf._out(20000).size)[1])
            assert calls_ok == "20000"
    finally:
        stop.set()
        for t in threads:
            t.join(30)


def test_no_room_to_map_or_to_lock(calls, monkeypatch):
    """An ordinary array each time, and nothing counted as locked."""
    def none(*args, **kw):
        raise OSError(12, "Cannot allocate memory")

    with monkeypatch.context() as m:
        m.setattr(vf.mmap, "mmap", none)
        for _ in range(4):
            a = vf._out(1 << 22)
            a[:] = 1
            assert a.size == 1 << 22 and not vf._POOL.owns(a.ctypes.data) and vf._POOL.locked == 0
    calls.rc = vf.VF_EINVAL
    assert not vf._POOL.owns(vf._out(20000).ctypes.data) and vf._POOL.locked == 0
    calls.rc = vf.VF_OK
    assert vf._POOL.owns(vf._out(20000).ctypes.data)


def test_an_array_made_read_only_can_be_made_writable_again(calls):
    a = vf._out(20000)
    assert vf._POOL.owns(a.ctypes.data)
    for q in (a, a[5:], a.reshape(100, 200)):
        q.flags.writeable = False
        with pytest.raises(ValueError):
            q[...] = 1
        q.flags.writeable = True
        q[...] = 2
    assert (a == 2).all() and a.dtype == np.float32 and a.shape == (20000,) and a.flags.aligned and a.flags.c_contiguous
    view = a[7:]
    del a, q
    gc.collect()
    b = vf._out(20000)
    b[:] = 3
    assert (view == 2).all()                            # a view keeps the block
    assert vf._out(20000, np.int32).dtype == np.int32


def test_arrays_of_all_sizes_keep_to_themselves(calls):
    """Taken and let go in any order, with sizes that slabs are left with room for and sizes that they are not: no two arrays
    meet, all lie in what is locked, and the locked memory stays near what is in use."""
    rng = np.random.default_rng(1)
    pool, held = vf._POOL, {}
    for k in range(4000):
        if held and rng.random() < 0.5:
            j = list(held)[rng.integers(len(held))]
            assert (held.pop(j) == j).all()
        else:
            a = vf._out(int(rng.integers(1, 200)) * int(rng.choice([100, 5000, 20000])), np.int32)
            a[:] = k
            if pool.owns(a.ctypes.data):
                assert pool.owns(a.ctypes.data + a.nbytes - 1) and a.ctypes.data % 256 == 0
            held[k] = a
        if len(held) > 60:
            held.clear()
        del a
        a = None
    assert all((a == k).all() for k, a in held.items())
    assert pool.locked <= pool.LIMIT


@pytest.mark.parametrize("n", [20000, 160000, 1 << 18, 550000, 1100000, 1400000, 3000000])
def test_what_is_locked_is_little_more_than_what_is_held(calls, n):
    """At most LIMIT; and of 100 MB and more in arrays of one size, at least six tenths."""
    pool = vf._POOL
    held = [vf._out(n) for _ in range(100_000_000 // (4 * n) + 1)]
    ours = [a for a in held if pool.owns(a.ctypes.data)]
    assert len(ours) == len(held) and sum(a.nbytes for a in ours) >= 0.6 * pool.locked


def test_a_programs_first_readout_locks_little(calls):
    a = vf._out(1000)
    assert vf._POOL.locked == vf._POOL.LEAST == 2 << 20
    b = [vf._out(1000) for _ in range(20)]
    assert vf._POOL.locked == vf._POOL.LEAST and vf._POOL.owns(vf._out(8 << 20).ctypes.data) and vf._POOL.locked == 34 << 20
    assert not vf._POOL.owns(vf._out((8 << 20) + 1).ctypes.data) and len(a) == len(b[0])
