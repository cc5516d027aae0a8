"""The page-locked blocks that readouts return: an array keeps its values for as long as it or a view of it lives, a block comes
back after, the pool stays within its bound, and a returned array takes what an ordinary one does."""
import gc
import threading

import numpy as np
import pytest

import vexfluid as vf
from _oracle import F

pytestmark = pytest.mark.gpu


def sim(n=30000, value=0.0):
    s = vf.ParticleSimulation(64, 64, n)
    x = (8 + np.random.default_rng(int(value)).random(n) * 40).astype(F)
    s.load(x, x[::-1].copy(), np.full(n, value, F), np.zeros(n, F), np.ones(n, F), vf.flip_params(1e-4, 0, -9.8, 10, 1))
    return s, x


def test_arrays_outlive_later_readouts_and_their_handle():
    s, x = sim()
    first = s.read("x")
    view = s.read("y")[5:]
    later = [s.read("u") for _ in range(4)]
    s.close()
    del s
    gc.collect()
    assert np.array_equal(first, x) and np.array_equal(view, x[::-1][5:]) and all((q == 0).all() for q in later)
    first += 1                                   # an ordinary, writable array
    assert np.array_equal(first, x + F(1))
    with vf.Pinned(view.base if isinstance(view.base, np.ndarray) else first, first):
        pass
    assert np.array_equal(first, x + F(1))


def test_blocks_come_back_and_the_bound_holds():
    pool = vf._POOL
    s, x = sim()
    before = pool.locked
    for _ in range(300):
        s.read("x")
    assert pool.locked <= before + pool.LEAST * 8    # one block, used again and again
    held = []
    for _ in range(3000):                            # past the bound readouts go on in ordinary arrays
        held.append(s.read("x"))
        if len(held) * 120000 > pool.LIMIT + (8 << 20):
            break
    assert pool.locked <= pool.LIMIT
    assert all(np.array_equal(q, x) for q in held[::97])
    del held
    gc.collect()
    assert pool.locked <= pool.IDLE and np.array_equal(s.read("x"), x)


def test_threads_read_their_own_handles():
    bad = []

    def work(k):
        s, x = sim(20000 + k, float(k))
        for _ in range(100):
            a, u = s.read("x"), s.read("u")
            if not (np.array_equal(a, x) and (u == k).all()):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
