"""Readouts before and after a fork, on the page-locked blocks that a device writes to. The child touches no CUDA: it looks at
arrays that it has, and ends."""
import os
import signal

import numpy as np
import pytest

import vexfluid as vf
from _oracle import F

pytestmark = pytest.mark.gpu


def test_parent_and_child_keep_their_own_frames():
    n = 200000
    rng = np.random.default_rng(1)
    x, y = (8 + rng.random((2, n)) * 40).astype(F)
    z = np.zeros(n, F)
    with vf.ParticleSimulation(64, 64, n) as s:
        s.load(x, y, z, z, z + 1, vf.flip_params(1e-4, 0, -9.8, 10, 1))
        s.sort()
        a, b = s.read("x"), s.read("y")
        assert vf._POOL.owns(a.ctypes.data)
        sums = float(a.sum(dtype=np.float64)), float(b.sum(dtype=np.float64))
        go, out = os.pipe(), os.pipe()
        pid = os.fork()
        if pid == 0:
            signal.alarm(30)
            code = 1
            try:
                os.read(go[0], 1)
                a *= 0                                  # the child's own
                os.write(out[1], repr((float(b.sum(dtype=np.float64)), float(a.max()))).encode())
                code = 0
            finally:
                os._exit(code)
        del b
        later = [s.read(k) for k in ("y", "x", "y", "x")]   # where b was, had its block been used again
        a += 0                                          # the parent's pages of it move now, if they do
        os.write(go[1], b"x")
        os.close(out[1])
        with os.fdopen(out[0], "rb") as f:
            said = f.read().decode()
        assert os.waitpid(pid, 0)[1] == 0
        assert said == repr((sums[1], 0.0))
        assert float(a.sum(dtype=np.float64)) == sums[0]
        for k, q in enumerate(later):
            assert float(q.sum(dtype=np.float64)) == sums[1 - k % 2]
        del a, later
        again = [s.read("x") for _ in range(3)]
        assert all(float(q.sum(dtype=np.float64)) == sums[0] for q in again)
