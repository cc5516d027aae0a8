"""A 2D grid within a stride of the launches of 2^31 nodes, the most a handle takes."""
import numpy as np
import pytest
import torch

import vexfluid as vf
from _oracle import F, Flip2State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
def test_a_particle_falls_in_the_far_corner_of_the_largest_grid(graph):
    """46340^2 = 2^31 - 88,048 nodes: fewer than the threads of a launch short of the end of an int, where an index that
    steps by the launch's threads would wrap. A free particle in the far corner has its velocity and gravity's, whatever a
    step before left in the grid: nine weights that add up to one within 9 roundings, four times over, within 1e-5."""
    n = 46340
    at = lambda v: np.full(1, v, F)
    with vf.ParticleSimulation(n, n, 1) as s:
        s.set_graph(graph)
        s.load(at(n - 9.5), at(n - 9.25), at(3), at(100), at(1), vf.flip_params(1e-3, 0, -1000, 0, 1))
        s.advance(4, 2)
        x, y, u, v = (float(s.read(k)[0]) for k in "xyuv")
    assert abs(u - 3) <= 3e-5 and abs(v - 96) <= 1e-3
    assert abs(x - (n - 9.5 + 0.012)) <= 0.02 and abs(y - (n - 9.25 + 0.39)) <= 0.02    # positions are 2^-8 apart there


def test_a_large_grid_takes_28_bytes_a_node():
    """The grid's 16, the sort's counts and starts 8, a readout's plane 4; and what a device rounds up, and no more."""
    n = 8192
    with vf.ParticleSimulation(3, 3, 1):    # the context and its first pages are not a grid's
        before = torch.cuda.mem_get_info()[0]
        with vf.ParticleSimulation(n, n, 1):
            assert before - torch.cuda.mem_get_info()[0] <= 28 * n * n + (64 << 20)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("nx,ny", [(4096, 4096), (4096, 4097)])
def test_steps_with_two_grid_buffers_and_with_one(nx, ny, graph):
    """The largest grid of two buffers and one row more; odd sort intervals, node velocities read after the params changed
    (twice) and after another step, against the oracle with the bars of the smaller grids' test."""
    count, every = 300, 3
    rng = np.random.default_rng(ny)
    x, y = (nx - 30 + rng.random(count) * 20).astype(F), (ny - 30 + rng.random(count) * 20).astype(F)
    m = np.full(count, F(1), F)
    params = vf.flip_params(1e-3, 0, -20, 200, 1)
    o = Flip2State(nx, ny, x, y, m)
    with vf.ParticleSimulation(nx, ny, count) as s:
        s.set_graph(graph)
        s.load(x, y, np.zeros_like(x), np.zeros_like(x), m, params)
        assert not s.read("gu").any() and not s.read("gm").any()
        for steps in (2 * every, 1):
            s.advance(steps, every)
            s.params(vf.flip_params(1e-3, 0, 500, 200, 1))
            s.params(params)
            got = {k: s.read(k) for k in ("gm", "gmu", "gmv", "gu", "gv", "x", "y")}
            for k in range(steps):
                if k % every == 0:
                    o.sort()
                o.step(params.view(F))
            for k in ("gm", "gmu", "gmv"):
                assert np.all(np.abs(got[k] - o.g[k]) <= 1e-4 * np.maximum(1, np.abs(o.g[k]))), k
            heavy = o.g["gm"] > 0.1
            for k in ("gu", "gv"):
                assert np.all(np.abs(got[k] - o.g[k])[heavy] <= 1e-3 * np.maximum(1, np.abs(o.g[k][heavy]))), k
            for k in ("x", "y"):
                assert np.all(np.abs(got[k] - o.a[k]) <= 1e-4 * np.abs(o.a[k])), k
