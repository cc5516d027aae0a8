"""The 2D sort's scan over block ranges at the sizes where a range, a block or a 16-byte access ends, and the single
scene's steps at the launch shapes that follow from particle and node counts.

Tolerances: the sort is exact; after tens of steps positions are within the step's bar of 1e-4 relative, so the grid's
sums are within 1e-4 of a node of unit mass, and a velocity (their quotient) within 1e-3 where a node holds a tenth."""
import numpy as np
import pytest

import vexfluid as vf
from _oracle import F, Flip2State, cells2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 2), (65, 65), (4097, 2), (4098, 2), (18, 242), (2049, 2051), (2050, 2052)])
def test_starts_and_order_equal_the_stable_sort(nx, ny):
    """1 cell; 2; one whole range of 4,096 cells and one more; 4,097 cells (a lone last count); 1,026 and 1,027 ranges,
    where a block takes two."""
    rng = np.random.default_rng(nx * ny)
    n = 5000
    x, y = (rng.random(n) * (nx - 1)).astype(F), (rng.random(n) * (ny - 1)).astype(F)
    x[:70], y[:70] = nx - 1, ny - 1        # a run in the last cell
    perm, starts = vf.sort2(nx, ny, x, y)
    cell = cells2(x, y, nx, ny)
    assert np.array_equal(starts, np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=(nx - 1) * (ny - 1)))]))
    assert np.array_equal(perm, np.argsort(cell, kind="stable"))


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("nx,ny,count,every", [(16, 12, 1, 1), (40, 33, 700, 3), (300, 200, 257, 2)])
def test_steps_follow_the_oracle(nx, ny, count, every, graph):
    """Odd sort intervals (the two grid buffers and the two particle sets come round at different steps), a packed scene
    with long runs in a warp, and a grid with far more nodes than particles. The node velocities read after the params
    change are those of the step that ran."""
    rng = np.random.default_rng(count)
    x = (6 + rng.random(count) * 4).astype(F)
    y = (5 + rng.random(count) * 3).astype(F)
    m = np.full(count, F(12.0 / count), F)
    params = vf.flip_params(1e-3, 0, -20, 200, 1)
    o = Flip2State(nx, ny, x, y, m)
    with vf.ParticleSimulation(nx, ny, count) as s:
        s.set_graph(graph)
        s.load(x, y, np.zeros_like(x), np.zeros_like(x), m, params)
        s.advance(7 * every, every)
        s.params(vf.flip_params(1e-3, 0, 500, 200, 1))
        got = {k: s.read(k) for k in ("gm", "gmu", "gmv", "gu", "gv", "x", "y", "m")}
    for k in range(7 * every):
        if k % every == 0:
            o.sort()
        o.step(params.view(F))
    for k in ("gm", "gmu", "gmv"):
        assert np.all(np.abs(got[k] - o.g[k]) <= 1e-4 * np.maximum(1, np.abs(o.g[k]))), k
    heavy = o.g["gm"] > 0.1
    for k in ("gu", "gv"):
        assert np.all(np.abs(got[k] - o.g[k])[heavy] <= 1e-3 * np.maximum(1, np.abs(o.g[k][heavy]))), k
        assert np.all(got[k][got["gm"] == 0] == 0)
    for k in ("x", "y"):
        assert np.all(np.abs(got[k] - o.a[k]) <= 1e-4 * np.abs(o.a[k])), k
