"""A 2D grid within a stride of the launches of 2^31 nodes, the most a handle takes."""
import numpy as np
import pytest

import vexfluid as vf
from _oracle import F

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
