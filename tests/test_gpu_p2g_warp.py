"""The scatter that sums runs of a cell in a warp, at its edges: one particle, a warp's, a block's, one more and one less;
runs that end with the warp, cross it, fill several; particles without mass inside a run; sorted and not. And the order that a step leaves them in.

A node's mass and momentum are sums of N products of a few factors, so they differ from the exact sums by at most
(N + 24) units in the last place of the sum of the products' absolute values."""
import numpy as np
import pytest

import vexfluid as vf
from _oracle import F, Flip3State

pytestmark = pytest.mark.gpu

U = 2.0 ** -24
DIMS = (37, 21, 18)
CELLS = {
    "1": {(5, 3, 2): 1},
    "31": {(8, 8, 8): 31},
    "32": {(8, 8, 8): 16, (9, 8, 8): 16},
    "33": {(7, 7, 7): 1, (8, 7, 7): 31, (9, 7, 7): 1},
    "128": {(x, 8, 8): 16 for x in range(8)},
    "129": {(x, 8, 8): 16 + x // 7 for x in range(8)},
    "runs": {(16, 9, 3): 319, (17, 9, 3): 1, (20, 8, 4): 70, (7, 7, 7): 641},
    "edge": {(x, y, z): 1 + (x + y + z) % 12 for x in range(30, 35) for y in range(14, 19) for z in range(12, 16)},
}


def particles(kind, seed):
    rng = np.random.default_rng(seed)
    at = np.concatenate([np.array(c) + 0.5 + rng.uniform(0.01, 0.99, (n, 3)) for c, n in CELLS[kind].items()])
    at = rng.permutation(at).astype(F)
    vel, c = rng.uniform(-3, 3, (3, len(at))).astype(F), rng.uniform(-1, 1, (9, len(at))).astype(F)
    m = (np.full(len(at), 0.125, F).view(np.int32) + np.arange(len(at), dtype=np.int32)).view(F)
    m[3::11] = 0
    return [np.ascontiguousarray(at[:, a]) for a in range(3)], list(vel), list(c), m


def exact_grid(at, vel, c, m):
    at, vel, c, m = [np.asarray(q, np.float64) for q in (at, vel, c, m)]
    cell = [np.minimum(np.floor(q - 0.5), n - 3).astype(int) for q, n in zip(at, DIMS)]
    f = [q - k for q, k in zip(at, cell)]
    w = [(0.5 * (1.5 - q) ** 2, 0.75 - (q - 1) ** 2, 0.5 * (q - 0.5) ** 2) for q in f]
    sums, bound = np.zeros((4, np.prod(DIMS))), np.zeros((4, np.prod(DIMS)))
    for k in range(27):
        o = (k % 3, k // 3 % 3, k // 9)
        node = ((cell[2] + o[2]) * DIMS[1] + cell[1] + o[1]) * DIMS[0] + cell[0] + o[0]
        wm = w[0][o[0]] * w[1][o[1]] * w[2][o[2]] * m
        np.add.at(sums[0], node, wm)
        np.add.at(bound[0], node, wm)
        for a in range(3):
            d = [c[3 * a + e] * (o[e] - f[e]) for e in range(3)]
            np.add.at(sums[1 + a], node, wm * (vel[a] + sum(d)))
            # formed from the stencil's middle node: m (v + C (1 - f)) + m C (o - 1)
            np.add.at(bound[1 + a], node, wm * (np.abs(vel[a]) + sum(np.abs(c[3 * a + e]) * (np.abs(1 - f[e]) + abs(o[e] - 1)) for e in range(3))))
    return sums, bound


@pytest.mark.parametrize("sort", [True, False])
@pytest.mark.parametrize("kind", sorted(CELLS))
def test_runs_match_the_exact_sums(kind, sort):
    at, vel, c, m = particles(kind, 7)
    n = len(m)
    with vf.ParticleSimulation3(*DIMS, n, tait=True, schedule=vf.VF_P2G_WARP, sort=sort) as s:
        s.load(at, vel, m, vf.flip3_params(1e-3, 0.0, 0.0, 0.0, 50.0, 1.0))
        for k in range(9):
            s.write(f"c{k // 3}{k % 3}", c[k])
        s.run(vf.VF3_PASS_SORT | vf.VF3_PASS_CLEAR | vf.VF3_PASS_SCATTER)
        grid = s.grid()
        sums, bound = exact_grid(at, vel, c, m)
        for f in range(4):
            assert np.all(np.abs(grid[f].ravel() - sums[f]) <= (n + 24) * U * bound[f]), f


@pytest.mark.parametrize("schedule", [vf.VF_P2G_WARP, vf.VF_P2G_ATOMIC, vf.VF_P2G_FIXED])
@pytest.mark.parametrize("kind", sorted(CELLS))
def test_a_step_leaves_the_particles_in_the_stable_order(kind, schedule):
    """The dense gather gives each particle its place in its cell: the oracle's stable counting sort."""
    at, vel, _, m = particles(kind, 9)
    o = Flip3State(*DIMS, *at, m)
    o.sort()
    with vf.ParticleSimulation3(*DIMS, len(m), tait=True, schedule=schedule) as s:
        s.load(at, vel, m, vf.flip3_params(1e-3, 0.0, 0.0, 0.0, 50.0, 1.0))
        s.advance(1)
        assert np.array_equal(s.read("m").view(np.int32), o.a["m"].view(np.int32))
        s.advance(2)
        assert np.array_equal(np.sort(s.read("m")), np.sort(m))


@pytest.mark.parametrize("n,count", [(32, 4999), (32, 5000), (32, 5001), (33, 5000), (64, 179999), (64, 180000)])
def test_replayed_steps_on_both_sides_of_the_overlap_rule(n, count):
    """Steps replayed from a graph, whose launches overlap or not by the size, against the same steps launched one by one:
    the order of the grid's additions differs, by units in the last place of the sums, over 16 short steps."""
    rng = np.random.default_rng(count)
    at = [np.clip(4 + rng.random(count) * (n - 8), 2, n - 3).astype(F) for _ in range(3)]
    vel = [rng.uniform(-20, 20, count).astype(F) for _ in range(3)]
    m = (np.full(count, 0.125, F).view(np.int32) + np.arange(count, dtype=np.int32)).view(F)
    out = []
    for graph in (False, True):
        with vf.ParticleSimulation3(n, n, n, count, tait=True, schedule=vf.VF_P2G_WARP) as s:
            s.set_graph(graph)
            s.load(at, vel, m, vf.flip3_params(1e-4, 0.0, -9.8, 0.0, 50.0, 1.0))
            s.advance(16)
            order = np.argsort(s.read("m"))
            out.append({k: s.read(k)[order] for k in ("m", "x", "y", "z", "u", "v", "w", "j")})
    for k, a in out[0].items():
        assert np.all(np.abs(out[1][k] - a) <= 1e-4 * max(1, np.abs(a).max())), k
