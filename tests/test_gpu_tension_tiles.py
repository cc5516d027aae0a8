"""Surface tension's passes over the tiles the fluid reaches, against the same passes over every tile.

Under the exact schedule the grid is the same bits in any particle order, and the passes and the gather round each
operation once, so a run whose steps sort (live tiles only) equals, particle by particle and bit for bit, the run of the
same particles that never sorts (every tile)."""
import numpy as np
import pytest

import vexfluid as vf
from _oracle import F

pytestmark = pytest.mark.gpu


def drops(dims, balls, seed):
    rng = np.random.default_rng(seed)
    at, vel = [], []
    for centre, radius, v in balls:
        k = np.stack(np.meshgrid(*[np.arange(n) for n in dims], indexing="ij"), -1).reshape(-1, 3)
        k = k[((k + 0.5 - np.array(centre)) ** 2).sum(1) <= radius ** 2]
        k = np.repeat(k, 8, axis=0)
        at.append(k + rng.random(k.shape) * 0.999)
        vel.append(np.tile(v, (len(k), 1)))
    at, vel = np.concatenate(at).astype(F), np.concatenate(vel).astype(F)
    m = np.full(len(at), F(1 / 8), F)
    m = (m.view(np.int32) + np.arange(len(m), dtype=np.int32)).view(F)   # a distinct mass tags each particle
    return [np.ascontiguousarray(at[:, a]) for a in range(3)], [np.ascontiguousarray(vel[:, a]) for a in range(3)], m


@pytest.mark.parametrize("dims,balls", [
    # a drop that crosses tiles along every axis and leaves the ones it started in; odd sizes, ragged last tiles
    ((75, 45, 37), [((12.0, 10.0, 9.0), 6.0, (900.0, 500.0, 400.0))]),
    # drops on a floor, in a corner and apart; an even row; a tile edge through a drop
    ((96, 32, 40), [((32.0, 5.0, 20.0), 4.5, (0.0, -50.0, 0.0)), ((4.0, 4.0, 4.0), 3.5, (0.0, 0.0, 0.0)),
                    ((70.0, 16.0, 30.0), 5.0, (-800.0, 0.0, 0.0))]),
    # a box smaller than one tile
    ((9, 7, 6), [((4.5, 3.5, 3.0), 2.0, (20.0, 0.0, 0.0))]),
])
def test_live_tiles_give_the_bits_of_every_tile(dims, balls):
    at, vel, m = drops(dims, balls, 3)
    p = vf.flip3_params(1e-3, 0.0, -30.0, 0.0, 2500.0, 1.0, 60.0)
    runs = []
    for sort in (True, False):
        with vf.ParticleSimulation3(*dims, len(m), tension=True, schedule=vf.VF_P2G_FIXED, sort=sort) as s:
            s.load(at, vel, m, p)
            s.advance(20)
            s.read("gu")        # a readout updates every node, between steps
            s.advance(23)
            order = np.argsort(s.read("m").view(np.int32))
            runs.append([s.read(f).view(np.int32)[order] for f in ("x", "y", "z", "u", "v", "w", "j", "c00", "c12", "c22")]
                        + [s.read(f).view(np.int32) for f in ("gm", "gmu", "gu", "gv", "gw")])
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
