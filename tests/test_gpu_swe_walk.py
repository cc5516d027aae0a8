"""The step kernel's walk over two columns a lane: tiles of every height at the sizes where a tile, a warp's 62 columns or a
pair ends, and states whose quotients leave the short way (vanishing momenta, dry cells, overflowing depths), against the
oracle bit for bit."""
import numpy as np
import pytest

from _oracle import F, OracleSweBackend, Stepper, swe_params
from test_gpu_swe import GpuSweBackend

pytestmark = pytest.mark.gpu


def run(nx, ny, edges, state, steps, width, params=None):
    params = swe_params(9.81, 0.45, 1, 1, 1e-6) if params is None else params
    a = Stepper(OracleSweBackend(nx, ny, edges), nx, ny)
    b = Stepper(GpuSweBackend(nx, ny, edges, width), nx, ny)
    for s in (a, b):
        s.set(*[np.ascontiguousarray(q, F).ravel() for q in state], params, 1e9)
    for k in range(steps):
        a.step(1)
        b.step(1)
        sa, sb = a.read(), b.read()
        for f in range(3):
            same = (sa[f].view(np.int32) == sb[f].view(np.int32)) | (np.isnan(sa[f]) & np.isnan(sb[f]))
            assert same.all(), (k, f, np.flatnonzero(~same)[:5])
        assert a.ticks() == b.ticks() and a.clamped() == b.clamped(), k


def sea(nx, ny, seed=1):
    rng = np.random.default_rng(seed)
    return [1 + 0.3 * rng.random((ny, nx)), 0.4 * rng.standard_normal((ny, nx)), 0.4 * rng.standard_normal((ny, nx))]


@pytest.mark.parametrize("width", [0, 32, 64])
@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 5), (61, 3), (62, 17), (63, 16), (123, 9), (247, 33), (248, 2), (249, 18),
                                   (496, 31), (501, 4)])
@pytest.mark.parametrize("edges", [(0, 0, 0, 0), (1, 0, 0, 1)])
def test_sizes_around_a_tile(nx, ny, edges, width):
    run(nx, ny, edges, sea(nx, ny), 6, width)


@pytest.mark.parametrize("nx,ny,width", [(2700, 520, 64), (1200, 1100, 64), (700, 600, 64)])
def test_grids_that_take_taller_tiles(nx, ny, width):
    run(nx, ny, (0, 1, 0, 0), sea(nx, ny), 3, width)


@pytest.mark.parametrize("width", [0, 64])
def test_momenta_through_every_power_of_two(width):
    """Signed momenta from the largest ordinary ones down through the subnormals to both zeros, in neighbouring cells, and a
    wave that runs out over still water."""
    nx, ny = 300, 40
    rng = np.random.default_rng(2)
    h, hu, hv = sea(nx, ny)
    e = np.linspace(-149, 2, nx * ny).reshape(ny, nx)
    hu = np.ldexp(rng.uniform(-1, 1, (ny, nx)), np.rint(e).astype(int))
    hv = np.ldexp(rng.uniform(-1, 1, (ny, nx)), np.rint(e[::-1, ::-1]).astype(int))
    hu[:, ::7], hv[::3] = -0.0, 0.0
    run(nx, ny, (0, 0, 1, 0), (h, hu, hv), 8, width)
    bump = np.ones((ny, nx))
    bump[:, 20:30] += 0.25
    run(nx, ny, (0, 0, 0, 0), (bump, 0 * bump, 1e-6 * (bump - 1)), 120, width)


@pytest.mark.parametrize("width", [0, 64])
def test_dry_beds_and_extreme_depths(width):
    """Dry cells beside wet ones, films at and under the dry depth, depths past the ordinary range either way, and momenta
    that overflow the fluxes."""
    nx, ny = 256, 48
    rng = np.random.default_rng(3)
    h, hu, hv = sea(nx, ny)
    h[:, 90:140] = 0.0
    h[10:20] *= 1e-6
    h[20:26, ::2] = F(1e-6)
    hu[:, 90:140] = 0.0
    hv[:, 95:120] = 0.0
    run(nx, ny, (0, 0, 0, 0), (h, hu * h, hv * h), 12, width)
    deep = np.ldexp(rng.uniform(1, 2, (ny, nx)), rng.integers(-60, 45, (ny, nx)))
    run(nx, ny, (0, 1, 0, 1), (deep, deep * rng.standard_normal((ny, nx)), deep * rng.standard_normal((ny, nx))), 4, width,
        swe_params(9.81, 0.45, 1, 1, 0.0))
    big = sea(nx, ny)
    big[1] *= F(1e25)
    big[2][::5] *= F(1e38)
    run(nx, ny, (0, 0, 0, 0), big, 1, width)


@pytest.mark.parametrize("width", [0, 32, 64])
def test_momenta_whose_velocities_overflow(width):
    """Depths from 2^-20 to 1 with momenta up to the largest float, infinite ones and none at all: velocities that overflow,
    in one component or both, alone among ordinary cells and in rows of their own."""
    nx, ny = 300, 48
    rng = np.random.default_rng(4)
    for share in (0.01, 0.3):
        for step_h in (False, True):
            h, hu, hv = sea(nx, ny)
            at = rng.random((ny, nx)) < share
            h[at] = np.ldexp(rng.uniform(1, 2, at.sum()), rng.integers(-20, 0, at.sum()))
            h = h.astype(F)
            for q in (hu, hv):
                some = at & (rng.random((ny, nx)) < 0.7)
                big = np.ldexp(rng.uniform(1, 2, some.sum()), rng.integers(100, 128, some.sum())) * rng.choice([-1, 1], some.sum())
                kind = rng.integers(0, 8, some.sum())
                big[kind == 0] = np.inf
                big[kind == 1] = -np.inf
                big[kind == 2] = np.finfo(F).max
                big[kind == 3] = np.nan
                q[some] = big
            if step_h:
                h[::3], hu[::3], hv[::3] = 0.25, 2e38, 0.1
            run(nx, ny, (0, 1, 0, 0), (h, hu.astype(F), hv.astype(F)), 2, width)


@pytest.mark.parametrize("width", [0, 32, 64])
def test_more_rows_than_a_launch_has_short_tiles(width):
    """65,536 tiles of four rows, one more than a launch takes: every tile width steps such a grid, and alike."""
    nx, ny = 4, 65535 * 4 + 1
    run(nx, ny, (0, 0, 0, 0), sea(nx, ny), 2, width)
