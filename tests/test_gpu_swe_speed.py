"""The wave speed measured from a state in place: the bits of the largest max(|u|, |v|) + sqrt(g h) over the cells, each
operation rounded once (numpy's float32), at sizes about a thread's, a block's and the grid's share of cells, and over
states with dry, subnormal, negative, infinite and missing values."""
import numpy as np
import pytest

import vexfluid as vf
from _oracle import F, swe_params

pytestmark = pytest.mark.gpu

G, DRY = F(9.81), F(1e-6)


def expected(h, hu, hv):
    """The largest bits; a NaN speed is the largest of all."""
    with np.errstate(all="ignore"):
        u, v = np.where(h > DRY, hu / h, F(0)), np.where(h > DRY, hv / h, F(0))
        s = np.fmax(np.abs(u), np.abs(v)) + np.sqrt(G * h)
    return F("nan") if np.isnan(s).any() else s.max()


def states(kind, nx, ny):
    rng = np.random.default_rng(nx + ny)
    h, hu, hv = (a.astype(F) for a in (1 + 0.3 * rng.random((ny, nx)), rng.standard_normal((ny, nx)),
                                       rng.standard_normal((ny, nx))))
    if kind == "dry":
        h *= rng.random((ny, nx)) < 0.3
        h[-1, -1] = 1e-6
    elif kind == "tiny":
        h = np.ldexp(rng.uniform(0.5, 1, (ny, nx)), rng.integers(-148, -100, (ny, nx))).astype(F)
        hu, hv = hu * F(1e-38), hv * F(0)
    elif kind == "wide":
        hu = np.ldexp(hu, rng.integers(-120, 90, (ny, nx))).astype(F)
        hv[::2] = -0.0
    elif kind == "missing momentum":
        hu[ny // 2, nx // 2] = F("nan")
    elif kind == "missing both":
        hu[ny // 2, nx // 2] = hv[ny // 2, nx // 2] = F("nan")
    elif kind == "negative":
        h[ny // 2, nx // 2] = -1.0
    elif kind == "missing depth":
        h[-1, -1] = F("nan")
    elif kind == "infinite":
        hv[-1, 0] = F("inf")
    elif kind == "infinite depth":
        h[0, -1] = F("inf")
    return h, hu, hv


@pytest.mark.parametrize("nx,ny,kind", [(1, 1, "sea"), (7, 3, "sea"), (257, 8, "sea"), (2049, 1, "sea"), (1700, 1500, "sea")] +
                         [(61, 47, k) for k in ("dry", "tiny", "wide", "missing momentum", "missing both", "negative",
                                                "missing depth", "infinite", "infinite depth")])
def test_measured_speed_is_the_largest_of_all_cells(nx, ny, kind):
    state = states(kind, nx, ny)
    with vf.PatchSimulation(nx, ny, (0, 0, 0, 0)) as p:
        p.load(*[a.ravel() for a in state], np.asarray(swe_params(G, 0.45, 1, 1, DRY), F).view(np.int32))
        p.measure_speed()
        got, want = F(p.fastest_wave()), expected(*state)
        assert got == want or (np.isnan(got) and np.isnan(want)), (got, want)


def wave_of(p, g, dry):
    with np.errstate(all="ignore"):
        h, hu, hv = (np.asarray(q, F) for q in p.read())
        u, v = np.where(h > dry, hu / h, F(0)), np.where(h > dry, hv / h, F(0))
        return (np.fmax(np.abs(u), np.abs(v)) + np.sqrt(g * h)).max()


@pytest.mark.parametrize("width", [0, 32, 64])
@pytest.mark.parametrize("g,dry", [(9.81, 0.0), (9.81, 1e-6), (1e-3, 1e-6)])
def test_a_steps_speed_over_a_film_of_subnormal_depth(g, dry, width):
    """The wave speed that a step leaves is that of the state it leaves, down to g h below the normal range."""
    nx, ny = 200, 20
    rng = np.random.default_rng(5)
    h = np.ldexp(rng.uniform(1, 2, nx * ny), rng.integers(-148, -127, nx * ny)).astype(F)
    with vf.PatchSimulation(nx, ny, (0, 0, 0, 0)) as p:
        p.set_tile_width(width)
        p.load(h, 0 * h, 0 * h, np.asarray(swe_params(g, 0.45, 1, 1, dry), F).view(np.int32))
        p.write_budget(0, 5)
        p.dispatch(1)
        got, want = F(p.fastest_wave()), wave_of(p, F(g), F(dry))
        assert want > 0 and got == want


def test_measured_speed_past_the_reciprocals_range():
    """A depth whose reciprocal is subnormal, under so little gravity that the current is most of the speed."""
    nx, ny = 61, 47
    rng = np.random.default_rng(6)
    h = np.ldexp(rng.uniform(1, 2, nx * ny), 126).astype(F)
    hu = (h * rng.uniform(0.5, 1.5, nx * ny)).astype(F)
    with vf.PatchSimulation(nx, ny, (0, 0, 0, 0)) as p:
        p.load(h, hu, 0 * h, np.asarray(swe_params(1e-38, 0.45, 1, 1, 0.0), F).view(np.int32))
        p.measure_speed()
        assert F(p.fastest_wave()) == wave_of(p, F(1e-38), F(0))
