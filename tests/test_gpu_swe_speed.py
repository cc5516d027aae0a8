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
