"""The last convolution's tiles of 112 output pixels (four warps of 28): widths about a warp's, a tile's and two tiles',
heights about a tile's four rows, a batch; against the CPU float64 restatement, which rounds to bf16 at the same points.

Bar: 1e-2 of the largest |value|: fp32 summation order and an occasional one-ulp flip of a bf16 activation, 2^-8 of one
of some 800 products."""
import sys

import numpy as np
import pytest

import vexfluid as vf
from conftest import ROOT
from test_gpu_cnn import random_params, state

sys.path.insert(0, str(ROOT / "oracle"))
import cnn_ref  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx", [(7, 27), (5, 28), (9, 29), (4, 57), (4, 111), (8, 112), (3, 113), (6, 140), (10, 225)])
def test_fluxes_at_the_tiles_edges(ny, nx):
    rng = np.random.default_rng(ny * 1000 + nx)
    params = random_params(rng, scale3=1.0)
    with vf.FluxNet(nx, ny) as net:
        net.params(params)
        S = state(rng, ny, nx)
        net.put(0, 0, *S)
        got = net.fluxes(0)
        want = cnn_ref.forward(S, params)["y3"]
        assert np.abs(got[:, :, :6] - want).max() <= 1e-2 * np.abs(want).max()
        assert not got[:, :, 6:].any()
