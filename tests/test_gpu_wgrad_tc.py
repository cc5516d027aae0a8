"""The weight and bias gradients on tcgen05 at the sizes where their tiles (4 rows x 128 pixels) end, against the
bf16-emulating restatement: the gradients' bar of the network's tests, 2e-2 of each block's norm."""
import numpy as np
import pytest

import vexfluid as vf
from test_gpu_cnn import blocks, cnn_ref, random_params, smooth, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx,batch", [(4, 128, 1), (5, 129, 1), (3, 3, 2), (1, 1, 1), (18, 260, 3), (7, 127, 1), (70, 40, 2)])
def test_gradients_at_tile_edges(ny, nx, batch):
    rng = np.random.default_rng(ny * 1000 + nx)
    params = random_params(rng)
    s_flux, s_res = 1e-2, 1e-3
    samples = []
    for _ in range(batch):
        S = state(rng, ny, nx)
        P = (S + np.stack([smooth(rng, ny, nx, 2e-3) for _ in range(3)])).astype(np.float32)
        T = (S + np.stack([smooth(rng, ny, nx, 2e-3) for _ in range(3)])).astype(np.float32)
        samples.append((S, P, T))
    with vf.FluxNet(nx, ny, batch=batch, samples=batch, s_flux=s_flux, s_res=s_res) as net:
        net.params(params)
        for k, parts in enumerate(samples):
            for kind, a in enumerate(parts):
                net.put(k, kind, *a)
        g, loss = net.gradients(list(range(batch)))
    ref_loss, ref = cnn_ref.loss_and_gradients(samples, params, s_flux, s_res)
    assert abs(loss - ref_loss) <= 1e-4 * ref_loss
    got = blocks(g)
    for name in ref:
        # a block that the image is too small to reach is zero on both sides
        assert np.linalg.norm(got[name] - ref[name]) <= 2e-2 * np.linalg.norm(ref[name]) + 1e-12, name


@pytest.mark.parametrize("ny,nx,batch", [(70, 40, 2), (18, 260, 3), (300, 500, 4)])
def test_bias_gradients_do_not_depend_on_which_warp_ends_first(ny, nx, batch):
    """A CTA's four warps sum the bias gradient from the stages that its weight gradients are then added up in; a row of a
    tile cleared too soon would be a 70th of a sum and more. Run to run the sums differ by the order of their additions: some
    N numbers of either sign add up to sqrt(N) of their size, so by 2^-24 N / sqrt(N) of it at most 3e-5 here, and by 3e-4
    of the block's norm never."""
    rng = np.random.default_rng(ny)
    with vf.FluxNet(nx, ny, batch=batch, samples=batch, s_flux=1e-2, s_res=1e-3) as net:
        net.params(random_params(rng))
        for k in range(batch):
            S = state(rng, ny, nx)
            for kind in range(3):
                net.put(k, kind, *(S + (kind > 0) * np.stack([smooth(rng, ny, nx, 2e-3) for _ in range(3)])).astype(np.float32))
        runs = [blocks(net.gradients(list(range(batch)))[0]) for _ in range(30)]
    for name in ("b1", "b2", "b3"):
        first = runs[0][name]
        assert np.linalg.norm(first) > 0
        for r in runs[1:]:
            assert np.linalg.norm(r[name] - first) <= 3e-4 * np.linalg.norm(first), name
