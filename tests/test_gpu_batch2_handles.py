"""Batches of different tiles and CTA sizes in one process."""
import gc

import numpy as np
import pytest

import vexfluid as vf
from _oracle import F, Flip2State

pytestmark = pytest.mark.gpu


def batch(tile, block, seed, n=60, count=500):
    rng = np.random.default_rng(seed)
    params = vf.flip_params(1e-3, 0, -20, 200, 1)
    x, y = (5 + rng.random(count) * (n - 10)).astype(F), (5 + rng.random(count) * (n - 10)).astype(F)
    b = vf.BatchSimulation([vf.Scene(n, n, count, params, tile)], block=block)
    b.load(x, y, 0 * x, 0 * x, np.ones_like(x))
    return b, Flip2State(n, n, x, y, np.ones_like(x)), params


def follow(b, o, params, steps):
    """The step's bar: 1e-5 relative of positions a step, no particle near a wall."""
    b.advance(steps)
    b.finish()
    for _ in range(steps):
        o.sort()
        o.step(params.view(F))
    # a batch keeps its particles by tile: compare the grids, which do not care
    for k in ("gm", "gmu", "gmv"):
        e = o.g[k]
        assert np.all(np.abs(b.read(0, k) - e) <= 1e-4 * np.maximum(1, np.abs(e))), k


@pytest.mark.parametrize("block", [128, 256, 512])
@pytest.mark.parametrize("first", [1, 20])
def test_a_batch_steps_on_after_one_with_less_shared_memory(block, first):
    """Large tiles, then small ones, of one CTA size: the first batch's first launch of its own and its first captured
    graph both come after the second batch was made, and then again after that one is gone."""
    big = batch((32, 16), block, 1)
    small = batch((8, 8), block, 2)
    follow(*big, first)
    follow(*small, 3)
    small[0].close()
    del small
    gc.collect()
    third = batch((16, 16), block, 3)
    follow(*big, 17)
    follow(*third, 17)
    big[0].close()
    third[0].close()
