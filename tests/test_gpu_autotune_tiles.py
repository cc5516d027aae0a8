"""The tuner's last choice: the tiles that each key's trial chose, or the default one for every scene, as the cache holds
it. A cache written before the choice existed, without it, still means the keys' tiles."""
import json

import numpy as np
import pytest

import vexfluid as vf

pytestmark = pytest.mark.gpu

SHAPES = [(48, 48, 3000), (40, 24, 1), (100, 60, 600)]


def scenes():
    rng = np.random.default_rng(5)
    params = vf.flip_params(1e-4, 0.0, -9.0, 4e3, 1.0)
    cols = [[rng.uniform(2, nx - 2, n).astype(np.float32) for nx, _, n in SHAPES],
            [rng.uniform(2, ny - 2, n).astype(np.float32) for _, ny, n in SHAPES]]
    cols += [[np.zeros(n, np.float32) for *_, n in SHAPES]] * 2 + [[np.full(n, 0.25, np.float32) for *_, n in SHAPES]]
    return [vf.Scene(nx, ny, n, params) for nx, ny, n in SHAPES], cols


@pytest.mark.parametrize("tiles", [None, (16, 16), (8, 8)])
def test_the_cache_holds_which_tiles(tmp_path, tiles):
    untuned, cols = scenes()
    cache = tmp_path / "tune.json"
    first, block, trials = vf.autotune(untuned, *cols, cache=cache, tait=True)
    assert trials >= len(vf.BATCH_TILES) + len(vf.BATCH_BLOCKS)
    doc = json.loads(cache.read_text())
    keyed = [e for e in doc["entries"] if "ppc" in e]
    last = [e for e in doc["entries"] if "keys" in e]
    assert len(last) == 1 and ("tile_x" in last[0]) == ("tile_y" in last[0])
    if "tile_x" in last[0]:
        assert {s.tile for s in first} == {(16, 16)} == {(last[0]["tile_x"], last[0]["tile_y"])}
    for e in keyed:   # tiles that are not the default's, so that it shows whose are taken
        e["tile_x"], e["tile_y"] = 32, 16
    for e in last:
        e.pop("tile_x", None)
        e.pop("tile_y", None)
        if tiles:
            us = e.pop("us_per_step")
            e.update(tile_x=tiles[0], tile_y=tiles[1], us_per_step=us)
    cache.write_text("\n".join(json.dumps(e) for e in keyed + last))
    again, block2, trials2 = vf.autotune(untuned, *cols, cache=cache, tait=True)
    assert trials2 == 0 and block2 == block
    assert {s.tile for s in again} == {tiles or (32, 16)}
