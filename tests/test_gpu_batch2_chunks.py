"""The batched step's work items at their edges: cells and tiles of one particle, of exactly a chunk, of one more and
one less, of several chunks; rounds of few cells (several lanes a cell) and of a warp's lanes and one; tiles that hang
past the grid; every block size and tile shape.

A node's mass and momentum are sums of N products of a few factors, so they differ from the exact sums by at most
(N + 16) units in the last place of the sum of the products' absolute values; what is gathered from them, by four
times that of the largest value (the affine matrix carries a factor of four)."""
import numpy as np
import pytest

import vexfluid as vf
from _oracle import F, Flip2State

pytestmark = pytest.mark.gpu

U = 2.0 ** -24
DT, GY, BULK = 1e-4, -9.0, 4e3
PER_THREAD = 5   # particles of a chunk per thread


def fills(kind, chunk):
    """Particles by cell, of a 40 x 37 grid."""
    if kind == "one particle":
        return {(7, 9): 1}
    if kind == "one cell":
        return {(20, 5): 2 * chunk + 1}
    if kind == "chunk edges":   # tiles of every shape: cells far apart
        out = {}
        for k, n in enumerate((chunk - 1, chunk, chunk + 1)):
            for c in range(64):
                out[(c % 8, 12 * k + c // 8)] = n // 64 + (c < n % 64)
        return out
    if kind.startswith("cells"):
        count = int(kind.split()[1])
        return {(c % 8, c // 8): 1 + (c * 7) % 23 for c in range(count)}
    if kind == "edge":          # the last cells of the grid
        return {(c, r): 1 + (c + r) % 5 for c in range(30, 38) for r in range(28, 35)}
    raise AssertionError(kind)


def scene(kind, chunk, seed):
    rng = np.random.default_rng(seed)
    x, y = [], []
    for (c, r), n in fills(kind, chunk).items():
        x.append(c + 0.5 + rng.uniform(0.01, 0.99, n))
        y.append(r + 0.5 + rng.uniform(0.01, 0.99, n))
    x, y = np.concatenate(x).astype(F), np.concatenate(y).astype(F)
    mix = rng.permutation(len(x))
    u, v = rng.uniform(-2, 2, (2, len(x))).astype(F)
    m = (np.full(len(x), 0.25, F).view(np.int32) + np.arange(len(x), dtype=np.int32)).view(F)
    return x[mix], y[mix], u, v, m


def exact_grid(nx, ny, x, y, u, v, m):
    """Mass and momenta of the first scatter (no affine matrix, no pressure) and the sums of the absolute values."""
    x, y, u, v, m = [np.asarray(a, np.float64) for a in (x, y, u, v, m)]
    col, row = np.minimum(np.floor(x - 0.5), nx - 3).astype(int), np.minimum(np.floor(y - 0.5), ny - 3).astype(int)

    def weights(f):
        return 0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2

    wx, wy = weights(x - col), weights(y - row)
    sums, bound = np.zeros((3, ny * nx)), np.zeros((3, ny * nx))
    for j in range(3):
        for i in range(3):
            node, w = (row + j) * nx + col + i, wx[i] * wy[j] * m
            for k, q in enumerate((w, w * u, w * v)):
                np.add.at(sums[k], node, q)
                np.add.at(bound[k], node, np.abs(q))
    return sums, bound


KINDS = ["one particle", "one cell", "chunk edges", "cells 2", "cells 3", "cells 16", "cells 17", "cells 33", "edge"]


@pytest.mark.parametrize("tile", vf.BATCH_TILES)
@pytest.mark.parametrize("block", vf.BATCH_BLOCKS)
def test_chunks_at_their_edges(block, tile):
    nx, ny = 40, 37
    parts = [scene(kind, PER_THREAD * block, 3 + k) for k, kind in enumerate(KINDS)]
    params = vf.flip_params(DT, 0.0, GY, BULK, 1.0)
    scenes = [vf.Scene(nx, ny, len(p[0]), params, tile) for p in parts]
    with vf.BatchSimulation(scenes, tait=True, block=block) as b:
        b.load(*[[p[f] for p in parts] for f in range(5)])
        for k, p in enumerate(parts):   # as loaded
            for name, want in zip(("x", "y", "u", "v", "m"), p):
                assert np.array_equal(b.read(k, name), want)
            assert np.all(b.read(k, "j") == 1) and not b.read(k, "c01").any()
        b.advance(1)
        b.finish()
        for k, p in enumerate(parts):
            n = len(p[0])
            sums, bound = exact_grid(nx, ny, *p)
            for name, want, limit in zip(("gm", "gmu", "gmv"), sums, bound):
                assert np.all(np.abs(b.read(k, name) - want) <= (n + 16) * U * limit), (KINDS[k], name)
            o = Flip2State(nx, ny, p[0], p[1], p[4], u=p[2], v=p[3])
            o.step(np.array((DT, 0.0, GY, BULK, 1.0), F), (1, 0))
            order, order_or = np.argsort(b.read(k, "m")), np.argsort(o.a["m"])
            for name in ("x", "y", "u", "v", "m", "j", "c00", "c01", "c10", "c11"):
                got, want = b.read(k, name)[order], o.a[name][order_or]
                assert np.max(np.abs(got - want)) <= 4 * (n + 16) * U * max(1, np.max(np.abs(want))), (KINDS[k], name)


@pytest.mark.parametrize("tile,block", [((8, 8), 512), ((16, 8), 128), ((16, 16), 256), ((32, 16), 128), ((32, 16), 512)])
@pytest.mark.parametrize("few", [0, 20, 60, 200])
def test_parts_of_a_chunk_at_their_edges(tile, block, few):
    """The gather's groups of 32, 64 and 128 threads take a chunk in parts of five particles a thread; how many threads goes
    by the chunks' mean length, which scenes of one particle bring down. Chunks of a part, of one more and one less, of two,
    and some of many, in one batch."""
    nx, ny = 40, 37
    rng = np.random.default_rng(few)
    parts = []
    for n in (159, 160, 161, 319, 320, 321, 639, 641, 1281):
        x, y = [np.concatenate([at + 0.5 + rng.uniform(0.01, 0.99, n) for at in (rng.integers(0, 8, n),)]).astype(F) for _ in "xy"]
        u, v = rng.uniform(-2, 2, (2, n)).astype(F)
        parts.append((x, y, u, v, (np.full(n, 0.25, F).view(np.int32) + np.arange(n, dtype=np.int32)).view(F)))
    parts += [scene("one particle", 1, k) for k in range(few)]
    params = vf.flip_params(DT, 0.0, GY, BULK, 1.0)
    with vf.BatchSimulation([vf.Scene(nx, ny, len(p[0]), params, tile) for p in parts], tait=True, block=block) as b:
        b.load(*[[p[f] for p in parts] for f in range(5)])
        b.advance(1)
        b.finish()
        for k, p in enumerate(parts):
            n = len(p[0])
            sums, bound = exact_grid(nx, ny, *p)
            for name, want, limit in zip(("gm", "gmu", "gmv"), sums, bound):
                assert np.all(np.abs(b.read(k, name) - want) <= (n + 16) * U * limit), (n, name)
            o = Flip2State(nx, ny, p[0], p[1], p[4], u=p[2], v=p[3])
            o.step(np.array((DT, 0.0, GY, BULK, 1.0), F), (1, 0))
            order, order_or = np.argsort(b.read(k, "m")), np.argsort(o.a["m"])
            for name in ("x", "y", "u", "v", "m", "j", "c00", "c01", "c10", "c11"):
                got, want = b.read(k, name)[order], o.a[name][order_or]
                assert np.max(np.abs(got - want)) <= 4 * (n + 16) * U * max(1, np.max(np.abs(want))), (n, name)
        b.advance(20)
        b.finish()


@pytest.mark.parametrize("block", vf.BATCH_BLOCKS)
@pytest.mark.parametrize("past", [-1, 0, 1, "twice"])
def test_as_many_chunks_as_warps(block, past):
    """The scatter's first chunks are dealt to the warps, the rest drawn: one chunk less than warps, as many, one more, and
    one more than two a warp. A chunk is one particle in a tile of its own."""
    import torch

    warps = torch.cuda.get_device_properties(0).multi_processor_count * 16   # the most that any of the kernels runs
    n = 2 * warps + 1 if past == "twice" else warps + past
    side = int(np.ceil(np.sqrt(n)))
    k = np.arange(n)
    x, y = (8 * (k % side) + 4.3).astype(F), (8 * (k // side) + 3.6).astype(F)
    u, v = np.random.default_rng(1).uniform(-2, 2, (2, n)).astype(F)
    m = (np.full(n, 0.25, F).view(np.int32) + np.arange(n, dtype=np.int32)).view(F)
    nx = 8 * side + 3
    with vf.BatchSimulation([vf.Scene(nx, nx, n, vf.flip_params(DT, 0.0, GY, BULK, 1.0), (8, 8))], tait=True, block=block) as b:
        b.load(*[[a] for a in (x, y, u, v, m)])
        b.advance(1)
        b.finish()
        sums, bound = exact_grid(nx, nx, x, y, u, v, m)
        for name, want, limit in zip(("gm", "gmu", "gmv"), sums, bound):
            assert np.all(np.abs(b.read(0, name) - want) <= 17 * U * limit), name
        o = Flip2State(nx, nx, x, y, m, u=u, v=v)
        o.step(np.array((DT, 0.0, GY, BULK, 1.0), F), (1, 0))
        order = np.argsort(b.read(0, "m"))
        assert np.array_equal(b.read(0, "m")[order], m)
        for name in ("x", "y", "u", "v", "j"):
            want = o.a[name][np.argsort(o.a["m"])]
            got = b.read(0, name)[order]
            assert np.max(np.abs(got - want)) <= 4 * 17 * U * max(1, np.max(np.abs(want))), name
