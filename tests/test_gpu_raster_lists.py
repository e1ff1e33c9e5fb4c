"""The raster's tile lists: numbers of triangles around which the lanes per warp
change, and triangles that meet many tiles (boxes of 12 and more), alone and
many of them one after another by their numbers."""
import numpy as np
import pytest

import oracle
from tests.conftest import random_seeds

pytestmark = pytest.mark.gpu

cu = pytest.importorskip("integer_delauney_b200._delauney_cuda")


def _check(W, H, seeds, P=8):
    tris, grid, _ = oracle.triangulate(W, H, oracle.sort_seeds(seeds, W, H), P, "reference")
    verts, got = cu.triangulate(W, H, seeds, border_padding=P, as_arrays=True)
    np.testing.assert_array_equal(verts, np.asarray(tris).reshape(-1, 5)[:, 2:5])
    np.testing.assert_array_equal(got, grid)


@pytest.mark.parametrize("n", [3, 2335, 2336, 2337, 4704, 4705, 9439, 9441, 18911, 18913])
def test_triangles_per_warp(n):
    """Twice the seeds and 64 more are 148 x 8 x 4, 8, 16 and 32 triangles here."""
    _check(400, 300, random_seeds(400, 300, n, n))


@pytest.mark.parametrize("W,H", [(97, 65), (400, 300), (1601, 1537)])
@pytest.mark.parametrize("kind", ["columns", "fan", "lattice"])
def test_triangles_across_many_tiles(W, H, kind):
    if kind == "columns":      # slivers from side to side
        y = np.arange(0, H, 5)
        seeds = np.concatenate([np.stack([0 * y, y], 1), np.stack([0 * y[:-1] + W - 1, y[:-1] + 2], 1)])
    elif kind == "fan":        # a blob whose rim meets far seeds
        x, y = np.meshgrid(np.arange(W), np.arange(H))
        m = (x - W // 3) ** 2 + (y - H // 2) ** 2 < 15 ** 2
        seeds = np.concatenate([np.stack([x[m], y[m]], 1), [[W - 1, 0], [W - 2, H - 1], [0, H - 1]]])
    else:
        s = max(W, H) // 7
        x, y = np.meshgrid(np.arange(3, W, s), np.arange(5, H, s + 2))
        seeds = np.stack([x.ravel(), y.ravel()], 1)
    seeds = np.unique(seeds.astype(np.int32), axis=0)
    np.random.default_rng(1).shuffle(seeds)
    _check(W, H, np.ascontiguousarray(seeds))


@pytest.mark.parametrize("side,n,limit", [(64, 40, 0), (64, 40, 1), (200, 300, 0), (200, 300, 700)])
def test_overlapping_triangles_of_a_callers_grid(side, n, limit):
    """A grid of labelled squares in no order: more triangles than twice the
    seeds, on top of each other, drawn by their lists and (limit) without."""
    import ctypes
    from integer_delauney_b200 import _capi
    rng = np.random.default_rng(side)
    seeds = random_seeds(side, side, n, 2)
    s = oracle.sort_seeds(seeds, side, side)
    vg = np.zeros((side, side, 2), np.int32)
    vg[..., 0] = rng.integers(0, n, (side // 4 + 1, side // 4 + 1)).repeat(4, 0).repeat(4, 1)[:side, :side]
    o_tris, o_grid, _ = oracle.triangulate(side, side, s, 0, "numpy", vgrid=vg)
    assert len(o_tris) > 2 * n + 64
    ctx = _capi.Context(0)
    lib = _capi.load()
    _capi.check(lib.idl_selftest_limit(ctx.handle, 3, limit))
    grid = np.empty((side, side, 3), np.int32)
    count = ctypes.c_int64()
    for _ in range(2):
        _capi.check(lib.idl_triangulate(ctx.handle, side, side, seeds.ctypes.data, n, vg.ctypes.data, 0,
                                        _capi.MODE_REFERENCE, grid.ctypes.data, ctypes.byref(count), None, None))
        np.testing.assert_array_equal(grid, o_grid)
        tris = np.empty((count.value, 5), np.int32)
        _capi.check(lib.idl_get_triangles(ctx.handle, tris.ctypes.data, count.value))
        np.testing.assert_array_equal(tris, o_tris)
    ctx.close()
