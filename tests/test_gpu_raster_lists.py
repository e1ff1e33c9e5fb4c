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
