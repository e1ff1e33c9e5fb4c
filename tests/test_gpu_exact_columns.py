"""The column pass at the edges of its 64-row bands and of the occupancy words:
canvases whose padding ends inside a band, at its edge and beyond it, columns
full of seeds, half full and with one seed; and the ids the row pass takes from
the seeds' ranks, alone and in a batch."""
import numpy as np
import pytest

import oracle
from tests.conftest import random_seeds

pytestmark = pytest.mark.gpu

cu = pytest.importorskip("integer_delauney_b200._delauney_cuda")


def _seeds(W, H, kind):
    if kind == "full":
        x, y = np.meshgrid(np.arange(W), np.arange(H))
        m = (x % 3 == 0) | (y % 7 == 2)
        return np.ascontiguousarray(np.stack([x[m], y[m]], 1).astype(np.int32)[::-1])
    n = W * H // 2 if kind == "half" else max(1, min(W * H, 5))
    return random_seeds(W, H, max(1, n), 7)


@pytest.mark.parametrize("P", [0, 1, 16, 63, 64, 65])
@pytest.mark.parametrize("W,H", [(1, 1), (3, 31), (33, 63), (31, 64), (5, 65), (64, 127), (7, 200), (257, 33)])
def test_bands(W, H, P):
    images, wants = [], []
    for kind in ("full", "half", "few"):
        seeds = _seeds(W, H, kind)
        s = oracle.sort_seeds(seeds, W, H)
        tris, grid, _ = oracle.triangulate(W, H, s, P, "exact")
        v, g = cu.triangulate(W, H, seeds, P, as_arrays=True, voronoi_mode="exact")
        np.testing.assert_array_equal(g, grid, err_msg=kind)
        np.testing.assert_array_equal(v, np.asarray(tris).reshape(-1, 5)[:, 2:5], err_msg=kind)
        images.append((W, H, seeds))
        wants.append(grid)
    for (v, g), grid in zip(cu.triangulate_batch(images, P, as_arrays=True, voronoi_mode="exact"), wants):
        np.testing.assert_array_equal(g, grid)


@pytest.mark.parametrize("W,H", [(33, 63), (31, 64), (64, 130)])
def test_bands_with_ties_by_insertion(W, H):
    """Dense lattices in a shuffled order: in a column and across columns, ties
    go to the seed inserted later, as through the passes."""
    from integer_delauney_b200 import _capi
    ctx = _capi.Context(0)
    ctx.set_schedule(0)
    for step in (1, 2, 4):
        x, y = np.meshgrid(np.arange(0, W, step), np.arange(1, H, 2 * step))
        seeds = np.stack([x.ravel(), y.ravel()], 1).astype(np.int32)
        np.random.default_rng(step).shuffle(seeds)
        got, want = (cu.Delaunay(W, H, len(seeds), 16) for _ in range(2))
        want.use_workspace(ctx)
        got.insert_deferred(seeds)
        want.insert_deferred(seeds)
        np.testing.assert_array_equal(got.get_voronoi_grid(), want.get_voronoi_grid())
        np.testing.assert_array_equal(got.get_triangles(), want.get_triangles())
        del want
    ctx.close()


@pytest.mark.parametrize("W,H", [(4224, 148), (4225, 148), (4225, 149), (4300, 1), (27001, 2)])
@pytest.mark.parametrize("n", [150, 900, 3500])
def test_wide_rows_that_are_few(W, H, n):
    """Rows of more than 4 224 columns, up to 148 of them: a block of 32 warps
    each; one more row or one column less: 8 warps."""
    seeds = random_seeds(W, H, n, 3)
    want, _ = oracle.voronoi("exact", W, H, oracle.sort_seeds(seeds, W, H))
    np.testing.assert_array_equal(cu.Voronoi().compute(W, H, seeds, voronoi_mode="exact"), want)
