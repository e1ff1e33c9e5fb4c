"""Timed and profiled calls: the same route as the plain ones, with the pass
count of the iteration beside the times."""
import ctypes

import numpy as np
import pytest

import oracle
from tests.conftest import clustered_seeds, random_seeds

pytestmark = pytest.mark.gpu

cu = pytest.importorskip("integer_delauney_b200._delauney_cuda")
from integer_delauney_b200 import _capi  # noqa: E402

W, H, P = 417, 301, 8


def _seeds(kind):
    if kind == "uniform":
        return random_seeds(W, H, 2000, 4)
    if kind == "sparse":
        return random_seeds(W, H, 30, 4)
    if kind == "dense":
        return random_seeds(W, H, W * H // 3, 4)
    if kind == "clustered":
        return clustered_seeds(W, H, 900, seed=4, blobs=5, sigma=7.0)
    if kind == "circle":
        a = np.linspace(0, 2 * np.pi, 109, endpoint=False)
        p = np.stack([np.rint(W / 2 + 121 * np.cos(a)), np.rint(H / 2 + 121 * np.sin(a))], 1)
    elif kind == "line":
        t = np.arange(W)
        p = np.stack([t, np.rint(t * 0.6)], 1)
    else:
        x, y = np.meshgrid(np.arange(2, W, 7), np.arange(1, H, 5))
        p = np.stack([x.ravel(), y.ravel()], 1)
    return np.ascontiguousarray(np.unique(p.astype(np.int32), axis=0)[::-1])


KINDS = ("uniform", "sparse", "dense", "clustered", "circle", "line", "lattice")


def _counts(ctx):
    out = (ctypes.c_int64 * 3)()
    _capi.check(_capi.load().idl_selftest_counts(ctx.handle, out, 3))
    return tuple(out)


@pytest.mark.parametrize("kind", KINDS)
def test_profiled_run(kind):
    seeds = _seeds(kind)
    s = oracle.sort_seeds(seeds, W, H)
    _, want_passes = oracle.voronoi("reference", W + 2 * P, H + 2 * P, s + P)
    o_tris, o_grid, _ = oracle.triangulate(W, H, s, P)
    ctx = _capi.Context(0)
    ctx.set_profiling(True)
    grid = np.empty((H, W, 3), np.int32)
    n = ctypes.c_int64()
    _capi.check(_capi.load().idl_triangulate(ctx.handle, W, H, seeds.ctypes.data, len(seeds), None, P,
                                             _capi.MODE_REFERENCE, grid.ctypes.data, ctypes.byref(n), None, None))
    np.testing.assert_array_equal(grid, o_grid)
    p = ctx.last_profile()
    assert p["passes"] == want_passes and p["n_triangles"] == len(o_tris) == n.value
    direct = _counts(ctx)[0] == 1
    assert direct or kind == "circle"
    if direct:   # what the profile describes is the run that was asked for
        assert p["rounds"] == 2 and p["tiles"] == 0
        # column offsets out and in, labels out, and in again for the roots
        assert p["prop_bytes"] == 12 * (W + 2 * P) * (H + 2 * P)
    assert all(p[k] > 0 for k in ("seeds_ms", "propagate_ms", "detect_ms", "dedup_ms", "assign_ms"))
    ctx.close()


@pytest.mark.parametrize("order", ["given", "xy"])
@pytest.mark.parametrize("kind", KINDS)
def test_timed_first_insert(kind, order):
    """The same route, state and pass count as through the passes."""
    seeds = _seeds(kind)
    direct, passes = _capi.Context(0), _capi.Context(0)
    passes.set_schedule(0)
    got, want = (cu.Delaunay(W, H, len(seeds) + 1, P) for _ in range(2))
    got.use_workspace(direct)
    want.use_workspace(passes)
    t = []
    for obj in (got, want):
        tb = (ctypes.c_float * _capi.T_COUNT)()
        obj._call("idl_delaunay_insert_ordered", seeds.ctypes.data, len(seeds), None, int(order == "xy"),
                  ctypes.cast(tb, ctypes.c_void_p))
        t.append(list(tb))
    assert sum(_counts(direct)[:2]) == 1 and sum(_counts(passes)[:2]) == 0
    assert t[0][_capi.T_BFS_ITERS] == t[1][_capi.T_BFS_ITERS]
    assert t[0][_capi.T_BFS_MS] > 0
    np.testing.assert_array_equal(got.get_voronoi_grid(), want.get_voronoi_grid())
    np.testing.assert_array_equal(got.get_triangles(), want.get_triangles())
    del got, want
    direct.close()
    passes.close()
