"""What happens where a workspace bound is met: the runs that are repeated
through the passes, with a larger hash table or with room for more triangles,
and the triangles drawn without tile lists.  The bounds are set small
(idl_selftest_limit), every result is compared with the oracle, and the counts
tell which way stage (a) went."""
import ctypes

import numpy as np
import pytest

import oracle
from tests.conftest import clustered_seeds, random_seeds

pytestmark = pytest.mark.gpu

cu = pytest.importorskip("integer_delauney_b200._delauney_cuda")
from integer_delauney_b200 import _capi  # noqa: E402

SUSPECTS, TRIANGLES, TABLE, TILE_LISTS, OPEN = range(5)
W, H, P = 301, 203, 8


def _seeds(kind):
    if kind == "uniform":
        return random_seeds(W, H, 900, 4)
    if kind == "clustered":
        return clustered_seeds(W, H, 900, seed=4, blobs=5, sigma=7.0)
    if kind == "circle":
        a = np.linspace(0, 2 * np.pi, 109, endpoint=False)
        p = np.stack([np.rint(W / 2 + 71 * np.cos(a)), np.rint(H / 2 + 71 * np.sin(a))], 1)
    else:
        x, y = np.meshgrid(np.arange(2, W, 7), np.arange(1, H, 5))
        p = np.stack([x.ravel(), y.ravel()], 1)
    return np.ascontiguousarray(np.unique(p.astype(np.int32), axis=0)[::-1])


KINDS = ("uniform", "clustered", "circle", "lattice")


@pytest.fixture
def ctx():
    c = _capi.Context(0)   # bounds and schedule at their defaults
    yield c
    c.close()


def _limit(ctx, which, limit):
    _capi.check(_capi.load().idl_selftest_limit(ctx.handle, which, limit))


def _counts(ctx):
    out = (ctypes.c_int64 * 3)()
    _capi.check(_capi.load().idl_selftest_counts(ctx.handle, out, 3))
    return tuple(out)


def _triangulate(ctx, seeds):
    grid = np.empty((H, W, 3), np.int32)
    n = ctypes.c_int64()
    lib = _capi.load()
    _capi.check(lib.idl_triangulate(ctx.handle, W, H, seeds.ctypes.data, len(seeds), None, P, _capi.MODE_REFERENCE,
                                    grid.ctypes.data, ctypes.byref(n), None, None))
    tris = np.empty((n.value, 5), np.int32)
    _capi.check(lib.idl_get_triangles(ctx.handle, tris.ctypes.data, n.value))
    return tris, grid


def _check_triangulate(ctx, kind):
    seeds = _seeds(kind)
    o_tris, o_grid, _ = oracle.triangulate(W, H, oracle.sort_seeds(seeds, W, H), P, "reference")
    tris, grid = _triangulate(ctx, seeds)
    np.testing.assert_array_equal(grid, o_grid, err_msg=kind)
    np.testing.assert_array_equal(tris, o_tris, err_msg=kind)


def test_default_bounds_are_not_met(ctx):
    for kind in KINDS:
        _check_triangulate(ctx, kind)
    assert _counts(ctx)[:2] == (len(KINDS), 0)


def test_too_few_suspects_run_the_passes(ctx):
    _limit(ctx, SUSPECTS, 1)
    lib = _capi.load()
    runs = 0
    for kind in ("uniform", "clustered"):   # each has several
        _check_triangulate(ctx, kind)
        runs += 1
        assert _counts(ctx)[:2] == (0, runs), kind
        seeds = _seeds(kind)
        s = oracle.sort_seeds(seeds, W, H)
        want, want_passes = oracle.voronoi("reference", W, H, s)
        got = np.empty((H, W, 2), np.int32)
        passes = ctypes.c_int64()
        _capi.check(lib.idl_voronoi(ctx.handle, W, H, seeds.ctypes.data, len(seeds), _capi.MODE_REFERENCE,
                                    got.ctypes.data, ctypes.byref(passes)))
        runs += 1
        np.testing.assert_array_equal(got, want, err_msg=kind)
        assert passes.value == want_passes
        assert _counts(ctx)[:2] == (0, runs), kind
        # first inserts, in the order given and in (x, y) order
        for order in ("given", "xy"):
            d, ref = (cu.Delaunay(W, H, len(seeds), P) for _ in range(2))
            d.use_workspace(ctx)
            for obj in (d, ref):
                if order == "xy":
                    obj.insert_deferred(seeds, order="xy")
                else:
                    obj.insert_deferred(seeds)
            runs += 1
            assert _counts(ctx)[:2] == (0, runs), (kind, order)
            np.testing.assert_array_equal(d.get_voronoi_grid(), ref.get_voronoi_grid(), err_msg=f"{kind} {order}")
            np.testing.assert_array_equal(d.get_triangles(), ref.get_triangles(), err_msg=f"{kind} {order}")
    # a batch, whole and labels only
    images = [_seeds(k) for k in KINDS]
    dims = np.array([(W, H)] * len(images), np.int32)
    counts = np.array([len(s) for s in images], np.int64)
    flat = np.ascontiguousarray(np.concatenate(images))
    grids = np.empty((len(images), H, W, 3), np.int32)
    _capi.check(lib.idl_triangulate_batch(ctx.handle, len(images), dims.ctypes.data, counts.ctypes.data,
                                          flat.ctypes.data, P, _capi.MODE_REFERENCE, grids.ctypes.data, None, None))
    runs += 1
    assert _counts(ctx)[:2] == (0, runs)
    _capi.check(lib.idl_voronoi_batch(ctx.handle, len(images), dims.ctypes.data, counts.ctypes.data,
                                      flat.ctypes.data, P, _capi.MODE_REFERENCE))
    runs += 1
    assert _counts(ctx)[:2] == (0, runs)
    for k, seeds in enumerate(images):
        s = oracle.sort_seeds(seeds, W, H)
        _, o_grid, _ = oracle.triangulate(W, H, s, P, "reference")
        np.testing.assert_array_equal(grids[k], o_grid, err_msg=KINDS[k])
        d = cu.Delaunay(W, H, len(seeds), P)
        _capi.check(lib.idl_delaunay_adopt(d._h, ctx.handle, k))
        np.testing.assert_array_equal(d.get_voronoi_grid()[..., 0], o_grid[..., 0], err_msg=KINDS[k])


@pytest.mark.parametrize("which,limit", [(TABLE, 256), (TRIANGLES, 1), (TRIANGLES, 100), (TILE_LISTS, 1),
                                         (TILE_LISTS, 500)])
def test_small_workspaces_give_the_same_triangles(ctx, which, limit):
    """Every layout has more triangles than the first table has slots and than
    the first drawing has room for, and more of them per tile than the lists."""
    _limit(ctx, which, limit)
    for kind in ("uniform", "clustered", "lattice"):
        _check_triangulate(ctx, kind)
    images = [_seeds(k) for k in KINDS]
    flat = np.ascontiguousarray(np.concatenate(images))
    dims = np.array([(W, H)] * len(images), np.int32)
    counts = np.array([len(s) for s in images], np.int64)
    grids = np.empty((len(images), H, W, 3), np.int32)
    _capi.check(_capi.load().idl_triangulate_batch(ctx.handle, len(images), dims.ctypes.data, counts.ctypes.data,
                                                   flat.ctypes.data, P, _capi.MODE_REFERENCE, grids.ctypes.data, None,
                                                   None))
    for k, seeds in enumerate(images):
        _, o_grid, _ = oracle.triangulate(W, H, oracle.sort_seeds(seeds, W, H), P, "reference")
        np.testing.assert_array_equal(grids[k], o_grid, err_msg=KINDS[k])


@pytest.mark.parametrize("radius", [40, 70])
def test_windows_decide_cells(ctx, radius):
    """Seeds on a circle leave cells near its centre, without a settled
    neighbour, to the 96-cell window; what matters to them reaches past the
    window of a wide circle, and the passes run."""
    lib = _capi.load()
    c = radius + 30
    for n in range(40, 400, 9):
        a = np.linspace(0, 2 * np.pi, n, endpoint=False)
        p = np.stack([np.rint(c + radius * np.cos(a)), np.rint(c + radius * np.sin(a))], 1).astype(np.int32)
        seeds = np.ascontiguousarray(np.unique(p, axis=0))
        side = 2 * c + 1
        want, _ = oracle.voronoi("reference", side, side, oracle.sort_seeds(seeds, side, side))
        got = np.empty((side, side, 2), np.int32)
        _capi.check(lib.idl_voronoi(ctx.handle, side, side, seeds.ctypes.data, len(seeds), _capi.MODE_REFERENCE,
                                    got.ctypes.data, None))
        np.testing.assert_array_equal(got, want, err_msg=str(n))
    direct, passes, windows = _counts(ctx)
    assert direct > 0
    if radius == 40:
        assert windows > 0 and passes == 0
    else:
        assert passes > 0


def test_too_many_windows_run_the_passes(ctx):
    """Circles that leave more than one cell to windows, with room for one."""
    lib = _capi.load()
    several = 0
    for n in range(40, 400, 9):
        a = np.linspace(0, 2 * np.pi, n, endpoint=False)
        p = np.stack([np.rint(70 + 40 * np.cos(a)), np.rint(70 + 40 * np.sin(a))], 1).astype(np.int32)
        seeds = np.ascontiguousarray(np.unique(p, axis=0))
        want, _ = oracle.voronoi("reference", 141, 141, oracle.sort_seeds(seeds, 141, 141))
        got = np.empty((141, 141, 2), np.int32)
        for limit in (0, 1):
            _limit(ctx, OPEN, limit)
            before = np.array(_counts(ctx))
            _capi.check(lib.idl_voronoi(ctx.handle, 141, 141, seeds.ctypes.data, len(seeds), _capi.MODE_REFERENCE,
                                        got.ctypes.data, None))
            np.testing.assert_array_equal(got, want, err_msg=f"{n} {limit}")
            direct, passes, windows = np.array(_counts(ctx)) - before
            if limit == 0:
                open_cells = windows
                assert passes == 0
            else:
                assert passes == (open_cells > 1) and windows == (open_cells if open_cells <= 1 else 0)
        several += open_cells > 1
    assert several > 0


@pytest.mark.parametrize("kind", ["lines", "circle"])
def test_more_suspects_than_warps(ctx, kind):
    """Tens of thousands of cells cut off: between slanted lines of seeds, all
    decided; in a wide circle, many of them without a settled neighbour."""
    W, H = 900, 800
    if kind == "lines":
        t = np.arange(W)
        p = np.concatenate([np.stack([t, np.rint(t * 0.37 + k * H / 6)], 1) for k in range(6)])
    else:
        a = np.linspace(0, 2 * np.pi, 8000, endpoint=False)
        p = np.stack([np.rint(W / 2 + 350 * np.cos(a)), np.rint(H / 2 + 350 * np.sin(a))], 1)
    p = p[(p[:, 0] >= 0) & (p[:, 0] < W) & (p[:, 1] >= 0) & (p[:, 1] < H)]
    seeds = np.ascontiguousarray(np.unique(p.astype(np.int32), axis=0))
    want, want_passes = oracle.voronoi("reference", W, H, oracle.sort_seeds(seeds, W, H))
    got = np.empty((H, W, 2), np.int32)
    passes = ctypes.c_int64()
    _capi.check(_capi.load().idl_voronoi(ctx.handle, W, H, seeds.ctypes.data, len(seeds), _capi.MODE_REFERENCE,
                                         got.ctypes.data, ctypes.byref(passes)))
    np.testing.assert_array_equal(got, want)
    assert passes.value == want_passes
    assert _counts(ctx)[:2] == ((1, 0) if kind == "lines" else (0, 1))
