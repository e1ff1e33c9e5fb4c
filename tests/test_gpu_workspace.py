"""What a context's workspace reports and gives back."""
import ctypes

import numpy as np
import pytest

from tests.conftest import random_seeds

pytestmark = pytest.mark.gpu

cu = pytest.importorskip("integer_delauney_b200._delauney_cuda")
from integer_delauney_b200 import _capi  # noqa: E402


def _triangulate(ctx, W, H, n, seed=1):
    seeds = random_seeds(W, H, n, seed)
    grid = np.empty((H, W, 3), np.int32)
    count = ctypes.c_int64()
    _capi.check(_capi.load().idl_triangulate(ctx.handle, W, H, seeds.ctypes.data, n, None, 16, _capi.MODE_REFERENCE,
                                             grid.ctypes.data, ctypes.byref(count), None, None))
    return count.value


def test_vertex_triples_are_part_of_the_workspace():
    """Their buffer is counted with the others, and freed with the context."""
    ctx = _capi.Context(0)
    n = _triangulate(ctx, 400, 300, 5000)
    before = ctx.workspace_bytes()
    verts = np.empty((n, 3), np.int32)
    _capi.check(_capi.load().idl_get_triangle_vertices(ctx.handle, verts.ctypes.data, n))
    assert ctx.workspace_bytes() >= before + 12 * n
    ctx.close()


def test_calls_on_a_context_between_calls_of_an_object_that_borrows_it():
    """The triangles and counters an object left on the context are not taken
    for its own after the context has served another call, nor the other way
    round."""
    lib = _capi.load()
    ctx = _capi.Context(0)
    W, H = 300, 200
    seeds = random_seeds(W, H, 700, 3)
    ref = cu.Delaunay(W, H, 1000, 16)
    ref.insert_deferred(seeds)
    want_tris, want_grid = ref.get_triangles(), ref.finalise(as_arrays=True)[1]
    other = random_seeds(120, 90, 50, 4)
    vor = np.empty((90, 120, 2), np.int32)
    dims, counts = np.array([[120, 90]], np.int32), np.array([50], np.int64)

    def voronoi():
        _capi.check(lib.idl_voronoi(ctx.handle, 120, 90, other.ctypes.data, 50, _capi.MODE_REFERENCE, vor.ctypes.data,
                                    None))

    def batch():
        _capi.check(lib.idl_triangulate_batch(ctx.handle, 1, dims.ctypes.data, counts.ctypes.data, other.ctypes.data,
                                              16, _capi.MODE_REFERENCE, None, None, None))

    def labels():
        _capi.check(lib.idl_voronoi_batch(ctx.handle, 1, dims.ctypes.data, counts.ctypes.data, other.ctypes.data, 16,
                                          _capi.MODE_REFERENCE))

    for between in (voronoi, lambda: _triangulate(ctx, 120, 90, 50), batch, labels):
        d = cu.Delaunay(W, H, 1000, 16)
        d.use_workspace(ctx)
        d.insert_deferred(seeds)
        np.testing.assert_array_equal(d.get_triangles(), want_tris)
        between()
        np.testing.assert_array_equal(d.finalise(as_arrays=True)[1], want_grid)
        between()
        np.testing.assert_array_equal(d.get_triangles(), want_tris)
    # the rows on the context are the object's by now
    _triangulate(ctx, 120, 90, 50)
    d.get_triangles()
    rows = np.empty((200, 5), np.int32)
    assert lib.idl_get_triangles(ctx.handle, rows.ctypes.data, 200) == _capi.IDL_ERR_STATE
    del d
    ctx.close()


@pytest.mark.parametrize("side,n", [(64, 20), (256, 300), (1024, 10000), (2048, 50000)])
def test_estimates_cover_what_a_context_grows_to(side, n):
    """Besides the label planes and the staged output: what the server's
    budget and estimate_bytes charge for scratch."""
    from integer_delauney_b200.serving import estimate_bytes
    ctx = _capi.Context(0)
    _triangulate(ctx, side, side, n)
    wd = side + 32
    planes, staged = (wd + 31) // 32 * 32 * wd * 8, side * side * 12
    scratch = estimate_bytes(side, side, n, 16) - estimate_bytes(side, side, n, 16, workspace=False)
    assert ctx.workspace_bytes() - planes - staged <= scratch
    ctx.close()
