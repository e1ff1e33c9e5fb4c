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
