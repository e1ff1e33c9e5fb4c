"""Objects used from another stream than the one they were created on, with
other work in flight on the default stream: their counters are allocated and
cleared in the order of their own work."""
import numpy as np
import pytest

import oracle
from tests.conftest import random_seeds

pytestmark = pytest.mark.gpu

cu = pytest.importorskip("integer_delauney_b200._delauney_cuda")


@pytest.mark.parametrize("mode", ["reference", "exact"])
def test_insert_on_a_side_stream_while_the_default_stream_is_busy(mode):
    """Above 131 072 pixels a scan takes two launches, joined by a counter."""
    import torch
    W, H, n = 701, 503, 4000
    side = torch.cuda.Stream()
    # an object before, so that the pool's memory holds other values
    used = cu.Delaunay(W, H, n, 8, voronoi_mode=mode)
    used.insert_deferred(random_seeds(W, H, n, 3))
    used.get_triangles()
    del used
    a = torch.randn(4096, 4096, device="cuda")
    for seed in (1, 2, 3):
        seeds = random_seeds(W, H, n, seed)
        want, _ = oracle.voronoi(mode, W + 16, H + 16, oracle.sort_seeds(seeds, W, H) + 8)
        want = want[8:-8, 8:-8, 0]
        d = cu.Delaunay(W, H, n, 8, voronoi_mode=mode)
        torch.cuda.synchronize()
        for _ in range(24):   # some 50 ms of ordinary work
            a = torch.tanh(a @ a)
        with torch.cuda.stream(side):
            d.insert_deferred(seeds, order="xy")
            got = d.get_voronoi_grid()[..., 0]
            tris = len(d.get_triangles())
        torch.cuda.synchronize()
        np.testing.assert_array_equal(got, want)
        o_tris, _, _ = oracle.triangulate(W, H, oracle.sort_seeds(seeds, W, H), 8, mode)
        assert tris == len(o_tris)
