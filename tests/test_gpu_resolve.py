"""The reference fixed point read off the exact diagram (resolve.cu) against
the oracle's iteration, bit for bit and pass count for pass count, on layouts
that leave cut-off cells: thin wedges (circles, dense discs, clusters), ties
(lattices, lines) and the edges of its tiles (128 columns, 16 rows, the 96-cell
window)."""
import ctypes

import numpy as np
import pytest

import oracle
from tests.conftest import clustered_seeds, random_seeds

pytestmark = pytest.mark.gpu

cu = pytest.importorskip("integer_delauney_b200._delauney_cuda")
from integer_delauney_b200 import _capi  # noqa: E402


def _layout(kind, W, H, seed):
    rng = np.random.default_rng(seed)
    if kind == "uniform":
        return random_seeds(W, H, max(3, W * H // 60), seed)
    if kind == "sparse":
        return random_seeds(W, H, max(3, W * H // 2500), seed)
    if kind == "dense":
        return random_seeds(W, H, max(3, W * H // 3), seed)
    if kind == "clustered":
        return clustered_seeds(W, H, max(3, W * H // 150), seed=seed, blobs=5, sigma=7.0)
    if kind == "lattice":
        step = int(rng.integers(3, 17))
        X, Y = np.meshgrid(np.arange(seed % 3, W, step), np.arange(seed % 2, H, step + seed % 4))
        p = np.stack([X.ravel(), Y.ravel()], 1)
    elif kind == "line":
        t = np.arange(0, max(W, H), 1 + seed % 3)
        p = np.stack([t, (t * (0.4 + 0.3 * seed)).astype(int)], 1)
        p = p[(p[:, 0] < W) & (p[:, 1] < H)]
    elif kind == "circle":
        a = np.linspace(0, 2 * np.pi, 40 + 23 * seed, endpoint=False)
        r = min(W, H) * 0.35
        p = np.stack([np.rint(W / 2 + r * np.cos(a)), np.rint(H / 2 + r * np.sin(a))], 1).astype(int)
    else:   # a solid disc beside a few far seeds
        X, Y = np.meshgrid(np.arange(W), np.arange(H))
        m = (X - W // 3) ** 2 + (Y - H // 2) ** 2 < (6 + 3 * seed) ** 2
        p = np.concatenate([np.stack([X[m], Y[m]], 1), random_seeds(W, H, 4, seed)])
    p = np.unique(p.astype(np.int32), axis=0)
    rng.shuffle(p)
    return np.ascontiguousarray(p)


@pytest.fixture
def ctx():
    c = _capi.Context(0)   # the default schedule
    yield c
    c.close()


def _voronoi(ctx, W, H, seeds):
    got = np.empty((H, W, 2), np.int32)
    passes = ctypes.c_int64(0)
    _capi.check(_capi.load().idl_voronoi(ctx.handle, W, H, seeds.ctypes.data, len(seeds), _capi.MODE_REFERENCE,
                                         got.ctypes.data, ctypes.byref(passes)))
    return got, passes.value


@pytest.mark.parametrize("W,H", [(1, 1), (1, 40), (128, 16), (129, 17), (127, 131), (260, 97), (417, 301)])
@pytest.mark.parametrize("kind", ["uniform", "sparse", "dense", "clustered", "lattice", "line", "circle", "disc"])
def test_fixed_point_and_passes(ctx, kind, W, H):
    for seed in (1, 2, 3):
        if W * H < 2000:
            if kind != "uniform":
                pytest.skip("too small for this layout")
            seeds = random_seeds(W, H, min(3, W * H), seed)
        else:
            seeds = _layout(kind, W, H, seed)
        want, want_passes = oracle.voronoi("reference", W, H, oracle.sort_seeds(seeds, W, H))
        got, passes = _voronoi(ctx, W, H, seeds)
        np.testing.assert_array_equal(got, want, err_msg=f"{kind} {W}x{H} seed {seed}")
        assert passes == want_passes, f"{kind} {W}x{H} seed {seed}"


def test_batch_labels_equal_single_images(ctx):
    """The atlas form: images of mixed layouts beside each other, image sides
    off every tile boundary, each equal to its own single-image diagram; then
    the same batch through the passes."""
    images = []
    for i, (kind, W, H) in enumerate([("circle", 131, 97), ("uniform", 64, 200), ("lattice", 97, 61),
                                      ("clustered", 180, 141), ("disc", 90, 120), ("sparse", 211, 57),
                                      ("line", 65, 129), ("uniform", 1, 1), ("dense", 33, 47)]):
        images.append((W, H, _layout(kind, W, H, 1 + i % 3) if W > 1 else np.zeros((1, 2), np.int32)))
    dims = np.array([(w, h) for w, h, _ in images], np.int32)
    counts = np.array([len(s) for _, _, s in images], np.int64)
    seeds = np.ascontiguousarray(np.concatenate([s for _, _, s in images]).astype(np.int32))
    lib = _capi.load()
    for schedule in (None, 3):
        if schedule is not None:
            ctx.set_schedule(schedule)
        grids = np.empty((int((dims[:, 0].astype(int) * dims[:, 1]).sum()), 3), np.int32)
        _capi.check(lib.idl_triangulate_batch(ctx.handle, len(images), dims.ctypes.data, counts.ctypes.data,
                                              seeds.ctypes.data, 8, _capi.MODE_REFERENCE, grids.ctypes.data, None,
                                              None))
        at = 0
        for w, h, s in images:
            _, want, _ = oracle.triangulate(w, h, oracle.sort_seeds(s, w, h), 8, "reference")
            np.testing.assert_array_equal(grids[at:at + w * h].reshape(h, w, 3), want, err_msg=f"{w}x{h} {schedule}")
            at += w * h


@pytest.mark.parametrize("W,H,n", [(31, 3, 5), (32, 65, 40), (33, 64, 33), (257, 5, 700), (528, 2, 3), (529, 4, 1500),
                                   (1025, 3, 9), (2113, 2, 2000), (4230, 3, 6000), (27001, 1, 20000),
                                   (32767, 1, 9000)])
def test_exact_rows(W, H, n):
    """The row pass at its interval (32, 256, 1024), warp share and list-length
    edges: few seeds, and more than half of the columns in the list."""
    seeds = random_seeds(W, H, n, 5)
    want, _ = oracle.voronoi("exact", W, H, oracle.sort_seeds(seeds, W, H))
    np.testing.assert_array_equal(cu.Voronoi().compute(W, H, seeds, voronoi_mode="exact"), want)


@pytest.mark.parametrize("W,H", [(129, 17), (127, 131), (417, 301)])
@pytest.mark.parametrize("kind", ["uniform", "sparse", "dense", "clustered", "lattice", "line", "circle", "disc"])
def test_first_insert_in_insertion_order(ctx, kind, W, H):
    """A first insert (ids, and so ties, in the order given) against the same
    insert through the passes, and a second insert on top of each."""
    for seed in (1, 2, 3):
        seeds = _layout(kind, W, H, seed)
        np.random.default_rng(seed).shuffle(seeds)
        taken = np.sort(seeds[:, 1].astype(np.int64) * W + seeds[:, 0])
        from integer_delauney_b200.workloads import fresh_points
        more = fresh_points(W, H, 5, taken, seed)
        ctx.set_schedule(0)
        got, want = (cu.Delaunay(W, H, len(seeds) + 5, 8) for _ in range(2))
        want.use_workspace(ctx)
        for batch in (seeds, more):
            if not len(batch):
                continue
            got.insert_deferred(batch)
            want.insert_deferred(batch)
            msg = f"{kind} {W}x{H} seed {seed}"
            np.testing.assert_array_equal(got.get_voronoi_grid(), want.get_voronoi_grid(), err_msg=msg)
            np.testing.assert_array_equal(got.get_triangles(), want.get_triangles(), err_msg=msg)


@pytest.mark.parametrize("W,H,kind", [(31, 15, "uniform"), (32, 16, "dense"), (33, 17, "lattice"), (64, 32, "uniform"),
                                      (65, 33, "dense"), (129, 47, "dense"), (260, 97, "line"), (417, 301, "circle"),
                                      (1601, 1537, "sparse")])
def test_detection_strips_and_raster_tiles(W, H, kind):
    """Triangles and their pixels at the edges of the detection's strips and
    the raster's tiles (32 x 16, from 1 184 of them up 64 x 32): strips with
    more vertex blocks than they keep, slivers across many tiles."""
    seeds = _layout(kind, W, H, 1)
    tris, grid, _ = oracle.triangulate(W, H, oracle.sort_seeds(seeds, W, H), 8, "reference")
    verts, got = cu.triangulate(W, H, seeds, border_padding=8, as_arrays=True)
    np.testing.assert_array_equal(verts, tris[:, 2:5])
    np.testing.assert_array_equal(got, grid)


@pytest.mark.parametrize("dx,dy", [(1, 0), (0, 1), (1, 1), (2, 1), (1, -2), (3, 5)])
def test_collinear_triangle(dx, dy):
    """A collinear triangle covers its line within the seed window, whatever
    the line's direction: a caller's grid in which one block sees three seeds
    of one line."""
    W, H = 201, 163
    x0, y0 = 100 - 10 * dx, 80 - 10 * dy
    seeds = np.array([(x0, y0), (x0 + 10 * dx, y0 + 10 * dy), (x0 + 18 * dx, y0 + 18 * dy), (199, 161)], np.int32)
    s = oracle.sort_seeds(seeds, W, H)
    vg = np.zeros((H, W, 2), np.int32)
    vg[..., 0] = 2
    vg[:70, :90, 0] = 0
    vg[:70, 90:, 0] = 1
    o_tris, o_grid, _ = oracle.triangulate(W, H, s, 0, "numpy", vgrid=vg)
    assert len(o_tris) == 1 and (o_grid[..., 2] == 0).sum() > 10
    tm, grid = cu.GridTriangulation().compute(vg, seeds, 0)
    assert len(tm) == 1
    np.testing.assert_array_equal(grid, o_grid)
