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
