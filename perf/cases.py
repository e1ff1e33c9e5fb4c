"""The calls whose speed this library is judged by, through its public entry points.

Each case is one call (or one short run of calls) a program makes: single
images from host and device seeds, batches, the incremental object and the
request server, over the sizes, densities and seed layouts of the repository's
configurations and tests.  ``listed()`` names fixed points of those ranges,
``draw()`` gives others.
"""
import ctypes
import math

import numpy as np
import torch

import integer_delauney_b200 as idl
from integer_delauney_b200 import _capi
from integer_delauney_b200.serving import Server
from integer_delauney_b200.workloads import clustered, fresh_points, uniform


def listed():
    return [
        # a thumbnail through the drop-in call: all latency and launches
        {"name": "tiny_host", "kind": "host", "width": 160, "height": 120, "seeds": 400, "layout": "uniform",
         "mode": "reference"},
        # the plain single-image configuration (512 x 512, 2 000 seeds)
        {"name": "small_host", "kind": "host", "width": 512, "height": 512, "seeds": 2000, "layout": "uniform",
         "mode": "reference"},
        # an ordinary photograph with an odd row length, host in and host out
        {"name": "photo_host", "kind": "host", "width": 1510, "height": 1018, "seeds": 30000, "layout": "uniform",
         "mode": "reference"},
        # the large single image on the device: the headline configuration
        {"name": "large_uniform", "kind": "device", "width": 4096, "height": 4096, "seeds": 200000,
         "layout": "uniform", "mode": "reference"},
        # the same image with clustered seeds: long fronts across empty space
        {"name": "large_clustered", "kind": "device", "width": 4096, "height": 4096, "seeds": 200000,
         "layout": "clustered", "mode": "reference"},
        # the same image in exact semantics
        {"name": "large_exact", "kind": "device", "width": 4096, "height": 4096, "seeds": 200000,
         "layout": "uniform", "mode": "exact"},
        # a ragged image at the low end of the served densities
        {"name": "sparse_ragged", "kind": "device", "width": 2731, "height": 1999, "seeds": 2800,
         "layout": "uniform", "mode": "reference"},
        # the diagram alone, in exact semantics
        {"name": "voronoi_exact", "kind": "voronoi", "width": 1021, "height": 767, "seeds": 6000,
         "layout": "uniform", "mode": "exact"},
        # the batched configuration: 512 images of uneven size in one call
        {"name": "batch_512", "kind": "batch", "images": 512, "side_lo": 64, "side_hi": 1024, "dens_lo": 0.001,
         "dens_hi": 0.02, "mode": "reference"},
        # an incremental session: a base set, then insert batches read back
        # through the device views after each
        {"name": "incremental_2k", "kind": "incremental", "width": 2048, "height": 2048, "base": 50000,
         "batches": 10, "per_batch": 1000, "hot_frac": 0.3, "hot": 256, "mode": "reference"},
        # adaptive refinement of a sampled scalar field
        {"name": "refine_1k", "kind": "refine", "width": 1024, "height": 1024, "base": 2000, "rounds": 6,
         "per_round": 500},
        # a burst of mixed requests to the server
        {"name": "serving_burst", "kind": "serving", "requests": 30, "side_lo": 128, "side_hi": 1024,
         "dens_lo": 0.0005, "dens_hi": 0.01, "insert_lo": 100, "insert_hi": 2000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "device", "device", "device", "voronoi", "batch", "incremental", "refine",
                       "serving"])
    if kind in ("host", "device", "voronoi"):
        w = _log(rng, 64, 2048 if kind == "voronoi" else 4096)
        h = _log(rng, 64, 2048 if kind == "voronoi" else 4096)
        n = max(3, int(math.exp(rng.uniform(math.log(0.0005), math.log(0.02))) * w * h))
        layout = rng.choice(["uniform", "uniform", "clustered"])
        mode = rng.choice(["reference", "reference", "exact"])
        return {"kind": kind, "width": w, "height": h, "seeds": n, "layout": layout, "mode": mode}
    if kind == "batch":
        return {"kind": kind, "images": _log(rng, 4, 300), "side_lo": 64, "side_hi": _log(rng, 128, 1024),
                "dens_lo": 0.001, "dens_hi": 0.02, "mode": rng.choice(["reference", "exact"])}
    if kind == "incremental":
        w, h = _log(rng, 256, 2048), _log(rng, 256, 2048)
        return {"kind": kind, "width": w, "height": h, "base": max(16, int(rng.uniform(0.002, 0.012) * w * h)),
                "batches": rng.randint(2, 10), "per_batch": max(4, int(rng.uniform(0.0001, 0.0005) * w * h)),
                "hot_frac": 0.3, "hot": min(w, h) // 4, "mode": rng.choice(["reference", "reference", "exact"])}
    if kind == "refine":
        w, h = _log(rng, 128, 1024), _log(rng, 128, 1024)
        return {"kind": kind, "width": w, "height": h, "base": max(16, int(0.002 * w * h)),
                "rounds": rng.randint(2, 6), "per_round": max(8, int(0.0005 * w * h))}
    return {"kind": kind, "requests": rng.randint(8, 30), "side_lo": 128, "side_hi": _log(rng, 256, 1024),
            "dens_lo": 0.0005, "dens_hi": 0.01, "insert_lo": 100, "insert_hi": 2000}


def _points(case, seed):
    make = clustered if case["layout"] == "clustered" else uniform
    return make(case["width"], case["height"], case["seeds"], seed=seed)


def _sided(case, rng):
    """Size and seed count of one image of a mixed set."""
    lo, hi = math.log(case["side_lo"]), math.log(case["side_hi"])
    w = int(round(math.exp(rng.uniform(lo, hi))))
    h = int(round(math.exp(rng.uniform(lo, hi))))
    return w, h, max(3, int(math.ceil(rng.uniform(case["dens_lo"], case["dens_hi"]) * w * h)))


def _rows_for(n):
    """Capacity for the triangles of n seeds (fewer than 2 n of them are expected)."""
    return 3 * n + 64


def _empty_rows(*shape):
    return np.full(shape, -1, dtype=np.int32)


def _key(width, points):
    return points[:, 1].astype(np.int64) * width + points[:, 0]


def _insert_batches(case, seed):
    """A uniform base set and batches of points new to it, a share of each in a hot square."""
    w, h = case["width"], case["height"]
    rng = np.random.default_rng(seed)
    base = uniform(w, h, case["base"], seed=seed)
    hot = case["hot"]
    hx, hy = int(rng.integers(0, w - hot + 1)), int(rng.integers(0, h - hot + 1))
    taken = np.sort(_key(w, base))
    batches = []
    for _ in range(case["batches"]):
        n_hot = int(case["hot_frac"] * case["per_batch"])
        inside = rng.integers(0, hot, size=(n_hot, 2)) + np.array([hx, hy])
        cand = np.unique(_key(w, inside))
        cand = cand[~np.isin(cand, taken)]
        got = np.stack([cand % w, cand // w], axis=1).astype(np.int32)
        taken = np.union1d(taken, cand)
        rest = fresh_points(w, h, case["per_batch"] - len(got), taken, int(rng.integers(1 << 31)))
        taken = np.union1d(taken, _key(w, rest))
        b = np.concatenate([got, rest])
        rng.shuffle(b)
        batches.append(np.ascontiguousarray(b))
    return base, batches


def _field(points, scale):
    """The sampled scalar field: smooth waves and one sharp front."""
    x, y = points[:, 0] / scale, points[:, 1] / scale
    return (np.sin(9.0 * x) * np.cos(7.0 * y) + np.tanh(40.0 * (x + 0.5 * y - 0.8))).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("host", "voronoi"):
        s["seeds"] = _points(case, seed)
        s["verts"] = _empty_rows(_rows_for(case["seeds"]), 3)
    elif kind == "device":
        s["ctx"] = _capi.context_for(torch.cuda.current_device())
        s["seeds"] = torch.from_numpy(_points(case, seed)).cuda()
        s["grid"] = torch.empty((case["height"], case["width"], 3), dtype=torch.int32, device="cuda")
        s["rows"] = torch.full((_rows_for(case["seeds"]), 5), -1, dtype=torch.int32, device="cuda")
    elif kind == "batch":
        sizes, points = np.random.default_rng(case["images"]), np.random.default_rng(seed)
        images = [_sided(case, sizes) for _ in range(case["images"])]
        images = [(w, h, uniform(w, h, n, seed=int(points.integers(1 << 31)))) for w, h, n in images]
        s["ctx"] = _capi.context_for(torch.cuda.current_device())
        s["dims"] = np.array([(w, h) for w, h, _ in images], dtype=np.int32)
        s["counts"] = np.array([len(p) for _, _, p in images], dtype=np.int64)
        s["seeds"] = torch.from_numpy(np.concatenate([p for _, _, p in images])).cuda()
        px = int((s["dims"][:, 0].astype(np.int64) * s["dims"][:, 1]).sum())
        s["grids"] = torch.empty((px, 3), dtype=torch.int32, device="cuda")
    elif kind == "incremental":
        s["base"], s["batches"] = _insert_batches(case, seed)
        s["cap"] = len(s["base"]) + sum(len(b) for b in s["batches"])
        s["mesh"] = idl.Delaunay(case["width"], case["height"], s["cap"], voronoi_mode=case["mode"])
        s["verts"] = _empty_rows(len(s["batches"]), _rows_for(s["cap"]), 3)
    elif kind == "refine":
        s["base"] = uniform(case["width"], case["height"], case["base"], seed=seed)
        s["cap"] = case["base"] + case["rounds"] * case["per_round"]
        s["mesh"] = idl.Delaunay(case["width"], case["height"], s["cap"])
        s["verts"], s["seeds"] = _empty_rows(_rows_for(s["cap"]), 3), _empty_rows(s["cap"], 2)
    elif kind == "serving":
        sizes, points = np.random.default_rng(case["requests"]), np.random.default_rng(seed)
        requests, held, taken = [], [], {}
        for i in range(case["requests"]):
            if i < 3 or sizes.random() < 0.7:
                w, h, n = _sided(case, sizes)
                p = uniform(w, h, n, seed=int(points.integers(1 << 31)))
                held.append((i, w, h))
                taken[i] = np.sort(_key(w, p))
                requests.append(("new", w, h, p))
            else:
                at, w, h = held[int(sizes.integers(len(held)))]
                n = min(int(sizes.integers(case["insert_lo"], case["insert_hi"] + 1)), w * h // 20)
                p = fresh_points(w, h, n, taken[at], int(points.integers(1 << 31)))
                taken[at] = np.union1d(taken[at], _key(w, p))
                requests.append(("insert", at, p))
            of = i if requests[-1][0] == "new" else at
            s.setdefault("verts", []).append(_empty_rows(_rows_for(len(taken[of])), 3))
        s["requests"] = requests
        s["server"] = Server()
    else:
        raise ValueError(kind)
    return s


class _Rows:
    """(n, 5) int32 triangle rows a context holds on the device, for torch.as_tensor."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n, 5), "typestr": "<i4", "data": (ptr, False), "strides": None,
                                         "version": 3}


def _device_rows(lib, ctx, n):
    if n == 0:
        return torch.empty((0, 5), dtype=torch.int32, device="cuda")
    rows, count = ctypes.c_void_p(), ctypes.c_void_p()
    _capi.check(lib.idl_triangles_device(ctx.handle, ctypes.byref(rows), ctypes.byref(count)))
    return torch.as_tensor(_Rows(rows.value, n), device="cuda")


def run(state):
    case, kind = state["case"], state["kind"]
    if kind == "host":
        verts, grid = idl.triangulate(case["width"], case["height"], state["seeds"], as_arrays=True,
                                      voronoi_mode=case["mode"])
        state["verts"][:len(verts)] = verts
        return {"verts": state["verts"], "grid": grid}
    if kind == "voronoi":
        return idl.Voronoi().compute(case["width"], case["height"], state["seeds"], voronoi_mode=case["mode"])
    lib = _capi.load()
    if kind == "device":
        ctx, n = state["ctx"], ctypes.c_int64(0)
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        _capi.check(lib.idl_triangulate_device(
            ctx.handle, case["width"], case["height"], state["seeds"].data_ptr(), state["seeds"].shape[0],
            _capi.AUTO_BORDER_PADDING, _capi.mode_id(case["mode"]), state["grid"].data_ptr(), ctypes.byref(n)))
        state["rows"][:n.value].copy_(_device_rows(lib, ctx, n.value))
        return {"grid": state["grid"], "triangles": state["rows"], "count": n.value}
    if kind == "batch":
        ctx, tri_counts = state["ctx"], np.zeros(case["images"], dtype=np.int64)
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        _capi.check(lib.idl_triangulate_batch_device(
            ctx.handle, case["images"], state["dims"].ctypes.data, state["counts"].ctypes.data,
            state["seeds"].data_ptr(), _capi.AUTO_BORDER_PADDING, _capi.mode_id(case["mode"]),
            state["grids"].data_ptr(), tri_counts.ctypes.data))
        return {"grids": state["grids"], "counts": tri_counts}
    if kind == "incremental":
        mesh = state["mesh"]
        mesh.reset(case["width"], case["height"], state["cap"])
        mesh.insert_deferred(state["base"])
        for batch, rows in zip(state["batches"], state["verts"]):
            mesh.insert_deferred(batch)
            verts, triangle, owner, outside = mesh.finalise_device()
            rows[:len(verts)] = verts
        return {"verts": state["verts"], "triangle": triangle.to_torch(), "owner": owner.to_torch(),
                "outside": outside.to_torch()}
    if kind == "refine":
        mesh, scale = state["mesh"], max(case["width"], case["height"])
        mesh.reset(case["width"], case["height"], state["cap"])
        mesh.insert_deferred(state["base"], _field(state["base"], scale))
        for _ in range(case["rounds"]):
            points = mesh.select_midpoints(2.0, case["per_round"])
            if len(points):
                mesh.insert_deferred(points, _field(points, scale))
        verts, grid = mesh.finalise(as_arrays=True)
        points = mesh.get_seeds()
        state["verts"][:len(verts)], state["seeds"][:len(points)] = verts, points
        return {"verts": state["verts"], "grid": grid, "seeds": state["seeds"]}
    server, tickets = state["server"], []
    for r in state["requests"]:
        if r[0] == "new":
            tickets.append(server.submit_new(r[1], r[2], r[3], fetch=True))
        else:
            tickets.append(server.submit_insert(tickets[r[1]].diagram_id, r[2], fetch=True))
    results = [t.result() for t in tickets]
    for r, t in zip(state["requests"], tickets):
        if r[0] == "new":
            server.recycle(t.diagram_id)
    for rows, r in zip(state["verts"], results):
        rows[:len(r.verts)] = r.verts
    return [(rows, r.grid) for rows, r in zip(state["verts"], results)]


def work(case):
    """Seeds read once, grids and triangle vertices written once."""
    kind = case["kind"]

    def image(px, n):
        return 8 * n + 12 * px + 24 * n

    if kind in ("host", "device"):
        total = image(case["width"] * case["height"], case["seeds"])
    elif kind == "voronoi":
        total = 8 * case["seeds"] + 8 * case["width"] * case["height"]
    elif kind in ("batch", "serving"):
        ratio = math.log(case["side_hi"] / case["side_lo"])
        side = (case["side_hi"] - case["side_lo"]) / ratio if ratio else case["side_lo"]
        px = side * side
        n = px * (case["dens_lo"] + case["dens_hi"]) / 2
        total = image(px, n) * (case["images"] if kind == "batch" else case["requests"])
    elif kind == "incremental":
        px, n = case["width"] * case["height"], case["base"] + case["batches"] * case["per_batch"]
        total = 8 * n + case["batches"] * (9 * px + 24 * n)
    else:
        total = image(case["width"] * case["height"], case["base"] + case["rounds"] * case["per_round"])
    return {"bytes": float(total), "flops": 0.0}


def exact(case, seed):
    """Where the result is a plain minimum: nearest seed, ties to the higher (x, y) rank."""
    if case["kind"] != "voronoi" or case["mode"] != "exact":
        return None
    w, h = case["width"], case["height"]
    p = _points(case, seed)
    p = p[np.lexsort((p[:, 1], p[:, 0]))].astype(np.int64)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = len(p)
    far = np.int64(1) << 60
    # each cell's best key d2 * n + (n - 1 - id) within its column, then over its row
    col = torch.full((w, h), int(far), dtype=torch.int64, device=dev)
    ys = torch.arange(h, dtype=torch.int64, device=dev)
    cut = np.searchsorted(p[:, 0], np.arange(w + 1))
    q = torch.from_numpy(p).to(dev)
    for x in range(w):
        a, b = int(cut[x]), int(cut[x + 1])
        if b > a:
            ids = torch.arange(a, b, dtype=torch.int64, device=dev)
            d = (ys[:, None] - q[None, a:b, 1]) ** 2
            col[x] = (d * n + (n - 1 - ids)[None, :]).amin(1)
    xs = torch.arange(w, dtype=torch.int64, device=dev)
    dx = (xs[:, None] - xs[None, :]) ** 2 * n
    out = torch.empty((h, w, 2), dtype=torch.int64, device=dev)
    for y in range(h):
        best = (col[None, :, y] + dx).amin(1)
        out[y, :, 0] = n - 1 - best % n
        out[y, :, 1] = best // n
    return out.cpu().numpy()
