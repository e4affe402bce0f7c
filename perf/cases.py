"""Workloads of this framework with their sizes, inputs, one pass of each and the tolerance of its results.

A skeletonization call takes a label volume to packed skeletons: vertices, edges and radii of every object. Its result
is discrete (paths through voxels, ties decided by float32 distances that every schedule reaches), so results are
compared exactly. The volumes are synthetic ones of the benchmark's kinds (random-walk tubes, dense Voronoi cells cut by
tubes, cells with nuclei), drawn on the GPU from the seed.
"""
import ctypes
import math

import numpy as np
import torch

import brook_b200
from brook_b200 import _native, device_post

# the benchmark's TEASAR parameters and dust threshold (bench.py)
TEASAR = dict(scale=1.5, const=300, pdrf_scale=100000, pdrf_exponent=4)
DUST = 100
DTYPES = {"uint8": (torch.uint8, torch.uint8), "uint16": (torch.int16, torch.uint16),
          "uint32": (torch.int32, torch.uint32), "uint64": (torch.int64, torch.uint64)}
BYTES = {"uint8": 1, "uint16": 2, "uint32": 4, "uint64": 8}


def _case(call, kind, shape, objects, dtype, spacing, const=300.0, order="F", memory="device", **more):
    x, y, z = shape
    ax, ay, az = spacing
    return dict(call=call, kind=kind, x=x, y=y, z=z, objects=objects, dtype=dtype, ax=float(ax), ay=float(ay),
                az=float(az), const=float(const), order=order, memory=memory, **more)


def listed():
    return [
        # the smallest request of a service: a cut-out of a few objects, where launches and waits are all there is
        dict(name="request 48", **_case("skeletonize", "tubes", (48, 48, 40), 5, "uint32", (16, 16, 40))),
        # a small volume of twenty tubes
        dict(name="tubes 128", **_case("skeletonize", "tubes", (128, 128, 128), 20, "uint32", (16, 16, 40))),
        # a ragged request as a torch program holds it: a C-ordered device tensor of uint64 labels, odd extents
        dict(name="request ragged", **_case("skeletonize", "tubes", (211, 97, 131), 10, "uint64", (16, 16, 40),
                                            order="C")),
        # an ordinary dense segmentation block
        dict(name="dense 256", **_case("skeletonize", "dense", (256, 256, 256), 80, "uint64", (8, 8, 40))),
        # the benchmark's block: a whole dense segmentation cut-out
        dict(name="dense 512", **_case("skeletonize", "dense", (512, 512, 512), 600, "uint64", (8, 8, 40))),
        # a NumPy program's call: C-ordered labels in ordinary host memory, odd extents
        dict(name="host dense", **_case("skeletonize", "dense", (253, 189, 161), 50, "uint16", (4, 4, 40), order="C",
                                        memory="host")),
        # a binary mask of one branched cell: a single object carries all the work
        dict(name="mask arbor", **_case("skeletonize", "arbor", (220, 201, 181), 1, "uint8", (1, 1, 1), const=10)),
        # compact cells with nuclei and cavities: hole filling, and the soma test of every cell
        dict(name="cells", **_case("skeletonize", "cells", (160, 144, 128), 27, "uint32", (1, 1, 1), const=10,
                                   fill_holes=True, soma=30.0)),
        # many volumes of uneven sizes in one call, the results left on the device
        dict(name="batch 16", **_case("batch", "tubes", (144, 128, 120), 30, "uint32", (4, 4, 4), count=16)),
        # the distance field alone, for programs that only want it
        dict(name="edt", **_case("edt", "dense", (320, 288, 255), 150, "uint32", (4, 4, 40))),
        # the components alone
        dict(name="components", **_case("components", "dense", (448, 416, 384), 400, "uint64", (8, 8, 40))),
        # canonical post-processing of a block's skeletons that are on the device
        dict(name="post", **_case("post", "dense", (256, 256, 256), 120, "uint32", (8, 8, 40))),
    ]


def _edges(rng, low, high, limit):
    """Three extents, each log-uniform in [low, high], with at most `limit` voxels."""
    while True:
        e = [int(round(math.exp(rng.uniform(math.log(low), math.log(high))))) for _ in range(3)]
        if e[0] * e[1] * e[2] <= limit:
            return e


def draw(rng):
    what = rng.choice(["tubes", "tubes", "dense", "dense", "dense", "host", "arbor", "cells", "batch", "edt", "components",
                       "post"])
    spacing = rng.choice([(1, 1, 1), (4, 4, 4), (4, 4, 40), (8, 8, 40), (16, 16, 40)])
    dtype = rng.choice(["uint8", "uint16", "uint32", "uint64"])
    order = rng.choice("FFC")
    if what == "tubes":  # service requests: edges 32-384, about one tube per 64^3 voxels
        e = _edges(rng, 32, 384, 1 << 24)
        return _case("skeletonize", "tubes", e, max(2, round(math.prod(e) / 64 ** 3)), dtype, (16, 16, 40), order=order)
    if what == "dense":
        e = _edges(rng, 96, 512, 100_000_000)
        n = min(250, max(4, math.prod(e) * 5 // 2 ** 20)) if dtype == "uint8" else max(4, math.prod(e) * 5 // 2 ** 20)
        return _case("skeletonize", "dense", e, n, dtype, rng.choice([(8, 8, 40), (16, 16, 40), (4, 4, 40)]), order=order)
    if what == "host":
        e = _edges(rng, 64, 320, 1 << 24)
        return _case("skeletonize", "dense", e, max(4, min(250, math.prod(e) * 7 // 2 ** 20)), dtype, (4, 4, 40),
                     order=order, memory="host")
    if what == "arbor":
        return _case("skeletonize", "arbor", _edges(rng, 96, 224, 8_000_000), 1, dtype, (1, 1, 1), const=10, order=order)
    if what == "cells":
        e = _edges(rng, 64, 176, 3_000_000)
        return _case("skeletonize", "cells", e, max(4, math.prod(e) // 100_000), dtype, (1, 1, 1), const=10, order=order,
                     fill_holes=rng.random() < 0.7, soma=30.0)
    if what == "batch":
        return _case("batch", "tubes", _edges(rng, 64, 160, 2_500_000), rng.randint(10, 40), "uint32", (4, 4, 4),
                     count=rng.randint(3, 16))
    if what == "post":
        e = _edges(rng, 128, 320, 17_000_000)
        return _case("post", "dense", e, max(8, math.prod(e) * 7 // 2 ** 20), "uint32", (8, 8, 40))
    e = _edges(rng, 64, 448, 64_000_000)
    n = max(4, math.prod(e) * 6 // 2 ** 20)
    return _case(what, "dense", e, min(250, n) if dtype == "uint8" else n, dtype, spacing)


# ------------------------------------------------------------------------------------------------------------ inputs

def _walks(rng, shape, starts, steps, sigma=0.2):
    """Random walks of unit steps reflected at the box, all at once: (walk, x, y, z) rows of their centres."""
    n = len(starts)
    p = np.array(starts, np.float64)
    h = rng.normal(size=(n, 3))
    h /= np.linalg.norm(h, axis=1, keepdims=True)
    hi = np.asarray(shape, np.float64) - 1
    rows = []
    for t in range(int(np.max(steps))):
        turn = rng.normal(scale=sigma, size=(n, 3))
        h = h + turn - h * np.sum(turn * h, axis=1, keepdims=True)
        h /= np.linalg.norm(h, axis=1, keepdims=True)
        p = p + h
        out = (p < 0) | (p > hi)
        h = np.where(out, -h, h)
        p = np.clip(p, 0, hi)
        live = np.flatnonzero(t < steps)
        rows.append(np.concatenate([live[:, None], np.rint(p[live])], axis=1))
    return np.concatenate(rows).astype(np.int64)


def _paint(volume, shape, rows, radius, value):
    """Balls of radius[w] around the rows' centres into the flat Fortran volume; the larger value wins."""
    sx, sy, sz = shape
    quarter = np.rint(np.asarray(radius) * 4).astype(np.int64)
    for q in np.unique(quarter):
        mine = rows[quarter[rows[:, 0]] == q]
        if not len(mine):
            continue
        r = q / 4.0
        g = np.arange(-math.ceil(r), math.ceil(r) + 1)
        ball = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
        ball = torch.from_numpy(ball[(ball ** 2).sum(1) <= r * r]).cuda()
        values = torch.from_numpy(np.asarray(value)[mine[:, 0]]).cuda()
        centres = torch.from_numpy(mine[:, 1:]).cuda()
        step = max(1, (1 << 24) // len(ball))
        for i in range(0, len(centres), step):
            at = centres[i:i + step, None, :] + ball[None]
            x, y, z = at[..., 0], at[..., 1], at[..., 2]
            keep = (x >= 0) & (x < sx) & (y >= 0) & (y < sy) & (z >= 0) & (z < sz)
            val = values[i:i + step, None].expand(keep.shape)[keep]
            volume.scatter_reduce_(0, (x + sx * (y + sy * z))[keep], val, "amax")


def _coordinates(flat, shape):
    sx, sy, _ = shape
    return torch.stack([flat % sx, (flat // sx) % sy, flat // (sx * sy)], dim=1).float()


def _nearest(flat, shape, seeds):
    """The nearest seed of each voxel (up to float32 rounding), and its distance."""
    points = torch.from_numpy(seeds).float().cuda()
    square = points.square().sum(1)
    owner = torch.empty(flat.numel(), dtype=torch.int64, device="cuda")
    near = torch.empty(flat.numel(), dtype=torch.float32, device="cuda")
    step = max(1, (1 << 29) // len(seeds))
    for i in range(0, flat.numel(), step):
        at = _coordinates(flat[i:i + step], shape)
        owner[i:i + step] = torch.addmm(square, at, points.T, alpha=-2).argmin(dim=1)
        near[i:i + step] = (at - points[owner[i:i + step]]).norm(dim=1)
    return owner, near


def _split(c3, joined=None):
    """Clears the voxels on a face between two different nonzero labels (modulo `joined`)."""
    cut = torch.zeros_like(c3, dtype=torch.bool)
    for axis in range(3):
        n = c3.shape[axis]
        a, b = c3.narrow(axis, 1, n - 1), c3.narrow(axis, 0, n - 1)
        differ = (a != 0) & (b != 0) & ((a != b) if joined is None else ((a - 1) % joined != (b - 1) % joined))
        cut.narrow(axis, 1, n - 1).logical_or_(differ)
        cut.narrow(axis, 0, n - 1).logical_or_(differ)
    c3[cut] = 0


def _volume(case, seed):
    """The case's labels as an int64 tensor (z, y, x) on the GPU."""
    rng = np.random.default_rng(seed)
    shape, n = (case["x"], case["y"], case["z"]), case["objects"]
    flat = torch.zeros(math.prod(shape), dtype=torch.int64, device="cuda")
    box = np.asarray(shape) - 1
    if case["kind"] == "tubes":
        # each tube with a branch that leaves it half way
        starts, steps = rng.uniform(0, box, size=(n, 3)), rng.integers(200, 601, size=n)
        trunk = _walks(rng, shape, starts, steps)
        radius = rng.uniform(2.0, 6.0, size=n)
        fork = np.stack([trunk[trunk[:, 0] == w][steps[w] // 2, 1:] for w in range(n)])
        branch = _walks(rng, shape, fork, np.maximum(1, steps // 3))
        _paint(flat, shape, np.concatenate([trunk, branch]), radius, np.arange(1, n + 1))
    elif case["kind"] == "arbor":
        starts, radius = [box / 2.0], []
        for level, (count, length) in enumerate([(3, 300), (9, 200), (24, 120)]):
            starts = [starts[i] for i in rng.integers(0, len(starts), size=count)]
            rows = _walks(rng, shape, np.asarray(starts), np.full(count, length))
            _paint(flat, shape, rows, np.full(count, 6.0 - 1.5 * level), np.ones(count, np.int64))
            starts = list(rows[:, 1:].astype(np.float64))
    elif case["kind"] == "dense":
        seeds = rng.uniform(0, box, size=(n, 3))
        rows = _walks(rng, shape, seeds, rng.integers(200, 601, size=n))
        _paint(flat, shape, rows, rng.uniform(3.0, 10.0, size=n), np.ones(n, np.int64))
        where = torch.nonzero(flat).squeeze(1)
        flat[where] = _nearest(where, shape, seeds)[0] + 1
        _split(flat.view(shape[::-1]))
        top = {"uint8": 255, "uint16": 32767, "uint32": 2 ** 31 - 1, "uint64": 2 ** 63 - 1}[case["dtype"]]
        ids = np.unique(rng.integers(1, top, size=8 * n, dtype=np.int64, endpoint=True))
        ids = np.concatenate([[0], rng.permutation(ids)[:n]])
        flat = torch.from_numpy(np.resize(ids, n + 1)).cuda()[flat]
    else:  # cells: each with a nucleus of its own label, about half with an empty cavity beside it
        seeds = rng.uniform(4, box - 4, size=(n, 3))
        every = torch.arange(flat.numel(), device="cuda")
        owner, near = _nearest(every, shape, seeds)
        gap = np.linalg.norm(seeds[:, None] - seeds[None], axis=2) + np.eye(n) * 1e9
        radius = gap.min(1) * rng.uniform(0.35, 0.5, size=n) / 2
        way = rng.normal(size=(n, 3))
        centre = seeds + way / np.linalg.norm(way, axis=1, keepdims=True) * (1.9 * radius)[:, None]
        hollow = np.where(rng.random(n) < 0.5, 0.5 * radius, -1.0)
        r, c, k = (torch.from_numpy(v).float().cuda()[owner] for v in (radius, centre, hollow))
        inside = near <= r
        flat = owner + 1 + n * inside
        flat[((_coordinates(every, shape) - c).norm(dim=1) <= k) & ~inside] = 0
        _split(flat.view(shape[::-1]), n)
    return flat.view(shape[::-1])


def _held(case, labels):
    """The labels (x, y, z) as the caller's program holds them: the case's type, order and memory."""
    signed, dtype = DTYPES[case["dtype"]]
    t = labels.to(signed).view(dtype) if signed is not dtype else labels.to(dtype)
    if case["order"] == "C":
        t = t.view(signed).permute(2, 1, 0).contiguous().view(dtype)
    else:
        t = t.permute(2, 1, 0)
    if case["memory"] == "device":
        return t
    return t.view(signed).cpu().numpy().view(case["dtype"])


def _options(case):
    teasar = dict(TEASAR, const=case["const"])
    if case.get("soma"):
        teasar.update(soma_detection_threshold=case["soma"], soma_acceptance_threshold=1e6)
    return dict(teasar_params=teasar, anisotropy=(case["ax"], case["ay"], case["az"]), dust_threshold=DUST)


def _room(case):
    """Where a program keeps one result after the other: arrays of a size that every result of the case fits."""
    device = case["call"] in ("batch", "post")
    objects, volumes = case["objects"] * case.get("count", 1), case.get("count", 1)
    skeletons, vertices = 4 * objects + 64, 1500 * objects + 16384

    def points(shape, dtype):
        return torch.zeros(shape, dtype=dtype, device="cuda") if device else \
            np.zeros(shape, {torch.int32: "uint32"}.get(dtype, "float32"))

    room = dict(labels=np.zeros(skeletons, np.int64), v_off=np.zeros(skeletons + 1, np.int64),
                e_off=np.zeros(skeletons + 1, np.int64), vertices=points((vertices, 3), torch.float32),
                edges=points((vertices, 2), torch.int32), radii=points((vertices,), torch.float32))
    if case["call"] == "batch":
        room.update(sample=np.zeros(skeletons, np.int64), s_off=np.zeros(volumes + 1, np.int64))
    return room


def prepare(case, seed):
    state = dict(case=case, options=_options(case))
    if case["call"] == "components":
        state["room"] = dict(mapping=np.zeros(64 * case["objects"] + 4096, np.int64),
                             roots=np.zeros(64 * case["objects"] + 4096, np.int64))
    elif case["call"] != "edt":
        state["room"] = _room(case)
    if case["call"] == "batch":
        rng = np.random.default_rng(seed)
        state["samples"] = []
        for i in range(case["count"]):  # extents from half to one and a half times the case's
            scale = np.exp(rng.uniform(np.log(0.5), np.log(1.5), size=3))
            x, y, z = (max(16, int(round(case[a] * s))) for a, s in zip("xyz", scale))
            n = max(1, int(case["objects"] * np.prod(scale)))
            one = dict(case, x=x, y=y, z=z, objects=n)
            state["samples"].append(_held(one, _volume(one, seed * 64 + i)))
        return state
    state["labels"] = _held(case, _volume(case, seed))
    if case["call"] == "skeletonize":
        state["options"]["fill_holes"] = case.get("fill_holes", False)
    elif case["call"] == "post":
        state["skeletons"] = brook_b200.skeletonize(state.pop("labels"), output="packed_device", **state["options"])
    return state


# ---------------------------------------------------------------------------------------------------------- one pass

def _kept(room, **arrays):
    """The results in the program's own arrays."""
    for name, a in arrays.items():
        if len(a):
            room[name][:len(a)] = _signed(a) if isinstance(a, torch.Tensor) else a
    return room


def _packed(room, p, **more):
    return _kept(room, labels=p.labels, v_off=p.v_off, e_off=p.e_off, vertices=p.vertices, edges=p.edges, radii=p.radii,
                 **more)


def _signed(t):
    return t.view({torch.uint16: torch.int16, torch.uint32: torch.int32}.get(t.dtype, t.dtype))


def run(state):
    case, options = state["case"], state["options"]
    if case["call"] == "skeletonize":
        return _packed(state["room"], brook_b200.skeletonize(state["labels"], output="packed", **options))
    if case["call"] == "batch":
        got = brook_b200.skeletonize_batch(state["samples"], **options)
        return _packed(state["room"], got.packed, sample=got.sample, s_off=got.s_off)
    if case["call"] == "post":
        return _packed(state["room"], device_post.postprocess(state["skeletons"], 1500, 3500))
    # the C interface's calls for the components and the distance field
    lib, context = _native.load(), _native.context(0)
    labels = state["labels"]
    _native.check(lib.brook_context_wait_stream(context, torch.cuda.current_stream().cuda_stream or 1))
    volume = _native.device_volume(labels.data_ptr(), tuple(labels.shape),
                                   [s * labels.element_size() for s in labels.stride()], case["dtype"])
    if case["call"] == "edt":
        field = ctypes.c_void_p()
        spacing = (ctypes.c_float * 3)(case["ax"], case["ay"], case["az"])
        _native.check(lib.brook_edt(context, ctypes.byref(volume), spacing, 0, ctypes.byref(field)))
        return _native.array_tensor(field)
    found, ids = ctypes.c_void_p(), ctypes.c_void_p()
    _native.check(lib.brook_connected_components(context, ctypes.byref(volume), ctypes.byref(found)))
    view, count = _native.Volume(), ctypes.c_size_t()
    mapping, roots = ctypes.POINTER(ctypes.c_int64)(), ctypes.POINTER(ctypes.c_int64)()
    _native.check(lib.brook_components_view(found, ctypes.byref(view), ctypes.byref(mapping), ctypes.byref(roots),
                                            ctypes.byref(count)))
    _native.check(lib.brook_components_labels(found, ctypes.byref(ids)))
    k = count.value
    room = _kept(state["room"], mapping=np.ctypeslib.as_array(mapping, shape=(k + 1,)),
                 roots=np.ctypeslib.as_array(roots, shape=(k,)))
    out = dict(room, ids=_signed(_native.array_tensor(ids)))
    lib.brook_components_destroy(found)
    return out


def work(case):
    """The labels read once and the results written once (a skeleton of a few hundred vertices per object)."""
    n = case["x"] * case["y"] * case["z"]
    skeletons = case["objects"] * 280 * (12 + 8 + 4)
    if case["call"] == "edt":
        return dict(bytes=n * BYTES[case["dtype"]] + 4 * n, flops=0)
    if case["call"] == "components":
        return dict(bytes=n * BYTES[case["dtype"]] + 2 * n, flops=0)
    if case["call"] == "post":
        return dict(bytes=2 * skeletons, flops=0)
    return dict(bytes=case.get("count", 1) * (n * BYTES[case["dtype"]] + skeletons), flops=0)


def tolerance(case):
    # the distance field: float32 sums of spacings and one float32 rounding of each pass's squared distance
    return {"rel": 1e-6, "max": 4e-6} if case["call"] == "edt" else "exact"


def exact(case, seed):
    """The distance field in 64 bits: per axis the least of the squared distances over a voxel's run of equal labels and
    to the run's walls (the volume's ends are no walls). The other calls' results are discrete."""
    if case["call"] != "edt":
        return None
    labels = _volume(case, seed)  # (z, y, x)
    inf = float("inf")
    field = torch.full(labels.shape, inf, dtype=torch.float64, device="cuda")
    for axis, w in ((2, case["ax"]), (1, case["ay"]), (0, case["az"])):
        lab, f = labels.movedim(axis, 2), field.movedim(axis, 2)
        n = lab.shape[2]
        place = torch.arange(n, device="cuda")
        lab, f = lab.reshape(-1, n), f.reshape(-1, n).clone()
        apart = (place[:, None] - place[None, :]).double().mul_(w).square_()
        rows = max(1, (1 << 26) // (n * n))
        for i in range(0, len(lab), rows):
            a = lab[i:i + rows]
            turn = torch.ones_like(a, dtype=torch.bool)
            turn[:, 1:] = a[:, 1:] != a[:, :-1]
            run = turn.long().cumsum(1)
            first = torch.where(turn, place, 0).cummax(1).values
            stop = torch.ones_like(turn)
            stop[:, :-1] = turn[:, 1:]
            last = torch.where(stop, place, n).flip(1).cummin(1).values.flip(1)
            left = torch.where(first > 0, ((place - first + 1) * w).double().square(), inf)
            right = torch.where(last < n - 1, ((last + 1 - place) * w).double().square(), inf)
            best = torch.minimum(left, right)
            if axis != 2:
                cost = torch.where(run[:, :, None] == run[:, None, :], f[i:i + rows, None, :] + apart, inf)
                best = torch.minimum(best, cost.min(2).values)
            f[i:i + rows] = best
        shape = labels.movedim(axis, 2).shape
        field = f.view(shape).movedim(2, axis)
    return torch.where(labels == 0, 0.0, field.sqrt()).permute(2, 1, 0)
