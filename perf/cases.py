"""The work that a user of the registration cost path has it do, as cases.

A case is one call sequence through the public entry points: batched scoring
(`api.Engine.eval`) at the batch sizes of a simplex step and of a swarm
iteration, a whole swarm run (`Engine.pso`), the serving loop's mixed batch
(`serve.SlotEngine.eval`), the drop-in per-pose form (`eval(plain=True)`), the
images of the tracking window, and the plain filter operators.  Volumes,
cameras, filter chains and batch sizes are those of the benchmark, the
autotuner and the tests, and generic odd ones between them.

`prepare` makes a seeded scene: ellipsoid phantoms (soft tissue 200, cortex
1800, core 900, noise 20) on the device, radiographs from the ellipsoids'
analytic chords plus noise, start poses off the truth as a registration has
them.  `exact` restates the path in 64 bits over the same inputs.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api, serve
from autoscoper_gb300 import scene as S

DEV = "cuda" if torch.cuda.is_available() else "cpu"
STORAGE = {"u16": L.ASC_STORE_U16, "f16": L.ASC_STORE_F16, "bf16": L.ASC_STORE_BF16, "f32": L.ASC_STORE_F32}
SID, SOD = 1200.0, 600.0  # source to image, source to isocentre (mm)
BENCH = "160x96x96,256x128x128,200x200x120"  # width x height x depth of the benchmark's three bones
TRACK = "256x128x128,192x192x160"            # of the tracking benchmark's two


# ------------------------------------------------------------------ the cases
def _eval(name, **kw):
    c = dict(name=name, kind="eval", volumes="128x128x128", voxel=0.5, render=512, height=512, image=512, pitch=0.4,
             views=2, filters="sobel", items=4, spread=2.0, storage="u16", rad="u16", sad=False, background=False,
             full=False)
    c.update(kw)
    return c


def listed():
    return [
        # one Downhill Simplex step of one bone: reflection, expansion and two contractions; latency decides
        _eval("simplex_step_one_bone", spread=0.5),
        # the same step for the four small bones of a wrist at uneven voxels, 8-bit radiographs
        _eval("simplex_step_wrist", volumes="45x59x60,112x112x128,75x88x101,64x97x83", voxel=0.396, render=512,
              height=512, image=880, pitch=0.25, rad="u8", items=16, spread=0.5),
        # the same step at the benchmark's size with its four-filter chain
        _eval("simplex_step_chain", volumes=BENCH, voxel=0.4, render=1024, height=1024, image=1024, pitch=0.3,
              filters="chain", items=12, spread=0.5),
        # one swarm iteration, one bone, small images
        _eval("swarm_one_bone", items=100, spread=3.0),
        # one swarm iteration of the benchmark: 3 bones x 100 particles, 1024^2, four-filter chain (the largest)
        _eval("swarm_bench", volumes=BENCH, voxel=0.4, render=1024, height=1024, image=1024, pitch=0.3,
              filters="chain", items=300, spread=5.0),
        # SAD cost, FP16 voxels, ragged sizes, background mask, every pixel counted
        _eval("swarm_sad_ragged", volumes="101x133x87,77x64x143", voxel=0.45, render=771, height=645, image=771,
              pitch=0.31, filters="smooth", items=64, spread=3.0, storage="f16", sad=True, background=True, full=True),
        # the largest volume served, three views
        _eval("swarm_large_volume", volumes="320x320x320", voxel=0.3, render=1024, height=1024, image=1024, pitch=0.25,
              views=3, items=32, spread=3.0),
        # a frame of the tracking benchmark's swarm, from call to best pose: 64 particles, 5 iterations
        _eval("swarm_run_tracking", kind="pso", volumes=TRACK, voxel=0.4, render=1024, height=1024, image=1024,
              pitch=0.3, items=64, spread=3.0),
        # the serving loop's merged batch: three jobs of different cameras, sizes and chains in one launch
        dict(name="serving_mix", kind="slots", jobs="a", items=96, spread=3.0),
        # the drop-in form: one pose, operator by operator, as an existing Tracker calls them
        _eval("dropin_pose", kind="plain", volumes="160x96x96", voxel=0.4, render=1024, height=1024, image=1024,
              pitch=0.3, filters="chain", items=1, spread=1.0),
        # the tracking window: every view's merged DRR and one bone's images
        _eval("view_images", kind="images", volumes=TRACK, voxel=0.4, render=1024, height=1024, image=1024, pitch=0.3,
              filters="chain", items=1),
        # the four filters alone on one odd-sized image
        dict(name="filters_image", kind="filters", width=1021, height=983, gaussian=1.5, sharpen=1.0, window=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval"] * 6 + ["pso", "slots", "plain", "images", "filters"])
    if kind == "filters":
        return dict(kind=kind, width=_log(rng, 130, 1760), height=_log(rng, 130, 1760),
                    gaussian=round(rng.uniform(0.5, 3.0), 2), sharpen=round(rng.uniform(0.5, 2.0), 2),
                    window=rng.choice([3, 3, 5]))
    if kind == "slots":
        return dict(kind=kind, jobs=rng.choice(["a", "b"]), items=_log(rng, 6, 150), spread=3.0)
    nb = rng.choice([1, 1, 2, 3, 4])
    side = lambda: _log(rng, 45, 220 if nb == 1 else 150)  # noqa: E731
    render = _log(rng, 256, 1024)
    pitch = round(0.3 * 1024 / render * rng.uniform(0.8, 1.3), 3)
    c = _eval("", kind=kind, volumes=",".join("%dx%dx%d" % (side(), side(), side()) for _ in range(nb)),
              voxel=round(rng.uniform(0.3, 0.6), 3), render=render, height=min(1024, _log(rng, 256, 1024)),
              image=render if rng.random() < 0.6 else _log(rng, 256, 1760), pitch=pitch, views=rng.choice([1, 2, 2, 3]),
              filters=rng.choice(["none", "sobel", "sobel", "chain", "chain", "smooth"]), items=_log(rng, 1, 200),
              spread=round(rng.uniform(0.3, 5.0), 2), storage=rng.choice(["u16", "u16", "f16", "bf16", "f32"]),
              rad=rng.choice(["u16", "u16", "u8"]), sad=rng.random() < 0.25, background=rng.random() < 0.25,
              full=rng.random() < 0.3)
    del c["name"]
    c["pitch"] = round(c["pitch"] * c["render"] / c["image"], 4)
    if kind == "pso":  # a swarm compares costs: the well-conditioned ones
        c.update(items=_log(rng, 4, 48), filters="sobel", sad=False)
    if kind in ("plain", "images"):
        c["items"] = 1
    while c["items"] > 1 and max(_marched(c) / 2.5e10, _pixels(c) / 1e8) > 1.0 / (5 * nb if kind == "pso" else 1):
        c["items"] = (c["items"] + 1) // 2
    return c


def _marched(case):
    """Samples of a pass through the volumes' whole boxes, about."""
    px = case["pitch"] * case["image"] / case["render"] * SOD / SID
    per = [w * h * d * case["voxel"] ** 2 / (px * px) * 2 for w, h, d in _shapes(case)]
    return sum(per) / len(per) * case["items"] * case["views"]


def _pixels(case):
    """Pixels of the candidates' crops, about."""
    px = case["pitch"] * case["image"] / case["render"] * SOD / SID
    per = [min((w * h * d) ** (2 / 3) * 1.3 * (case["voxel"] / px) ** 2, case["render"] * case["height"])
           for w, h, d in _shapes(case)]
    return sum(per) / len(per) * case["items"] * case["views"]


# ------------------------------------------------------------------ frames (4 x 4, 64 bits)
def _rot(axis, deg):
    a = np.asarray(axis, float)
    n = np.linalg.norm(a)
    if n == 0:
        return np.eye(3)
    x, y, z = a / n
    K = np.array([[0, -z, y], [z, 0, -x], [-y, x, 0]])
    t = math.radians(deg)
    return np.eye(3) + math.sin(t) * K + (1 - math.cos(t)) * (K @ K)


def _frame(R, t):
    f = np.eye(4)
    f[:3, :3], f[:3, 3] = R, t
    return f


def _pose(v):  # xyz, then yaw about z, pitch about the new y, roll about the new x
    return _frame(_rot((0, 0, 1), v[3]) @ _rot((0, 1, 0), v[4]) @ _rot((1, 0, 0), v[5]), v[:3])


def _manip(v):  # xyz, then the rotation about v[3:6] by its length in degrees
    return _frame(_rot(v[3:6], float(np.linalg.norm(v[3:6]))), v[:3])


def _inv(f):
    return _frame(f[:3, :3].T, -f[:3, :3].T @ f[:3, 3])


def _columns(f):  # the package's 12 numbers: the rotation's columns, then the translation
    return np.concatenate([f[:3, :3].T.reshape(-1), f[:3, 3]])


# ------------------------------------------------------------------ a seeded scene, as plain arrays
def _shapes(case):
    return [tuple(int(x) for x in s.split("x")) for s in case["volumes"].split(",")]


def _semi(whd):
    return (40.0, 25.0, 25.0) if whd == (128, 128, 128) else tuple(0.31 * n for n in whd)


def _phantom(whd, gen):
    W, H, D = whd
    ax = [torch.arange(n, device=DEV, dtype=torch.float32) - (n - 1) / 2 for n in (W, H, D)]
    a, b, c = _semi(whd)

    def inside(s):
        return ((ax[0] / (a - s)) ** 2)[None, None, :] + ((ax[1] / (b - s)) ** 2)[None, :, None] + (
            (ax[2] / (c - s)) ** 2)[:, None, None] <= 1

    v = torch.full((D, H, W), 200.0, device=DEV)
    v[inside(0.0)] = 1800.0
    v[inside(3.0)] = 900.0
    v += 20.0 * torch.randn((D, H, W), generator=gen, device=DEV)
    return v.round_().clamp_(1, 65535).to(torch.int32)


def _scene(case, seed):
    """Cameras, volumes, radiographs, poses and settings of a case: numpy
    arrays and plain numbers, made from the seed alone."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed + 17)
    W = case["image"]
    H = max(1, round(case["image"] * case["height"] / case["render"]))
    f = SID / case["pitch"]
    cams = []
    for deg in (0.0, 90.0, 45.0)[:case["views"]]:
        eye = SOD * np.array([math.cos(math.radians(deg)), math.sin(math.radians(deg)), 0.0])
        back = eye / SOD
        right = np.cross((0.0, 0.0, 1.0), back)
        cams.append(_frame(np.stack([right, np.cross(back, right), back], 1), eye))
    shapes = _shapes(case)
    sizes = [np.array(s) * case["voxel"] for s in shapes]
    n = len(shapes)
    room = 0.62 * SOD / SID * H * case["pitch"]  # the bones share the height of the view
    bones, truth = [], []
    for i, (whd, mm) in enumerate(zip(shapes, sizes)):
        ypr = rng.uniform(-10, 10, 3)
        R = _pose([0, 0, 0, *ypr])[:3, :3]
        at = np.array([0.0, 0.0, 0.0 if n == 1 else room * (i / (n - 1) - 0.5)]) + rng.uniform(-2, 2, 3)
        t = at - R @ (mm * [0.5, 0.5, -0.5])
        truth.append(np.array([*t, *ypr]))
        bones.append(_phantom(whd, gen))
    vmax = [int(b.max()) for b in bones]
    cutoff = [float(np.float32((100 + 0.1 * (m - 100)) / 65535)) for m in vmax]
    # radiographs: the chords of each bone's shell and core along the ray of every texel
    ip = np.array([0.0, 0.0, 2.0 * W / f, 2.0 * H / f])
    u = ((torch.arange(W, device=DEV, dtype=torch.float64) + 0.5) / W - 0.5) * ip[2]
    v = (0.5 - (torch.arange(H, device=DEV, dtype=torch.float64) + 0.5) / H) * ip[3]
    rads = []
    for cam in cams:
        acc = torch.zeros((H, W), device=DEV, dtype=torch.float64)
        for whd, mm, pose in zip(shapes, sizes, truth):
            M = _inv(_pose(pose)) @ cam
            o = M[:3, 3] - mm * [0.5, 0.5, -0.5]
            ray = [float(M[i, 0]) * u[None, :] + float(M[i, 1]) * v[:, None] - 2.0 * float(M[i, 2]) for i in range(3)]
            length = (u[None, :] ** 2 + v[:, None] ** 2 + 4.0).sqrt()
            for shell, level in ((0.0, 1800.0), (3.0, 900.0 - 1800.0)):
                s = [(r - shell) * case["voxel"] for r in _semi(whd)]
                A = sum((ray[i] / s[i]) ** 2 for i in range(3))
                B = sum(ray[i] * (float(o[i]) / s[i] ** 2) for i in range(3))
                C = float(sum((o[i] / s[i]) ** 2 for i in range(3))) - 1.0
                acc += level / 65535 * 2.0 * ((B * B - A * C).clamp(min=0).sqrt() / A) * length
        img = 1.0 - acc.clamp(max=1.0) + 0.01 * torch.randn((H, W), generator=gen, device=DEV, dtype=torch.float64)
        top = 255 if case["rad"] == "u8" else 65535
        rads.append((img * top).round().clamp(0, top).to(torch.int32))
    bg = None
    if case["background"]:  # the field of view of an image intensifier: bright inside a circle
        r2 = (u[None, :] / ip[2]) ** 2 + (v[:, None] / ip[3]) ** 2
        bg = (0.9 - 1.2 * r2 + 0.02 * torch.rand((H, W), generator=gen, device=DEV, dtype=torch.float64)).float()
    start = [np.asarray(t + np.concatenate([rng.uniform(-2, 2, 3), rng.uniform(-2, 2, 3)]), np.float32) for t in truth]
    items = case["items"]
    which = np.sort(np.arange(items) % n).astype(np.int32)
    man = rng.uniform(-case["spread"], case["spread"], (items, 6))
    return dict(cams=cams, W=W, H=H, f=f, ip=ip, shapes=shapes, voxel=case["voxel"], bones=bones, cutoff=cutoff,
                step=float(np.float32(0.5 * case["voxel"])), rads=rads, bg=bg, pivots=[m * [-0.5, -0.5, 0.5] for m in sizes],
                start=start, which=which, man=man, render=case["render"], height=case["height"])


def _filters(name):
    if name == "smooth":
        return [S.Filter.gaussian(radius=2.0), S.Filter.sharpen(radius=1.3, contrast=2.0, threshold=0.01),
                S.Filter.sobel(scale=1.0, blend=0.3)]
    return S.config_filters(name)


def _host(t, dtype):
    return t.cpu().numpy().astype(dtype)


def _package_scene(case, sc):
    """The scene as the package's own description (what a trial file loads to)."""
    cams = [S.Camera(_columns(c), sc["W"], sc["H"], sc["W"] / 2.0, sc["H"] / 2.0, sc["f"], sc["f"]) for c in sc["cams"]]
    bg = None if sc["bg"] is None else sc["bg"].cpu().numpy()
    rads = [_host(r, np.uint8 if case["rad"] == "u8" else np.uint16) for r in sc["rads"]]
    views = [S.View(c, r, _filters(case["filters"]), _filters(case["filters"]), bg, 0.75 if case["background"] else -1.0)
             for c, r in zip(cams, rads)]
    vols = [S.Volume(_host(b, np.uint16), (sc["voxel"],) * 3) for b in sc["bones"]]
    ray = [[S.RayParams(sc["step"], 1.0, cut) for cut in sc["cutoff"]] for _ in cams]
    pivots = [_columns(_frame(np.eye(3), p)) for p in sc["pivots"]]
    return S.Scene(views, vols, ray, sc["render"], sc["height"], pivots, sc["start"], int(case["sad"]))


# ------------------------------------------------------------------ the serving mix
def _jobs(case):
    """The jobs of a merged batch, each as an `eval` case of its share of the candidates."""
    if case["jobs"] == "a":
        jobs = [dict(volumes="160x96x96,200x200x120", voxel=0.4, render=1024, height=1024, image=1024, pitch=0.3,
                     filters="chain"),
                dict(volumes="96x130x110", voxel=0.5, render=512, height=512, image=512, pitch=0.4, views=3),
                dict(volumes="64x64x64", voxel=0.6, render=300, height=256, image=300, pitch=0.5, views=1,
                     filters="smooth", rad="u8")]
    else:
        jobs = [dict(volumes="211x140x160", voxel=0.35, render=768, height=768, image=900, pitch=0.3),
                dict(volumes="72x90x65,80x64x99,66x101x77", voxel=0.5, render=640, height=512, image=640, pitch=0.35,
                     filters="chain")]
    n = case["items"] // len(jobs)
    return [_eval("", items=max(1, n), spread=case["spread"], **j) for j in jobs]


def _prepare_slots(case, seed):
    eng = serve.SlotEngine(n_views=8, n_bones=8, render=(1024, 1024), max_items=256)
    view = bone = 0
    keep, which, man = [], [], []
    for j, job in enumerate(_jobs(case)):
        sc = _scene(job, seed * 10 + j)
        ps = _package_scene(job, sc)
        vs = list(range(view, view + len(ps.views)))
        for slot, v in zip(vs, ps.views):
            eng.set_view(slot, v, api.DeviceImage(v.radiograph), sc["render"], sc["height"])
        for b, vol in enumerate(ps.volumes):
            dv = api.DeviceVolume(vol)
            keep.append(dv)
            eng.set_bone(bone + b, dv, ps.pivots[b], ps.poses[b], [row[b] for row in ps.ray], vs)
        which.append(sc["which"] + bone)
        man.append(sc["man"])
        view, bone = view + len(vs), bone + len(ps.volumes)
    return dict(kind="slots", eng=eng, keep=keep, which=np.concatenate(which).astype(np.int32), man=np.concatenate(man))


# ------------------------------------------------------------------ prepare, run
class _Image:
    """A torch image in the place of an api.DeviceArray."""

    def __init__(self, t):
        self.t, self.shape, self.ptr = t, tuple(t.shape), t.data_ptr()


def _test_image(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    H, W = case["height"], case["width"]
    y = torch.linspace(-1, 1, H, device=DEV)[:, None]
    x = torch.linspace(-1, 1, W, device=DEV)[None, :]
    img = 0.75 * (1 - (x / 0.7) ** 2 - (y / 0.8) ** 2).clamp(min=0) + 0.2 * (torch.sin(9 * x) * torch.cos(7 * y)).clamp(min=0)
    return (img + 0.01 * torch.randn((H, W), generator=gen, device=DEV)).clamp(0, 1).float().contiguous()


def _four(case):
    return [S.Filter.contrast_filter(alpha=2.5, beta=0.9, size=case["window"]),
            S.Filter.sharpen(radius=case["sharpen"], contrast=1.0), S.Filter.gaussian(radius=case["gaussian"]),
            S.Filter.sobel(scale=1.0, blend=0.0)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "filters":
        src = _test_image(case, seed)
        return dict(kind=kind, src=_Image(src), filters=_four(case), out=[_Image(torch.empty_like(src)) for _ in range(4)])
    if kind == "slots":
        return _prepare_slots(case, seed)
    sc = _scene(case, seed)
    ps = _package_scene(case, sc)
    n = len(sc["shapes"]) * case["items"] if kind == "pso" else max(case["items"], 8)
    eng = api.Engine(ps, max_items=n, coverage=L.ASC_SUM_FULL if case["full"] else L.ASC_SUM_TREE,
                     storage=STORAGE[case["storage"]])
    st = dict(kind=kind, eng=eng, which=sc["which"], man=sc["man"], items=case["items"], spread=case["spread"], seed=seed)
    if kind == "images":
        st["poses"] = np.stack([np.asarray(p, np.float64) for p in sc["start"]])
        shape = (sc["height"], sc["render"])
        st["drr"] = [torch.empty(shape, device=DEV) for _ in ps.views]
        st["images"] = [[torch.empty(shape, device=DEV) for _ in range(3)] for _ in ps.views]
    return st


def run(st):
    kind = st["kind"]
    if kind == "filters":
        src = st["src"]
        for f, out in zip(st["filters"], st["out"]):
            src = api.apply_filter(f, src, out)
        return [o.t for o in st["out"]]
    eng = st["eng"]
    if kind == "slots":
        return eng.eval(st["which"], st["man"])
    if kind == "pso":
        return eng.pso(n_particles=st["items"], n_iter=5, lo=-st["spread"], hi=st["spread"], seed=st["seed"])
    if kind == "images":
        p = st["poses"].ctypes.data_as(L.P(L.f64))
        first = st["poses"][0].ctypes.data_as(L.P(L.f64))
        for v, (drr, (rad, one, mask)) in enumerate(zip(st["drr"], st["images"])):
            L.call("asc_engine_render_drr", eng.handle, v, p, None, drr.data_ptr(), None)
            L.call("asc_engine_image_data", eng.handle, v, 0, first, rad.data_ptr(), one.data_ptr(), mask.data_ptr(),
                   None, None, None)
        return {"drr": st["drr"], "images": st["images"]}
    return eng.eval(st["which"], st["man"], plain=kind == "plain")


# ------------------------------------------------------------------ the least work
def work(case):
    """Each input once and each result once, as bytes; the operations of the
    samples inside the bones (a position, eight taps blended, a test and a
    sum: 32 each) and of the filters over the bones' shadows."""
    kind = case["kind"]
    if kind == "filters":
        n = case["width"] * case["height"]
        taps = sum(2 * (2 * int(3 * case[k]) + 1) for k in ("gaussian", "sharpen"))
        return {"bytes": 4.0 * n * 5, "flops": float(n * (2 * taps + case["window"] ** 2 + 30))}
    if kind == "slots":
        w = [work(j) for j in _jobs(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    shapes = _shapes(case)
    px = case["pitch"] * case["image"] / case["render"] * SOD / SID  # a render pixel at the isocentre (mm)
    samples = shadow = 0.0
    for whd in shapes:
        a, b, c = (r * case["voxel"] for r in _semi(whd))
        samples += 4 / 3 * math.pi * a * b * c / (px * px * 0.5 * case["voxel"])
        shadow += math.pi * (a * b * c) ** (2 / 3) / (px * px)
    per_pixel = {"none": 0, "sobel": 20, "chain": 110, "smooth": 110}[case["filters"]]
    poses = {"pso": 5 * len(shapes) * case["items"], "images": len(shapes) + 1}.get(kind, case["items"])
    flops = poses * case["views"] * (32 * samples + (2 * per_pixel + 30) * shadow) / len(shapes)
    bytes_ = sum(2.0 * w * h * d for w, h, d in shapes)
    bytes_ += case["views"] * case["image"] ** 2 * case["height"] / case["render"] * (1 if case["rad"] == "u8" else 2)
    bytes_ += case["items"] * 60.0
    if kind == "images":
        bytes_ += 16.0 * case["views"] * case["render"] * case["height"]
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------ the path in 64 bits
def _viewport(mv, cam, sc, mm):
    """The film-plane box of the projected volume within the image; None out of view."""
    corners = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (-1, 0)]) * mm
    q = corners @ mv[:3, :3].T + mv[:3, 3]
    p = -2.0 * q[:, :2] / q[:, 2:]
    lo, hi = np.minimum(1.0, p.min(0)), np.maximum(-1.0, p.max(0))
    a, b = -0.5 * sc["ip"][2:], 0.5 * sc["ip"][2:]
    if (lo > b).any() or (hi < a).any():
        return None
    lo, hi = np.maximum(lo, a), np.minimum(hi, b)
    return np.array([lo[0], lo[1], hi[0] - lo[0], hi[1] - lo[1]])


def _stored(vol, storage):
    v = vol.to(torch.float32)
    return (v.half() if storage == "f16" else v.bfloat16() if storage == "bf16" else v).to(torch.float64)


def _drr(sc, vol, mv, mm, vp, w, h, cutoff):
    """Samples of `step` mm from the far side of the box to the near one, those above the cutoff summed."""
    f64 = dict(device=DEV, dtype=torch.float64)
    D, H, W = vol.shape
    inv = 1.0 / np.asarray(mm, np.float32).astype(np.float64)
    inv = np.asarray(inv, np.float32).astype(np.float64)
    m = _inv(mv)[:3] * inv[:, None]
    m = m.astype(np.float32).astype(np.float64)
    u = (vp[0] + vp[2] * (torch.arange(w, **f64) / w))[None, :].expand(h, w).reshape(-1)
    v = (vp[1] + vp[3] * (torch.arange(h, **f64) / h))[:, None].expand(h, w).reshape(-1)
    s = sc["step"] / (u * u + v * v + 4.0).sqrt()
    d = [float(m[i, 0]) * u * s + float(m[i, 1]) * v * s - 2.0 * float(m[i, 2]) * s for i in range(3)]
    o = [float(x) for x in m[:, 3]]
    near = torch.full_like(u, -math.inf)
    far = torch.full_like(u, math.inf)
    for i, (lo, hi) in enumerate(((0.0, 1.0), (0.0, 1.0), (-1.0, 0.0))):
        a, b = (lo - o[i]) / d[i], (hi - o[i]) / d[i]
        near, far = torch.maximum(near, torch.minimum(a, b)), torch.minimum(far, torch.maximum(a, b))
    ray = (far > near).nonzero().reshape(-1)
    near, far, d = near.clamp(min=0.0)[ray], far[ray], [x[ray] for x in d]
    acc = torch.zeros_like(far)
    flat = vol.reshape(-1)
    count = int((far - near).max().ceil()) if ray.numel() else 0
    chunk = max(1, (1 << 25) // max(1, ray.numel()))
    thr = cutoff * 65535.0
    for k0 in range(0, count, chunk):
        t = far[:, None] - torch.arange(k0, min(count, k0 + chunk), **f64)[None, :]
        live = t > near[:, None]
        at, part = [], []
        for i, (n, sign, off) in enumerate(((W, 1.0, 0.0), (H, -1.0, 1.0), (D, -1.0, 0.0))):
            c = (off + sign * (o[i] + t * d[i][:, None])) * n - 0.5
            fl = c.floor()
            part.append(c - fl)
            at.append((fl.long().clamp(0, n - 1), (fl.long() + 1).clamp(0, n - 1)))
        val = 0.0
        for z in (0, 1):
            for y in (0, 1):
                row = (at[2][z] * H + at[1][y]) * W
                a, b = flat[row + at[0][0]], flat[row + at[0][1]]
                wy = part[1] if y else 1 - part[1]
                wz = part[2] if z else 1 - part[2]
                val = val + wz * wy * (a + part[0] * (b - a))
        acc += torch.where(live & (val > thr), val, 0.0).sum(1)
    img = torch.zeros_like(u)
    img[ray] = (acc * (sc["step"] / 65535.0)).clamp(0.0, 1.0)
    return img.reshape(h, w)


def _shift(x, dy, dx):
    """x moved so that out[y, x] = in[y + dy, x + dx], 0 outside."""
    h, w = x.shape
    out = torch.zeros_like(x)
    out[max(0, -dy):h - max(0, dy), max(0, -dx):w - max(0, dx)] = x[max(0, dy):h + min(0, dy), max(0, dx):w + min(0, dx)]
    return out


def _apply(f, x):
    if f.kind == S.CONTRAST:
        one, total, count = torch.ones_like(x), 0.0, 0.0
        for dy in range(-(f.size // 2), (f.size + 1) // 2):
            for dx in range(-(f.size // 2), (f.size + 1) // 2):
                total, count = total + _shift(x, dy, dx), count + _shift(one, dy, dx)
        mean = total / count
        return torch.where(mean > 0.01, mean ** (f.alpha - f.beta) * x ** f.beta, 0.0)
    if f.kind == S.SOBEL:
        p = torch.nn.functional.pad(x[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
        h, w = x.shape
        t = [[p[i:i + h, j:j + w] for j in range(3)] for i in range(3)]
        gx = t[0][2] + 2 * t[1][2] + t[2][2] - t[0][0] - 2 * t[1][0] - t[2][0]
        gy = t[0][0] + 2 * t[0][1] + t[0][2] - t[2][0] - 2 * t[2][1] - t[2][2]
        g = f.scale * (gx * gx + gy * gy).sqrt()
        return (g + 2 * f.blend * x if f.blend < 0.5 else 2 * (1 - f.blend) * g + x).clamp(0, 1)
    R = int(3 * f.radius)
    g = [2.71828 ** (-(i * i) / (2 * f.radius)) for i in range(-R, R + 1)]
    blur = sum(g[i + R] / sum(g) * _shift(x, 0, i) for i in range(-R, R + 1))
    blur = sum(g[i + R] / sum(g) * _shift(blur, i, 0) for i in range(-R, R + 1))
    if f.kind == S.GAUSSIAN:
        return blur.clamp(0, 1)
    return torch.where((x - blur).abs() > f.threshold, (x + f.contrast * (x - blur)).clamp(0, 1), x) if R else x


def _chain(case, x):
    for f in _filters(case["filters"]):
        x = _apply(f, x)
    return x


def _sample(sc, img, vp, w, h):
    """Bilinear read of an image over the viewport, and where it lies inside the image."""
    ip = sc["ip"].astype(np.float32).astype(np.float64)
    H, W = img.shape
    f64 = dict(device=DEV, dtype=torch.float64)
    sx = (vp[0] + vp[2] * (torch.arange(w, **f64) / w) - ip[0]) / ip[2] + 0.5
    sy = 0.5 - (vp[1] + vp[3] * (torch.arange(h, **f64) / h) - ip[1]) / ip[3]
    X, Y = sx * W - 0.5, sy * H - 0.5
    x0, y0 = X.floor(), Y.floor()
    ax, ay = (X - x0)[None, :], (Y - y0)[:, None]
    xi = [(x0.long() + i).clamp(0, W - 1) for i in (0, 1)]
    yi = [(y0.long() + i).clamp(0, H - 1) for i in (0, 1)]
    r = [img[yi[i]][:, xi[0]] * (1 - ax) + img[yi[i]][:, xi[1]] * ax for i in (0, 1)]
    inside = ((sx >= 0) & (sx <= 1))[None, :] & ((sy >= 0) & (sy <= 1))[:, None]
    return r[0] * (1 - ay) + r[1] * ay, inside


def _covered(n):
    """Which of n pixels the reference's multi-level sum adds: a level folds T =
    min(256, n) partials in halves and drops what an odd half leaves over."""
    at, keep = np.arange(n), np.ones(n, bool)
    while n > 1:
        T = min(n, 256)
        t, s = at % T, T // 2
        while s > 0:
            keep &= t < 2 * s
            t = np.where(t >= s, t - s, t)
            s //= 2
        at, n = at // T, -(-n // T)
    return torch.from_numpy(keep).to(DEV)


def _images(case, sc, vol, bone, cam, pose, whole=False):
    """Filtered radiograph, filtered DRR and mask of a bone in a view; None out of view."""
    mm = np.float32(np.float32(sc["voxel"]) * np.array(sc["shapes"][bone], np.float32)).astype(np.float64)
    mv = _inv(cam) @ pose
    if whole:
        vp = np.array([-sc["ip"][2] / 2, -sc["ip"][3] / 2, sc["ip"][2], sc["ip"][3]])
    else:
        inv = (1.0 / mm.astype(np.float32)).astype(np.float32).astype(np.float64)
        vp = _viewport(mv, cam, sc, 1.0 / inv)
        if vp is None:
            return None
    w, h = (sc["render"], sc["height"]) if whole else (int(vp[2] * sc["render"] / sc["ip"][2]), int(vp[3] * sc["height"] / sc["ip"][3]))
    if w == 0 or h == 0:
        return torch.zeros(0), torch.zeros(0), torch.zeros(0)
    vp = vp.astype(np.float32).astype(np.float64)
    raw = _drr(sc, vol, mv, mm, vp, w, h, sc["cutoff"][bone])
    drr = _chain(case, raw)
    return raw, drr, vp, w, h


def _rad(case, sc, view, vp, w, h):
    val, inside = _sample(sc, sc["rads"][view].to(torch.float64) / (255.0 if case["rad"] == "u8" else 65535.0), vp, w, h)
    rad = _chain(case, torch.where(inside, 1.0 - val, 0.0))
    if sc["bg"] is None:
        return rad, torch.ones_like(rad)
    val, inside = _sample(sc, sc["bg"].to(torch.float64), vp, w, h)
    return rad, (inside & (0.75 <= val)).to(torch.float64)


def _score(case, f, g, mask):
    n = f.numel()
    f, g, mask = f.reshape(-1), g.reshape(-1), mask.reshape(-1)
    if not case["full"]:
        keep = _covered(n)
        f, g, mask = f[keep], g[keep], mask[keep]
    F, G = f.sum() / mask.sum(), g.sum() / mask.sum()
    m = mask > 0.5
    a, b = f[m] - F, g[m] - G
    if case["sad"]:
        return float((a - b).abs().sum())
    den = float((a * a).sum() * (b * b).sum()) ** 0.5
    return 1.0 - (float((a * b).sum()) / den if den >= 1e-5 else 1e5)


def _candidate(case, sc, vols, item):
    bone = int(sc["which"][item])
    pivot = _frame(np.eye(3), sc["pivots"][bone])
    pose = _pose(sc["start"][bone].astype(np.float64)) @ _inv(pivot) @ _manip(sc["man"][item]) @ pivot
    out = []
    for view, cam in enumerate(sc["cams"]):
        r = _images(case, sc, vols[bone], bone, cam, pose)
        if r is None:
            out.append(9999.0)
            continue
        if r[0].numel() == 0:
            out.append(0.0 if case["sad"] else 1.0 - 1e5)
            continue
        _, drr, vp, w, h = r
        rad, bg = _rad(case, sc, view, vp, w, h)
        mask = bg * (drr != 0).to(torch.float64)
        out.append(_score(case, drr * mask, rad * mask, mask))
    return out


def _exact_eval(case, seed):
    sc = _scene(case, seed)
    vols = [_stored(b, case["storage"]) for b in sc["bones"]]
    per_view = np.array([_candidate(case, sc, vols, i) for i in range(case["items"])])
    cost = np.array([9999.0 if s < 0 else s for s in (float(sum(r)) for r in per_view)])
    return cost, per_view


def exact(case, seed):
    kind = case["kind"]
    if kind == "pso":
        return None
    if kind == "filters":
        x, out = _test_image(case, seed).double(), []
        for f in _four(case):
            x = _apply(f, x)
            out.append(x)
        return out
    if kind == "slots":
        jobs = _jobs(case)
        if sum(_marched(j) for j in jobs) > 1.2e10:
            return None
        return np.concatenate([_exact_eval(j, seed * 10 + i)[0] for i, j in enumerate(jobs)])
    if kind == "images":
        sc = _scene(case, seed)
        vols = [_stored(b, case["storage"]) for b in sc["bones"]]
        poses = [_pose(p.astype(np.float64)) for p in sc["start"]]
        drrs, images = [], []
        for view, cam in enumerate(sc["cams"]):
            each = [_images(case, sc, v, b, cam, p, whole=True) for b, (v, p) in enumerate(zip(vols, poses))]
            drrs.append(_chain(case, sum(e[0] for e in each).clamp(max=1.0)))
            _, drr, vp, w, h = each[0]
            rad, bg = _rad(case, sc, view, vp, w, h)
            mask = bg * (drr != 0).to(torch.float64)
            images.append([rad * mask, drr * mask, mask])
        return {"drr": drrs, "images": images}
    if _marched(case) > 1.2e10:
        return None
    return _exact_eval(case, seed)
