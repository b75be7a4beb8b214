"""Performance cases of the rebin library, through its public entry points.

A case is one call that a user's program makes over and over: an interactive
frame (GaussianSplatRenderer.render, then gs3d_composite into a device
buffer), a batch of views (rebinBatch), the six stage entry points in order,
a PLY load, one forward and backward step of the cost model.  Scenes follow
the distributions of gs3d.scenes and are drawn on the GPU from the seed;
cameras are the orbit, random and close-up poses of the benchmark and tests.

  listed()            the named cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) inputs, context, resident scene and first frame
  run(state)          one pass; returns the library's device buffers
  work(case)          bytes and flops a pass cannot do without
  exact(case, seed)   the pass's computed numbers in 64 bits, plain torch
"""
import ctypes as C
import functools
import json
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "webgpu-3dgs_gb300") not in sys.path:
    sys.path.insert(0, str(ROOT / "webgpu-3dgs_gb300"))

from gs3d import GaussianSplatRenderer, RenderFrameInfo, Scene, _lib, learned, ply, scenes  # noqa: E402
from gs3d.renderer import DeviceSplats  # noqa: E402

SCHEDULES = {"row": _lib.SCHEDULE_ROW_MAJOR, "keys": _lib.SCHEDULE_KEY_COUNT,
             "learned": _lib.SCHEDULE_LEARNED}
MODELS = {(16, 16): "cost_mlp_c1.npz", (32, 32): "cost_mlp_c1_t32.npz",
          (64, 32): "cost_mlp_c1_t64x32.npz", (32, 64): "cost_mlp_c1_t32x64.npz"}
# the view sizes of a mixed batch, taken in turn
MIXED = [(640, 360), (1280, 720), (1920, 1080), (2560, 1440), (3840, 2160), (1000, 563)]


def _frame(name, scene, n, sh, w, h, radius, tw=16, th=16, batch=0, schedule="row"):
    return dict(name=name, kind="frame", scene=scene, n=n, sh=sh, w=w, h=h, radius=radius, tw=tw,
                th=th, raster_batch=batch, schedule=schedule)


def _batch(name, scene, n, sh, views, w, h, radius, tw, th, batch, schedule, graph, scenes_=1,
           mixed=False):
    return dict(name=name, kind="batch", scene=scene, n=n, sh=sh, views=views, w=w, h=h,
                radius=radius, tw=tw, th=th, raster_batch=batch, schedule=schedule, graph=graph,
                scenes=scenes_, mixed=mixed)


def listed():
    return [
        # a thumbnail or preview of a small scene: launches and latency count
        _frame("frame 20k 320x240", "small", 20_000, 0, 320, 240, 6.0),
        # the small benchmark scene, interactive, at the reference's settings
        _frame("frame 100k 720p", "small", 100_000, 0, 1280, 720, 6.0),
        # a mid-sized capture with low SH in a window of odd size
        _frame("frame 400k sh1 1000x563", "clusters", 400_000, 1, 1000, 563, 12.0),
        # a full capture, interactive, at the reference's 16x16 tiles
        _frame("frame 3m sh3 1080p", "clusters", 3_000_000, 3, 1920, 1080, 12.0),
        # opaque clusters beside dense translucent ones: skewed tile costs, so
        # the frame is drawn in key-count order
        _frame("frame mix 1.9m 1080p keys", "mix", 1_900_000, 0, 1920, 1080, 12.0,
               schedule="keys"),
        # a camera inside a dense scene of heavy-tailed scales, 4K: the most
        # references per splat
        _frame("frame skew 3m sh3 4k close", "skew", 3_000_000, 3, 3840, 2160, 4.0, 32, 32, 512),
        # the benchmark's throughput path: views of one scene in one launch
        # sequence, tuned, replayed as a graph
        _batch("batch8 3m sh3 1080p 64x32", "clusters", 3_000_000, 3, 8, 1920, 1080, 12.0, 64, 32,
               512, "keys", True),
        # several resident scenes, uneven view sizes up to 4K, tuned
        _batch("batch12 mixed 3 scenes 32x64", "clusters", 3_000_000, 3, 12, 0, 0, 12.0, 32, 64,
               512, "keys", True, 3, True),
        # many small views of a mid-sized scene (data generation), eager, in
        # the learned order
        _batch("batch16 200k sh2 640x360", "clusters", 200_000, 2, 16, 640, 360, 10.0, 32, 32, 256,
               "learned", False),
        # the reference's six stages called one by one
        dict(name="stages 150k sh2 800x600", kind="stages", scene="clusters", n=150_000, sh=2,
             w=800, h=600, radius=12.0, tw=16, th=16),
        # opening a trained scene: the whole call on the file's bytes
        dict(name="ply 300k sh3", kind="ply", n=300_000, sh=3, format="binary_little_endian"),
        # one step of training the cost model: forward and backward
        dict(name="cost model step 65536", kind="train", n=65_536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "batch", "batch", "batch", "stages", "ply",
                       "train"])
    if kind == "ply":
        return dict(kind="ply", n=_log(rng, 1_000, 300_000), sh=rng.choice([0, 1, 2, 3]),
                    format=rng.choice(["binary_little_endian", "binary_little_endian",
                                       "binary_big_endian"]))
    if kind == "train":
        return dict(kind="train", n=_log(rng, 500, 65_536))
    scene = rng.choice(["small", "clusters", "clusters", "mix", "skew"])
    sh = 0 if scene in ("small", "mix") else rng.choice([0, 1, 2, 3])
    radius = {"small": rng.uniform(4.0, 8.0), "clusters": rng.uniform(8.0, 16.0),
              "mix": rng.uniform(10.0, 14.0), "skew": rng.uniform(4.0, 34.0)}[scene]
    radius = round(radius, 3)
    if kind == "stages":
        w = _log(rng, 320, 1280)
        return dict(kind="stages", scene=scene, n=_log(rng, 10_000, 300_000), sh=sh, w=w,
                    h=max(200, int(w * rng.uniform(0.5, 0.8))), radius=radius, tw=16, th=16)
    tile = rng.choice([(16, 16), (16, 16), (32, 32), (8, 8), (64, 32), (32, 64)])
    sched = rng.choice(["row", "keys", "learned"] if tile in MODELS else ["row", "keys"])
    staged = rng.choice([128, 256, 512]) if tile != (16, 16) else 0
    if kind == "frame":
        w = _log(rng, 300, 2600)
        top = 1_000_000 if scene in ("skew", "mix") else 3_000_000
        return dict(kind="frame", scene=scene, n=_log(rng, 15_000, top), sh=sh, w=w,
                    h=max(200, int(w * rng.uniform(0.5, 0.8))), radius=radius, tw=tile[0],
                    th=tile[1], raster_batch=staged, schedule=sched)
    if tile == (8, 8):
        tile = (32, 32)
        sched = "keys"
    mixed = rng.random() < 0.4
    w = _log(rng, 320, 1920)
    return dict(kind="batch", scene=scene, n=_log(rng, 20_000, 800_000), sh=sh,
                views=rng.randint(2, 9), w=0 if mixed else w,
                h=0 if mixed else max(200, int(w * rng.uniform(0.5, 0.8))), radius=radius,
                tw=tile[0], th=tile[1], raster_batch=staged, schedule=sched,
                graph=rng.random() < 0.6, scenes=rng.randint(1, 3), mixed=mixed)


# ---- scenes (the distributions of gs3d.scenes, drawn with torch) ---------------


def _raw(kind, n, sh, seed, device):
    g = torch.Generator(device=device).manual_seed(int(seed))
    f64 = dict(dtype=torch.float64, device=device, generator=g)

    def normal(*size):
        return torch.randn(*size, dtype=torch.float32, device=device, generator=g)

    def clusters(m, k, radius, smin, smax):
        d = torch.randn(k, 3, **f64)
        d /= d.norm(dim=1, keepdim=True)
        c = d * (radius * torch.rand(k, 1, **f64) ** (1.0 / 3.0))
        sigma = smin + (smax - smin) * torch.rand(k, 1, **f64)
        which = torch.randint(0, k, (m,), device=device, generator=g)
        return (c[which] + sigma[which] * torch.randn(m, 3, **f64)).float()

    if kind == "small":
        xyz, scale, opacity = 1.5 * normal(n, 3), 0.8 * normal(n, 3) - 4.5, 1.5 * normal(n)
    elif kind == "clusters":
        xyz = clusters(n, 64, 8.0, 0.2, 1.5)
        scale, opacity = normal(n, 3) - 4.0, 1.5 * normal(n)
    elif kind == "skew":
        bg = n // 5
        u = torch.randn(bg, 3, **f64)
        u /= u.norm(dim=1, keepdim=True)
        u *= 20.0 * torch.rand(bg, 1, **f64) ** (1.0 / 3.0)
        xyz = torch.cat([clusters(n - bg, 16, 8.0, 0.05, 0.3), u.float()])
        scale, opacity = 1.5 * normal(n, 3) - 3.5, 1.5 * normal(n) + 1.0
    else:  # mix: opaque clusters beside dense translucent ones
        t = n * 4 // 19
        xyz = torch.cat([clusters(n - t, 12, 7.0, 0.3, 0.9), clusters(t, 6, 7.0, 0.05, 0.15)])
        scale = torch.cat([0.6 * normal(n - t, 3) - 4.2, 0.4 * normal(t, 3) - 3.0])
        opacity = torch.cat([0.5 * normal(n - t) + 4.0, 0.15 * normal(t) - 5.0])
    k = 3 * ((sh + 1) ** 2 - 1)
    return dict(xyz=xyz, f_dc=0.5 * normal(n, 3), opacity=opacity, scale_log=scale,
                rot=normal(n, 4), f_rest=0.1 * normal(n, k) if k else None, sh_degree=sh)


def _activated(raw):
    """(pos, scale, rot, color, sh) in 64 bits, as the loader activates them."""
    d = {k: v.double() if torch.is_tensor(v) else v for k, v in raw.items()}
    one = torch.ones_like(d["opacity"])[:, None]
    pos = torch.cat([d["xyz"], one], 1)
    scale = torch.cat([torch.exp(d["scale_log"]), 0 * one], 1)
    length = d["rot"].norm(dim=1, keepdim=True)
    rot = d["rot"] / torch.where(length > 0, length, torch.ones_like(length))
    rgb = (0.5 + scenes.SH_C0 * d["f_dc"]).clamp(0, 1)
    color = torch.cat([rgb, torch.sigmoid(d["opacity"])[:, None].clamp(0, 1)], 1)
    return pos, scale, rot, color, d["f_rest"]


def _scene(kind, n, sh, seed, device="cuda"):
    a = _activated(_raw(kind, n, sh, seed, device))
    return [None if x is None else x.float().contiguous() for x in a]


def _eye(scene, radius, rng):
    """A pose on the orbit (elevation within 20 degrees); inside the skewed
    scene anywhere on the sphere, as its close-up and wide poses are."""
    az = rng.uniform(0, 2 * math.pi)
    el = math.asin(rng.uniform(-1, 1)) if scene == "skew" else math.radians(rng.uniform(-20, 20))
    if scene == "skew":
        el *= 0.9  # not along the up vector
    return (radius * math.cos(el) * math.sin(az), radius * math.sin(el),
            radius * math.cos(el) * math.cos(az))


def _views(case, seed):
    """[(scene index, 72-float camera block, width, height)] of a case."""
    rng = np.random.default_rng(1000 + int(seed))
    out = []
    for i in range(case.get("views", 1)):
        w, h = MIXED[i % len(MIXED)] if case.get("mixed") else (case["w"], case["h"])
        eye = _eye(case["scene"], case["radius"], rng)
        out.append((i % case.get("scenes", 1), scenes.camera_at(eye, w, h).getUniformData(w, h),
                    w, h))
    return out


def _scene_sizes(case):
    """Splats of each resident scene: n, n / 3, n / 6 ..."""
    return [max(1, case["n"] // (1 if i == 0 else 3 * i)) for i in range(case.get("scenes", 1))]


# ---- the library's buffers as tensors ------------------------------------------


class _Holder:
    """Owns a renderer; buffers handed out keep it alive."""

    def __init__(self, renderer):
        self.r = renderer

    def __del__(self):
        self.r.destroy()


class _Device:
    def __init__(self, holder, ptr, shape, typestr):
        self.holder = holder
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr,
                                         "version": 3}


class _State:
    """What a program keeps between calls."""

    def __init__(self, case):
        self.case = case
        self.seen = {}

    def buffer(self, name, shape, typestr):
        ptr, _ = self.holder.r.bufferInfo(name)
        key = (name, ptr)
        if key not in self.seen:
            self.seen[key] = torch.as_tensor(_Device(self.holder, ptr, shape, typestr),
                                             device="cuda")
        return self.seen[key]


def _load_scene(r, case, index, tensors):
    """gs3d_set_splats / gs3d_add_scene from device memory."""
    pos, scale, rot, color, sh = tensors
    torch.cuda.synchronize()  # the library copies on its own stream
    p = lambda t: None if t is None else C.c_void_p(t.data_ptr())  # noqa: E731
    n, deg = pos.shape[0], case["sh"] if sh is not None else 0
    if index == 0:
        r._call("gs3d_set_splats", n, p(pos), p(scale), p(rot), p(color), p(sh), deg, 1)
        r.scene.splats = DeviceSplats(n, deg)
    else:
        out = C.c_uint32()
        r._call("gs3d_add_scene", n, p(pos), p(scale), p(rot), p(color), p(sh), deg, 1,
                C.byref(out))


def _renderer(case, seed):
    r = GaussianSplatRenderer(Scene())
    r.init()
    for i, n in enumerate(_scene_sizes(case)):
        _load_scene(r, case, i, _scene(case["scene"], n, case["sh"], 17 * int(seed) + i))
    tile = (case["tw"], case["th"])
    if case["kind"] != "stages":
        r.setTuning(tile, 8, case["raster_batch"])
        if case["schedule"] == "learned":
            model = Path(learned.__file__).with_name(MODELS[tile])
            r.setCostModel(model)
        r.setSchedule(SCHEDULES[case["schedule"]])
        r.setCudaGraph(bool(case.get("graph")))
    return r


def prepare(case, seed):
    s = _State(case)
    if case["kind"] == "ply":
        raw = {k: v.cpu().numpy() if torch.is_tensor(v) else v
               for k, v in _raw("clusters", case["n"], case["sh"], seed, "cuda").items()}
        s.data = ply.write_ply(raw, case["format"])
        r = GaussianSplatRenderer(Scene())
        r.init()
        s.holder = _Holder(r)
        return s
    if case["kind"] == "train":
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        s.lib = _lib.load()
        n = case["n"]
        s.x = torch.randn(n, learned.F, device="cuda", generator=g)
        s.t = torch.randn(n, device="cuda", generator=g) * 0.7 + 6.0
        s.params = torch.from_numpy(learned.init_params(int(seed), 6.0)).cuda()
        s.acts = torch.empty(n, 2 * learned.H + 1, device="cuda")
        s.y = torch.empty(n, device="cuda")
        s.grads = torch.zeros_like(s.params)
        return s
    r = _renderer(case, seed)
    s.holder = _Holder(r)
    s.views = _views(case, seed)
    if case["kind"] == "frame":
        _, u, w, h = s.views[0]
        r.setAlwaysRebin(True)
        s.frame = RenderFrameInfo(w, h, u)
        s.rgba = torch.empty(h, w, 4, dtype=torch.uint8, device="cuda")
        s.background = np.array([0.1, 0.1, 0.12, 1.0], np.float32)
        r.render(s.frame)  # the first frame sizes the buffers
    elif case["kind"] == "batch":
        r.rebinBatch(s.views)
        r.rebinBatch(s.views)
    else:
        r.setStagewise(True)
        _, u, w, h = s.views[0]
        r.rebin(case["n"], -(-w // case["tw"]), -(-h // case["th"]), w, h, u)
    # sorted references beyond this many depend on the scene drawn: outputs
    # have the shape of their case
    s.refs = max(1, int(0.2 * sum(_estimated_refs(json.dumps(case, sort_keys=True)))))
    if r.refCount() < s.refs:
        raise RuntimeError(f"{r.refCount()} references, {s.refs} expected at least")
    s.pixels = sum(w * h for _, _, w, h in s.views)
    s.tiles = sum((-(-w // case["tw"])) * (-(-h // case["th"])) for _, _, w, h in s.views)
    return s


def _rebin_outputs(s):
    return {"image": s.buffer("splat_target", (s.pixels, 4), "<f2"),
            "tile_costs": s.buffer("tile_costs", (s.tiles,), "<i4"),
            "keys": s.buffer("sort_keys_a", (s.refs, 2), "<i4"),
            "values": s.buffer("sort_values_a", (s.refs,), "<i4"),
            "tile_offsets": s.buffer("tile_offsets", (s.tiles + 1,), "<i4")}


def run(s):
    kind = s.case["kind"]
    if kind == "train":
        p = learned._dev
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        n = s.case["n"]
        s.lib.gs3d_mlp_forward(p(s.params), p(s.x), n, p(s.acts), p(s.y), stream)
        s.grads.zero_()
        s.lib.gs3d_mlp_backward(p(s.params), p(s.x), p(s.acts), p(s.t), n, p(s.grads), stream)
        return {"acts": s.acts, "y": s.y, "grads": s.grads}
    r = s.holder.r
    if kind == "ply":
        r.loadPly(s.data)
        n, k = s.case["n"], 3 * ((s.case["sh"] + 1) ** 2 - 1)
        out = {f: s.buffer("splat_" + f, (n, 4), "<f4")
               for f in ("positions", "scales", "rotations", "colors")}
        if k:
            out["sh_rest"] = s.buffer("splat_sh_rest", (n, k), "<f4")
        return out
    if kind == "batch":
        r.rebinBatch(s.views, check=False)
        return _rebin_outputs(s)
    if kind == "frame":
        r.render(s.frame)
        bg = s.background.ctypes.data_as(C.c_void_p)
        r._call("gs3d_composite", 0, _lib.COMPOSITE_SPLATS, 0, bg,
                C.c_void_p(s.rgba.data_ptr()), s.rgba.numel(), 1)
        return {**_rebin_outputs(s), "rgba": s.rgba}
    _, u, w, h = s.views[0]
    r.setCamera(u, w, h)
    r.preprocess()
    r.prefixScan()
    r.emitTileRefs()
    r.radixSort()
    r.identifyTileRanges()
    r.rasterizeTiles()
    n = s.case["n"]
    return {**_rebin_outputs(s),
            "projected": s.buffer("projected_splats", (n, 16), "<i4"),
            "offsets": s.buffer("splat_ref_offsets", (n + 1,), "<i4")}


# ---- what a pass cannot do without ---------------------------------------------


@functools.lru_cache(maxsize=None)
def _estimated_refs(text):
    """Expected (splat, tile) references of each view, from a small sample."""
    case, sample = json.loads(text), 20_000
    splats = _scene(case["scene"], sample, 0, 5, "cpu")
    out, sizes = [], _scene_sizes(case)
    for sid, u, w, h in _views(case, 1):
        pr = _project([x if x is None else x.double() for x in splats], 0, u, w, h)
        lo, hi = _tile_rect(pr, case, w, h)
        out.append(float(((hi - lo + 1).prod(1) * pr["valid"]).sum()) * sizes[sid] / sample)
    return out


def work(case):
    if case["kind"] == "ply":
        k = 3 * ((case["sh"] + 1) ** 2 - 1)
        # the file's rows in, the activated arrays out
        return {"bytes": case["n"] * (4 * (14 + k) + 64 + 4 * k), "flops": case["n"] * 60}
    if case["kind"] == "train":
        n, p = case["n"], learned.P
        macs = 64 * 16 + 64 * 64 + 64
        # forward, and the two products of backward (none for the inputs)
        flops = 2 * n * (2 * macs + 64 * 64 + 64)
        # features and targets in, activations out and in, y and gradients out
        return {"bytes": 4 * (n * (16 + 1 + 2 * 129 + 1) + 3 * p), "flops": flops}
    total, flops = 0.0, 0.0
    views = _views(case, 1)
    sizes = _scene_sizes(case)
    k = 3 * ((case["sh"] + 1) ** 2 - 1)
    for i, n in enumerate(sizes):
        if any(v[0] == i for v in views):
            total += n * (64 + 4 * k)  # each scene's splats, read once a pass
    for (sid, u, w, h), refs in zip(views, _estimated_refs(json.dumps(case, sort_keys=True))):
        n = sizes[sid]
        tiles = (-(-w // case["tw"])) * (-(-h // case["th"]))
        # the projected record and count of every splat, a key and a value per
        # (splat, tile) reference, the tile offsets and the image
        total += n * (64 + 4) + refs * 12 + 4 * (tiles + 1) + 8 * w * h
        if case["kind"] == "frame":
            total += 4 * w * h
        flops += n * (250 + 2 * k)
    return {"bytes": total, "flops": flops}


# ---- 64-bit values of the computed outputs --------------------------------------


def _project(splats, deg, u, w, h):
    """preprocess_splats in 64 bits (the culls and radius as defined there)."""
    pos, scale, rot, color, sh = splats
    dev = pos.device
    u = torch.from_numpy(np.asarray(u, np.float64)).to(dev)
    V, P = u[0:16].reshape(4, 4).T, u[16:32].reshape(4, 4).T
    vp = pos @ V.T
    cp = vp @ P.T
    wc = torch.where(cp[:, 3] > 0, cp[:, 3], torch.ones_like(cp[:, 3]))
    ndc = cp[:, :3] / wc[:, None]
    valid = (cp[:, 3] > 0) & (ndc[:, :2].abs() <= 1).all(1) & (ndc[:, 2] >= 0) & (ndc[:, 2] <= 1)
    mean = torch.stack([(ndc[:, 0] * 0.5 + 0.5) * w, (1 - (ndc[:, 1] * 0.5 + 0.5)) * h], 1)
    q, x, y, z = rot.unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - q * z), 2 * (x * z + q * y),
                     2 * (x * y + q * z), 1 - 2 * (x * x + z * z), 2 * (y * z - q * x),
                     2 * (x * z - q * y), 2 * (y * z + q * x), 1 - 2 * (x * x + y * y)],
                    1).reshape(-1, 3, 3)
    M = R * scale[:, None, :3]
    S = M @ M.transpose(1, 2)
    fx, fy = P[0, 0] * w * 0.5, P[1, 1] * h * 0.5
    iz = 1.0 / torch.where(valid, -vp[:, 2], torch.ones_like(wc))
    zero = torch.zeros_like(iz)
    J = torch.stack([fx * iz, zero, fx * vp[:, 0] * iz * iz, zero, -fy * iz,
                     -fy * vp[:, 1] * iz * iz], 1).reshape(-1, 2, 3)
    T = J @ V[:3, :3]
    cov = T @ S @ T.transpose(1, 2)
    a, b, c = cov[:, 0, 0] + 0.3, cov[:, 1, 0], cov[:, 1, 1] + 0.3
    det = a * c - b * b
    valid &= det > 0
    mid = 0.5 * (a + c)
    lam = mid + torch.sqrt((mid * mid - det).clamp(min=0.1))
    radius = torch.ceil(3.0 * torch.sqrt(lam.clamp(min=0))).clamp(min=2.0)
    conic = torch.stack([c, -b, a], 1) / torch.where(valid, det, torch.ones_like(det))[:, None]
    rgb = color[:, :3]
    if deg:
        d = pos[:, :3] - u[64:67]
        d = d / d.norm(dim=1, keepdim=True).clamp(min=1e-300)
        x, y, z = d.unbind(1)
        c1 = 0.4886025119029199
        basis = [-c1 * y, c1 * z, -c1 * x]
        if deg > 1:
            basis += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
                      0.31539156525252005 * (2 * z * z - x * x - y * y),
                      -1.0925484305920792 * x * z, 0.5462742152960396 * (x * x - y * y)]
        if deg > 2:
            basis += [-0.5900435899266435 * y * (3 * x * x - y * y),
                      2.890611442640554 * x * y * z,
                      -0.4570457994644658 * y * (4 * z * z - x * x - y * y),
                      0.3731763325901154 * z * (2 * z * z - 3 * x * x - 3 * y * y),
                      -0.4570457994644658 * x * (4 * z * z - x * x - y * y),
                      1.445305721320277 * z * (x * x - y * y),
                      -0.5900435899266435 * x * (x * x - 3 * y * y)]
        B = torch.stack(basis, 1)
        rgb = (rgb + (sh.reshape(len(B), 3, -1) * B[:, None]).sum(2)).clamp(0, 1)
    return dict(valid=valid, mean=mean, depth=-vp[:, 2], radius=radius, conic=conic,
                opacity=color[:, 3], rgb=rgb)


def _tile_rect(pr, case, w, h):
    size = torch.tensor([case["tw"], case["th"]], dtype=torch.float64)
    top = torch.tensor([w - 1.0, h - 1.0], dtype=torch.float64)
    last = torch.ceil((top + 1) / size) - 1
    lo = torch.floor((pr["mean"] - pr["radius"][:, None]).clamp(min=0) / size)
    hi = torch.floor(torch.minimum(pr["mean"] + pr["radius"][:, None], top) / size)
    return torch.minimum(lo, last), torch.minimum(hi, last)


def _image(splats, deg, u, w, h):
    """The blended image, (h, w, 4) in 64 bits, block by block."""
    pr = _project(splats, deg, u, w, h)
    keep = pr["valid"].nonzero()[:, 0]
    keep = keep[torch.argsort(pr["depth"][keep], stable=True)]
    m, r, conic = pr["mean"][keep], pr["radius"][keep], pr["conic"][keep]
    op, rgb = pr["opacity"][keep], pr["rgb"][keep]
    dev, B, L = m.device, 32, 4096
    img = torch.zeros(h, w, 4, dtype=torch.float64, device=dev)
    for y0 in range(0, h, B):
        y1 = min(h, y0 + B)
        row = ((m[:, 1] + r >= y0) & (m[:, 1] - r <= y1)).nonzero()[:, 0]
        mx, rr = m[row, 0], r[row]
        for x0 in range(0, w, B):
            x1 = min(w, x0 + B)
            ids = row[(mx + rr >= x0) & (mx - rr <= x1)]
            yy, xx = torch.meshgrid(torch.arange(y0, y1, device=dev, dtype=torch.float64) + 0.5,
                                    torch.arange(x0, x1, device=dev, dtype=torch.float64) + 0.5,
                                    indexing="ij")
            px, py = xx.reshape(-1, 1), yy.reshape(-1, 1)
            T = torch.ones(len(px), 1, dtype=torch.float64, device=dev)
            acc = torch.zeros(len(px), 3, dtype=torch.float64, device=dev)
            for k in range(0, len(ids), L):
                j = ids[k:k + L]
                dx, dy = px - m[j, 0], py - m[j, 1]
                c = conic[j]
                power = -0.5 * (c[:, 0] * dx * dx + 2 * c[:, 1] * dx * dy + c[:, 2] * dy * dy)
                alpha = (op[j] * torch.exp(power)).clamp(max=0.99)
                alpha *= ((dx * dx + dy * dy <= r[j] * r[j]) & (power <= 0) &
                          (alpha >= 1.0 / 255.0))
                before = torch.cumprod(torch.cat([T, 1 - alpha], 1), 1)[:, :-1]
                alpha *= before >= 1e-4  # a pixel stops once T < 1e-4
                acc += (alpha * before) @ rgb[j]
                T = T * torch.prod(1 - alpha, 1, keepdim=True)
                if len(ids) > k + L and float(T.max()) < 1e-4:
                    break
            img[y0:y1, x0:x1] = torch.cat([acc, 1 - T], 1).reshape(y1 - y0, x1 - x0, 4)
    return img


def exact(case, seed):
    if case["kind"] == "ply":
        raw = _raw("clusters", case["n"], case["sh"], seed, "cuda")
        pos, scale, rot, color, sh = _activated(raw)
        out = {"positions": pos, "scales": scale, "rotations": rot, "colors": color}
        if sh is not None:
            out["sh_rest"] = sh
        return out
    if case["kind"] == "train":
        s = prepare(case, seed)
        H, F = learned.H, learned.F
        p = s.params.double().requires_grad_()
        w1, b1, w2, b2, w3, b3 = torch.split(p, [H * F, H, H * H, H, H, 1])
        h1 = torch.relu(s.x.double() @ w1.reshape(H, F).T + b1)
        h2 = torch.relu(h1 @ w2.reshape(H, H).T + b2)
        y = h2 @ w3 + b3
        ((y - s.t.double()) ** 2).mean().backward()
        acts = torch.cat([h1, h2, y[:, None]], 1).detach()
        return {"acts": acts, "y": y.detach(), "grads": p.grad}
    pixels = sum(w * h for _, _, w, h in _views(case, seed))
    if case["scene"] == "skew" or pixels > 2_100_000 or case["n"] * case.get("views", 1) > 3_500_000:
        return None  # more than some seconds in 64 bits
    sizes = _scene_sizes(case)
    splats = [[x if x is None else x.double() for x in
               _scene(case["scene"], n, case["sh"], 17 * int(seed) + i)]
              for i, n in enumerate(sizes)]
    img = [_image(splats[sid], case["sh"], u, w, h).reshape(-1, 4)
           for sid, u, w, h in _views(case, seed)]
    out = {"image": torch.cat(img), "keys": None, "values": None, "tile_offsets": None,
           "tile_costs": None}
    if case["kind"] == "frame":
        out["rgba"] = None
    if case["kind"] == "stages":
        out.update(projected=None, offsets=None)
    return out
