"""Performance cases: calls of this framework's public entry points as a rendering host makes them,
from a viewport thumbnail to a batch of many views.

A case is a dict of plain values. ``kind`` says which chain of passes one call of ``run`` makes:

* ``raycast``    primary visibility with the Depth / Albedo / Normal AOVs (what a viewport asks for first)
* ``restir``     one progressive frame: raycast, RIS or ReSTIR direct light, accumulation
* ``orbit``      one frame of a moving camera: reprojected history, capped M, spatial neighbours
* ``path``       one progressive path-traced frame
* ``views``      path-traced views of one scene in one batched call
* ``accumulate`` accumulation of a frame into the running mean and its hand-off in a display format
* ``serve``      render jobs of mixed sizes and pipelines through the job server, images taken back to the host

Every frame is handed off as a Hydra render buffer takes it: resolved into device memory of the caller.
Scenes are the seeded benchmark scenes of ``hdrestir_b200.configs``; the seed moves the camera, scales the
lights, and picks the frame index (and with it every random stream).
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from hdrestir_b200 import abi, configs
from hdrestir_b200.context import Context, path_trace_batch
from hdrestir_b200.scene import make_camera
from hdrestir_b200.server import Server

TERRAIN = dict(scene="terrain", grid=512, spheres=2000, lights=10000)  # the benchmark's 1.03M-triangle scene
BOXES = dict(scene="boxes", lights=1024)
BOX = dict(scene="box")


def _restir(name, scene, width, height, candidates=32, reservoir=True, skip_visibility=False, depth=1):
    return dict(name=name, kind="restir", **scene, width=width, height=height, candidates=candidates,
                reservoir=reservoir, skip_visibility=skip_visibility, depth=depth)


def listed():
    return [
        # the first image of a viewport and a thumbnail: latency and launches count
        dict(name="raycast_thumb", kind="raycast", **BOX, width=321, height=181),
        # the benchmark's closed box (config 0): a small path-traced frame, many short launches
        dict(name="path_box_256", kind="path", **BOX, width=256, height=256, depth=4),
        # a reduced-resolution interactive frame of a light scene, odd width
        _restir("restir_preview", dict(scene="terrain", grid=96, spheres=200, lights=500), 401, 225, candidates=8),
        # the benchmark's boxes (config 1): RIS without history, visibility of the winner only
        _restir("ris_boxes_512", BOXES, 512, 512, candidates=16, reservoir=False, skip_visibility=True),
        # the reference's default is more than one bounce: ReSTIR at the first hit, RIS after it
        _restir("restir_deep", BOXES, 480, 270, candidates=16, depth=4),
        # textured materials (all four PreviewSurface maps)
        _restir("restir_textured", dict(scene="textured"), 960, 540, candidates=32),
        # the benchmark's headline frame (config 2)
        _restir("restir_1080p", TERRAIN, 1920, 1080),
        # the benchmark's moving camera (config 2's orbit)
        dict(name="orbit_1080p", kind="orbit", **TERRAIN, width=1920, height=1080, candidates=32, neighbors=5,
             m_cap=20),
        # AOVs of a full-resolution 4K image
        dict(name="raycast_4k", kind="raycast", **TERRAIN, width=3840, height=2160),
        # progressive accumulation of a 4K image and its half-float hand-off (bytes only)
        dict(name="accumulate_4k", kind="accumulate", width=3840, height=2160, firefly=True, mode="parity",
             format="float16"),
        # config 3's shape: deep paths of uneven length under a dome, several views in one call
        dict(name="views_dome", kind="views", scene="dome", grid=256, spheres=2000, lights=10000, width=1280,
             height=720, views=9, view_size=512, depth=16),
        # config 4's shape: jobs of several sizes, scenes and pipelines served together
        dict(name="serve_mixed", kind="serve", jobs=8, max_frames=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """An image of lo..hi pixels (log-uniform), aspect 4:3 to 21:9, any parity."""
    px = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = rng.uniform(1.3, 2.35)
    h = max(16, int(math.sqrt(px / aspect)))
    return max(16, int(px / h)), h


def _any_scene(rng):
    pick = rng.choice(("box", "boxes", "terrain", "terrain", "textured"))
    if pick == "boxes":
        return dict(scene="boxes", lights=_log_int(rng, 16, 1024))
    if pick == "terrain":
        return dict(scene="terrain", grid=_log_int(rng, 64, 512), spheres=_log_int(rng, 50, 2000),
                    lights=_log_int(rng, 100, 10000))
    return dict(scene=pick)


def draw(rng):
    kind = rng.choice(("raycast", "restir", "restir", "restir", "orbit", "path", "path", "views", "accumulate",
                       "serve"))
    scene = _any_scene(rng)
    if kind == "raycast":
        w, h = _size(rng, 4e4, 8e6)
        return dict(kind=kind, **scene, width=w, height=h)
    if kind == "restir":
        if rng.random() < 0.25:  # several bounces
            w, h = _size(rng, 3e4, 2e5)
            return dict(kind=kind, **scene, width=w, height=h, candidates=rng.choice((4, 8, 16)),
                        reservoir=rng.random() < 0.7, skip_visibility=rng.random() < 0.3, depth=rng.randint(2, 5))
        w, h = _size(rng, 4e4, 2e6)
        return dict(kind=kind, **scene, width=w, height=h, candidates=rng.choice((4, 8, 16, 24, 32)),
                    reservoir=rng.random() < 0.75, skip_visibility=rng.random() < 0.3, depth=1)
    if kind == "orbit":
        w, h = _size(rng, 4e4, 2e6)
        return dict(kind=kind, scene="terrain", grid=_log_int(rng, 64, 512), spheres=_log_int(rng, 50, 2000),
                    lights=_log_int(rng, 100, 10000), width=w, height=h, candidates=rng.choice((8, 16, 32)),
                    neighbors=rng.randint(0, 8), m_cap=rng.choice((0, 10, 20)))
    if kind == "path":
        w, h = _size(rng, 4e4, 1e6)
        return dict(kind=kind, **scene, width=w, height=h, depth=rng.randint(2, 8))
    if kind == "views":
        w, h = _size(rng, 1e5, 9e5)
        return dict(kind=kind, scene="dome", grid=_log_int(rng, 64, 256), spheres=_log_int(rng, 50, 2000),
                    lights=_log_int(rng, 100, 10000), width=w, height=h, views=rng.randint(2, 9),
                    view_size=_log_int(rng, 100, 500), depth=rng.randint(3, 16))
    if kind == "accumulate":
        w, h = _size(rng, 1e5, 8e6)
        return dict(kind=kind, width=w, height=h, firefly=rng.random() < 0.7, mode=rng.choice(("parity", "shader")),
                    format=rng.choice(("float16", "float32", "unorm8")))
    return dict(kind=kind, jobs=rng.randint(2, 8), max_frames=rng.randint(1, 4))


# ------------------------------------------------------------------ inputs
def _scene(case, rng):
    """The case's scene and a function angle -> camera; the lights' intensities scaled by the seed."""
    w, h, kind = case.get("width", 64), case.get("height", 64), case["scene"]

    def orbit(angle, width=w, height=h):
        return configs.orbit_camera(angle, width, height)

    if kind == "box":
        sc, _ = configs.config0(w, h)

        def orbit(angle, width=w, height=h):  # inside the box, looking at its far half
            return make_camera((0.3 * math.sin(angle), 0.2 * math.cos(angle), 0.95), (0.0, -0.2, 0.0), width, height,
                               fov=70.0)
    elif kind == "boxes":
        sc, _ = configs.config1(w, h, n_lights=case["lights"])

        def orbit(angle, width=w, height=h):
            return make_camera((9.0 * math.sin(angle), 6.0, 9.0 * math.cos(angle)), (0.0, 0.0, 0.0), width, height,
                               fov=55.0)
    elif kind == "textured":
        sc, _ = configs.textured_variant(w, h)
    elif kind == "dome":
        sc, _, _ = configs.config3(w, h, n_small=1, small=64, grid=case["grid"], n_spheres=case["spheres"],
                                   n_lights=case["lights"], dome_size=(1024, 512))
    else:
        sc, _ = configs.config2(w, h, grid=case["grid"], n_spheres=case["spheres"], n_lights=case["lights"])
    scale = rng.uniform(0.5, 2.0, len(sc.lights))
    sc.lights = [dataclasses.replace(light, intensity=light.intensity * float(s))
                 for light, s in zip(sc.lights, scale)]
    return sc, orbit


def _color_plane(rng, pixels):
    """A noisy frame: mostly dim, a few bright samples (what the firefly clamp is for), alpha 1."""
    img = rng.exponential(0.3, (pixels, 4)).astype(np.float32)
    hot = rng.integers(0, pixels, max(1, pixels // 500))
    img[hot] *= np.float32(200.0)
    img[:, 3] = 1.0
    return img


FORMATS = {"float16": (abi.FMT_FLOAT16, torch.float16), "float32": (abi.FMT_FLOAT32, torch.float32),
           "unorm8": (abi.FMT_UNORM8, torch.uint8)}
ACCUMULATED = 7  # frames already in the running mean of an `accumulate` case


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    angle, frame = float(rng.uniform(0.0, 2.0 * math.pi)), int(rng.integers(0, 4096))
    st = dict(case=case, frame=0, first=frame, angle=angle)
    kind = case["kind"]
    if kind == "serve":
        sv = Server()
        ids, cams = [], []
        for sc_case in (BOX, BOXES, dict(scene="terrain", grid=128, spheres=500, lights=2000)):
            sc, orbit = _scene(sc_case, rng)
            ids.append(sv.add_scene(sc))
            cams.append(orbit)
        sizes = ((256, 256), (512, 512), (640, 360), (1280, 720))
        jobs = []
        for k in range(case["jobs"]):
            w, h = sizes[k % len(sizes)]
            which = int(rng.integers(3)) if k >= 3 else k
            jobs.append(dict(scene_id=ids[which], cam=cams[which](angle + 0.7 * k, w, h),
                             frames=1 + (3 * k) % case["max_frames"], pipeline="ris" if k % 2 else "pt"))
        st.update(server=sv, jobs=jobs)
        return st
    ctx = Context(timings=False)
    st["ctx"] = ctx
    if kind == "accumulate":
        w, h = case["width"], case["height"]
        sc, cam = configs.config0(w, h)
        ctx.upload_scene(sc)
        ctx.raycast(cam, 0)
        ctx.upload("Color", _color_plane(rng, w * h))
        ctx.upload("__accum_color", _color_plane(rng, w * h) * np.float32(ACCUMULATED))
        ctx.synchronize()
        st["out"] = torch.empty((h, w, 4), dtype=FORMATS[case["format"]][1], device="cuda")
        return st
    sc, orbit = _scene(case, rng)
    ctx.upload_scene(sc)
    st["orbit"] = orbit
    st["cam"] = orbit(angle)
    if kind == "views":
        ctxs, cams = [ctx], [st["cam"]]
        for k in range(1, case["views"]):
            c = Context(timings=False)
            c.share_scene(ctx)
            ctxs.append(c)
            cams.append(orbit(angle + 2.0 * math.pi * k / case["views"], case["view_size"], case["view_size"]))
        st.update(ctxs=ctxs, cams=cams)
        st["outs"] = [torch.empty((c.height, c.width, 4), device="cuda") for c in cams]
    elif kind == "raycast":
        st["outs"] = {n: torch.empty((case["height"], case["width"], c), device="cuda") for n, c in AOVS}
    else:
        st["out"] = torch.empty((case["height"], case["width"], 4), device="cuda")
    ctx.synchronize()
    return st


AOVS = (("Depth", 1), ("Albedo", 3), ("Normal", 3))


# ------------------------------------------------------------------ one pass
def _ris_settings(case):
    return dict(candidate_count=case["candidates"], use_reservoir=case["reservoir"],
                skip_visibility=case["skip_visibility"], max_depth=case["depth"])


def _hand_off(ctx, out):
    ctx.resolve("Color", 4, abi.FMT_FLOAT32, 4, device_ptr=out.data_ptr())
    return out


def run(state):
    case, kind, k = state["case"], state["case"]["kind"], state["frame"]
    state["frame"] = k + 1
    index = state["first"] + k  # the frame index seeds the random streams
    if kind == "serve":
        sv = state["server"]
        ids = [sv.submit(j["scene_id"], j["cam"], j["frames"], j["pipeline"],
                         **(configs.RIS_CONFIG2 if j["pipeline"] == "ris" else configs.PT_CONFIG4))
               for j in state["jobs"]]
        left = len(ids)
        while left:
            left -= sv.step()
        sv.finished()
        return [sv.take(i) for i in ids]
    ctx = state["ctx"]
    if kind == "accumulate":
        fmt = FORMATS[case["format"]][0]
        ctx.accumulate(ACCUMULATED + k, firefly=case["firefly"], mode=case["mode"])
        ctx.resolve("Color", 4, fmt, 4, device_ptr=state["out"].data_ptr())
        return state["out"]
    if kind == "raycast":
        ctx.raycast(state["cam"], index, aovs=[n for n, _ in AOVS])
        for n, c in AOVS:
            ctx.resolve(n, c, abi.FMT_FLOAT32, c, device_ptr=state["outs"][n].data_ptr())
        return state["outs"]
    if kind == "views":
        ctxs, cams = state["ctxs"], state["cams"]
        for c, cam in zip(ctxs, cams):
            c.raycast(cam, index)
        path_trace_batch(ctxs, cams, [index] * len(cams), max_depth=case["depth"])
        for c, out in zip(ctxs, state["outs"]):
            c.accumulate(k)
            _hand_off(c, out)
        return state["outs"]
    if kind == "orbit":  # a moving camera shows each frame as it is
        cam = state["orbit"](state["angle"] + 0.002 * k)
        ctx.raycast(cam, index)
        ctx.ris_path_trace(cam, index, candidate_count=case["candidates"], use_reservoir=True, max_depth=1,
                           m_cap=case["m_cap"], spatial_neighbors=case["neighbors"], spatial_radius=30.0,
                           reproject=True)
        return _hand_off(ctx, state["out"])
    cam = state["cam"]
    ctx.raycast(cam, index)
    if kind == "path":
        ctx.path_trace(cam, index, max_depth=case["depth"])
    else:
        ctx.ris_path_trace(cam, index, **_ris_settings(case))
    ctx.accumulate(k)
    return _hand_off(ctx, state["out"])


# ------------------------------------------------------------------ what a pass cannot do without
def _triangles(case):
    s = case["scene"]
    if s == "box":
        return 24
    if s == "boxes":
        return 770
    if s == "textured":
        return 2 * 63 * 63 + 80 * 256
    return 2 * (case["grid"] - 1) ** 2 + case["spheres"] * 256


def _ray_flops(case):
    """About one box test of 12 operations per child of a 4-wide tree's path, and four triangle tests."""
    return 4 * 12 * max(1.0, math.log(_triangles(case), 4)) + 4 * 50


def work(case):
    kind = case["kind"]
    if kind == "serve":
        px = sum(w * h * (1 + (3 * k) % case["max_frames"])
                 for k in range(case["jobs"]) for w, h in (((256, 256), (512, 512), (640, 360), (1280, 720))[k % 4],))
        return {"bytes": 150 * px, "flops": 18 * px * 400}
    px = case["width"] * case["height"]
    if kind == "accumulate":  # frame and sum in, sum, mean and display pixel out
        return {"bytes": px * (64 + 4 * {"float16": 2, "float32": 4, "unorm8": 1}[case["format"]]), "flops": px * 60}
    scene = 48 * min(_triangles(case), 600_000)
    ray = _ray_flops(case)
    if kind == "raycast":  # GBuffer and AOVs out
        return {"bytes": scene + px * (96 + 28), "flops": px * ray}
    if kind == "views":
        px += (case["views"] - 1) * case["view_size"] ** 2
    if kind in ("views", "path"):  # GBuffer, mean in and out, image out; two rays per vertex
        return {"bytes": scene + px * (96 + 64), "flops": px * ray * (1 + 2 * min(case["depth"], 6))}
    # GBuffer, reservoir and mean in and out, image out; a shadow ray per light candidate
    rays = 1 if case.get("skip_visibility") else 1 + case["candidates"] // 2
    return {"bytes": scene + px * (96 + 160 + 64), "flops": px * (rays * ray + case["candidates"] * 200)
            * case.get("depth", 1)}


# ------------------------------------------------------------------ 64-bit values
def _exact_raycast_box(case, seed):
    rng = np.random.default_rng(seed)
    angle = float(rng.uniform(0.0, 2.0 * math.pi))
    rng.integers(0, 4096)
    sc, orbit = _scene(case, rng)
    cam = orbit(angle)
    w, h = cam.width, cam.height
    inv_view, inv_proj = np.linalg.inv(cam.view), np.linalg.inv(cam.proj)

    def transform(p, m):
        q = np.concatenate([p, np.ones((len(p), 1))], 1) @ m
        return q[:, :3] / q[:, 3:]

    y, x = np.divmod(np.arange(w * h), w)
    ndc = np.stack([2.0 * (x + 0.5) / w - 1.0, 2.0 * (y + 0.5) / h - 1.0, -np.ones(w * h)], 1)
    o = transform(np.zeros((1, 3)), inv_view)[0]
    d = transform(transform(ndc, inv_proj), inv_view) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    best = np.full(w * h, np.inf)
    albedo, normal = np.zeros((w * h, 3)), np.zeros((w * h, 3))
    for inst in sc.instances:  # identity transforms
        mesh = sc.meshes[inst.mesh]
        col = np.asarray(sc.materials[inst.material].diffuse_color, np.float64)
        for a, b, c in mesh.points[mesh.indices].astype(np.float64):
            e1, e2 = b - a, c - a
            p = np.cross(d, e2)
            det = p @ e1
            with np.errstate(divide="ignore", invalid="ignore"):
                u = (p @ (o - a)) / det
                q = np.cross(o - a, e1)
                v = (d @ q) / det
                t = (q @ e2) / det
                hit = (np.abs(det) > 1e-8) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-4) & (t < best)
            n = np.cross(e1, e2)
            best[hit], albedo[hit], normal[hit] = t[hit], col, n / np.linalg.norm(n)
    depth = np.where(np.isfinite(best), best, 1.0)
    shape = (h, w, -1)
    return {"Depth": depth.reshape(shape), "Albedo": albedo.reshape(shape), "Normal": normal.reshape(shape)}


def _exact_accumulate(case, seed):
    rng = np.random.default_rng(seed)
    rng.uniform(0.0, 2.0 * math.pi)
    rng.integers(0, 4096)
    w, h = case["width"], case["height"]
    color = _color_plane(rng, w * h).astype(np.float64).reshape(h, w, 4)
    accum = (_color_plane(rng, w * h) * np.float32(ACCUMULATED)).astype(np.float64).reshape(h, w, 4)
    if case["firefly"]:
        lum = color[..., :3] @ np.array([0.2126, 0.7152, 0.0722])
        pad = np.pad(lum, 1, mode="edge")
        around = np.zeros_like(lum)
        for dy in range(3):
            for dx in range(3):
                if (dy, dx) != (1, 1):
                    around = np.maximum(around, pad[dy:dy + h, dx:dx + w])
        limit = 4.0 * around + 0.5
        clamp = (lum > limit) & (lum > 0.0)
        color[..., :3] *= np.where(clamp, limit / np.where(clamp, lum, 1.0), 1.0)[..., None]
    return (accum + color) / (ACCUMULATED + 1)


def exact(case, seed):
    """Rendered images follow float32 random decisions and have no 64-bit value; primary visibility of the
    closed box and the accumulated mean have one."""
    if case["kind"] == "raycast" and case["scene"] == "box" and case["width"] * case["height"] <= 4_000_000:
        return _exact_raycast_box(case, seed)
    if case["kind"] == "accumulate" and case["format"] != "unorm8":
        return _exact_accumulate(case, seed)
    return None
