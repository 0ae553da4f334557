#!/usr/bin/env python3
"""ReSTIR 1080p frames/s on the B200 passes (one JSON line on rank 0).

Workload (the benchmark's headline configuration): the seeded config-2 scene
(512x512-vertex noise terrain + 2000 instanced 256-triangle spheres = 1.03M
triangles, 10,000 rect lights), 1920x1080, RaycastPass -> RISPathTracePass
(32 candidates = 16 NEE + 16 BSDF, reservoir with temporal reuse, shadow rays
for every NEE candidate, maxDepth 1) -> AccumulationPass (firefly filter,
parity semantics). One step = one frame of that pipeline.

  value : frames/s with the scene and frame buffers resident in HBM, device
          time of the whole timed region (CUDA events on the library stream),
          max over ranks.
  e2e   : the same loop through the public API with the camera passed from the
          host and the "Color" image read back to pinned host memory every frame
          (hdr_download_async: each read-back overlaps the next frame's passes;
          the timed region ends after the last read-back).
  cpu_baseline / --impl reference : the reference's CPU implementation of the
          path timed on the host cores over a bounded sample of the frame.

Multi-GPU: frames are independent (replicas, weak scaling): every rank renders
its own frames, no collective on the data path; the barrier and a MAX of the
per-rank device times are the only communication.
"""
from __future__ import annotations

import argparse
import json
import os
import re
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

WIDTH, HEIGHT, CANDIDATES = 1920, 1080, 32
METRIC = "ReSTIR 1080p frames/s"
# algorithmic bytes per pixel of the ReSTIR integration pass: reservoir read 80 B +
# reservoir write 80 B + GBuffer read 64 B + colour write 16 B (five float4 reservoir planes,
# four float4 GBuffer planes)
INTEGRATE_BYTES_PER_PX = 80 + 80 + 64 + 16
# accumulation: colour in 16 + accum in 16 + accum out 16 + colour out 16, plus the sums, which
# pass through a plane of their own (16 out, 16 in) until the firefly clamp's check has run
ACCUM_BYTES_PER_PX = 64 + 32
# trace_shadow4_kernel, the dominant kernel: per shadow ray it must read its queue record
# (origin, slot, direction, limit: 32 B) and write one occlusion byte; the BVH and the
# triangles it reads are the scene's, shared by all rays of the launch
SHADOW_BYTES_PER_RAY = 32 + 1


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-serving", action="store_true", help="skip the batched and served legs")
    ap.add_argument("--serving-jobs", type=int, default=80, help="config-4 jobs per serving leg")
    ap.add_argument("--width", type=int, default=1920, help="smaller frames only for profiler captures")
    ap.add_argument("--height", type=int, default=1080)
    return ap.parse_args()


from hdrestir_b200.replicas import barrier as replica_barrier  # noqa: E402
from hdrestir_b200.replicas import dist_env, max_over_ranks, whole_job_rate  # noqa: E402


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def ncu_traffic(kernel_key: str):
    """Per-launch DRAM bytes from the committed ncu summary, scaled to the bench frame."""
    for f in sorted((ROOT / "profiles").glob("*.md")):
        m = re.search(rf"^{kernel_key}_dram_bytes_per_1080p_launch:\s*([0-9.eE+]+)", f.read_text(), re.M)
        if m:
            return float(m.group(1)), f.name
    return None, None


class ClockSampler:
    """nvidia-smi clocks + throttle reasons sampled every 200 ms during the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.dev = device_index
        self.proc = None
        self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.dev), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"], stdout=self.file,
                                         stderr=subprocess.DEVNULL)
        except FileNotFoundError:
            self.proc = None

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        self.proc.wait()
        self.file.flush()
        rows = [r.split(",") for r in Path(self.file.name).read_text().splitlines() if r.strip()]
        os.unlink(self.file.name)
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            try:
                sm.append(float(r[1]))
                mx = float(r[2])
                for k, n in enumerate(names):
                    if r[5 + k].strip().lower() == "active":
                        reasons.add(n)
            except (ValueError, IndexError):
                continue
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


# the CPU sample: tile rows 3, 11, 19, ... (every 8th 16-pixel row of tiles, 144 of the 1080
# image rows) of the real frame, the same rows every frame so their reservoirs keep history
SAMPLE_STRIDE, SAMPLE_OFFSET, TILE = 8, 3, 16


def sample_rows(height):
    return [y for ty in range(SAMPLE_OFFSET, (height + TILE - 1) // TILE, SAMPLE_STRIDE)
            for y in range(ty * TILE, min(height, ty * TILE + TILE))]


def cpu_sample_port(orc, cam, frame: int):
    """The C restatement on the sampled tile rows of one frame (raycast + ReSTIR
    integration; reservoirs of those rows persist in `orc` from frame to frame)
    and its accumulation over the whole frame; returns seconds per full frame."""
    rows = sample_rows(cam.height)
    t0 = time.perf_counter()
    for ty in range(SAMPLE_OFFSET, (cam.height + TILE - 1) // TILE, SAMPLE_STRIDE):
        orc.frame_band(cam, frame, ty * TILE, min(cam.height, ty * TILE + TILE), ris=True,
                       candidate_count=CANDIDATES, use_reservoir=True)
    t_rows = time.perf_counter() - t0
    t0 = time.perf_counter()
    orc.accumulate(cam, frame, firefly=True)
    return t_rows * cam.height / len(rows) + (time.perf_counter() - t0)


def cpu_frames(scene, cam, frames, threads):
    """Seconds per full 1920x1080 frame for each of `frames` (consecutive frame
    indices: the sampled rows carry their reservoir history) on the host cores:
    the reference's own passes compiled in place when built, else the restatement.
    Also returns the accumulated "Color" after the last frame (valid on the
    sampled rows)."""
    import numpy as np
    color = np.zeros((cam.width * cam.height, 4), np.float32)
    if _ref_available():
        from oracle import refharness
        got = refharness.cpu_sample(scene, cam, threads, frames=frames, stride=SAMPLE_STRIDE, offset=SAMPLE_OFFSET,
                                    candidate_count=CANDIDATES, color_out=color)
        return [sec for _, sec, _ in got], "reference", color
    from oracle.oracle import Oracle
    orc = Oracle(scene, threads=threads)
    try:
        secs = [cpu_sample_port(orc, cam, f) for f in frames]
        return secs, "port", orc.color.copy()
    finally:
        orc.close()


def mse_block(ctx, cam, cpu_color, frames, high_frames=64):
    """Equal MSE at the headline workload: the GPU image after `frames` accumulated
    frames and the CPU reference's image after the same frames, each against a
    high-sample image of the same estimator (GPU, `high_frames` frames of other
    random streams), over the sampled tile rows without their first and last row
    (the firefly clamp there sees the unrendered neighbours of the CPU sample).
    MSE normalised by the high-sample image's peak, as the reference's image tests do."""
    import numpy as np
    from hdrestir_b200 import configs
    from hdrestir_b200.context import Context
    ris = dict(candidate_count=CANDIDATES, use_reservoir=True, skip_visibility=False, max_depth=1)
    rows = [y for ty in range(SAMPLE_OFFSET, (cam.height + TILE - 1) // TILE, SAMPLE_STRIDE)
            for y in range(ty * TILE + 1, min(cam.height, ty * TILE + TILE) - 1)]
    imgs = {}
    c = Context(device=ctx.device, timings=False)
    try:
        c.share_scene(ctx)
        for name, start, n in (("gpu", 0, frames), ("high", 10_000, high_frames)):
            c.clear_persistent()
            for f in range(start, start + n):
                c.raycast(cam, f)
                c.ris_path_trace(cam, f, **ris)
                c.accumulate(f - start, firefly=True, mode="parity")
            imgs[name] = c.download("Color").reshape(cam.height, cam.width, 4)[rows, :, :3].astype(np.float64)
    finally:
        c.close()
    cpu = cpu_color.reshape(cam.height, cam.width, 4)[rows, :, :3].astype(np.float64)
    peak = max(float(imgs["high"].max()), 1e-12)
    m_gpu = float(np.mean(((imgs["gpu"] - imgs["high"]) / peak) ** 2))
    m_cpu = float(np.mean(((cpu - imgs["high"]) / peak) ** 2))
    return {"frames": frames, "high_sample_frames": high_frames, "rows": len(rows), "mse_gpu": m_gpu,
            "mse_cpu_reference": m_cpu, "ratio": m_gpu / m_cpu if m_cpu > 0 else None,
            "note": "same estimator and random streams on both sides, so equal MSE; the frames/s above are at "
                    "this MSE"}


def cpu_sample_label(height, frames_desc):
    rows = len(sample_rows(height))
    return (f"tile rows {SAMPLE_OFFSET}, {SAMPLE_OFFSET + SAMPLE_STRIDE}, ... (every {SAMPLE_STRIDE}th row of "
            f"16x16 tiles: {rows} of {height} image rows) of the real {WIDTH}x{height} frame, the same rows every "
            f"frame so their reservoirs keep history; RaycastPass + RISPathTracePass on those rows scaled by "
            f"{height}/{rows}, plus AccumulationPass over the whole frame; {frames_desc}")


def _ref_available() -> bool:
    return (ROOT / "oracle" / "_ref" / "libhdr_ref.so").exists()


def run_reference(args, rank, world):
    """--impl reference: the reference's CPU path on the host cores (rank 0 only).
    Each step is one frame (consecutive frame indices, history carried) on the
    sampled tile rows, with all the host threads."""
    if rank != 0:
        return None
    from hdrestir_b200 import configs
    threads = os.cpu_count() or 1
    scene, cam = configs.config2(WIDTH, HEIGHT)
    n = args.warmup + args.steps
    if _ref_available():
        from oracle import refharness
        ref = refharness.Reference(scene)  # scene build, untimed like the GPU arm's upload
        secs = [s for _, s, _ in refharness.cpu_sample(scene, cam, threads, frames=range(n), stride=SAMPLE_STRIDE,
                                                        offset=SAMPLE_OFFSET, ref=ref, candidate_count=CANDIDATES)]
        ref.close()
        kind = "reference"
    else:
        from oracle.oracle import Oracle
        orc = Oracle(scene, threads=threads)
        secs = [cpu_sample_port(orc, cam, f) for f in range(n)]
        orc.close()
        kind = "port"
    timed = secs[args.warmup:]
    value = len(timed) / sum(timed)
    return {
        "metric": METRIC, "value": value, "unit": "frames/s", "n_gpus": args.gpus, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": 1000.0 / value, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "impl": "reference",
        "data": "synthetic seeded config-2 scene (1.03M triangles, 10k rect lights)",
        "config": config_block(),
        "cpu_baseline": {"value": value, "unit": "frames/s", "cores": threads, "kind": kind,
                         "sample": cpu_sample_label(HEIGHT, f"frames {args.warmup}..{n - 1} timed after "
                                                            f"{args.warmup} warm-up frames")},
        "e2e": {"value": value, "unit": "frames/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }


def config_block():
    return {"workload": "config2: ReSTIR 1920x1080, 32 candidates (16 NEE + 16 BSDF), reservoir temporal reuse, "
                        "shadow ray per NEE candidate, maxDepth 1, firefly accumulation",
            "width": WIDTH, "height": HEIGHT, "candidates": CANDIDATES, "triangles": 1034242, "lights": 10000,
            "pipeline": "RaycastPass -> RISPathTracePass -> AccumulationPass",
            "l2": "inputs larger than L2 (scene ~0.3 GB + frame buffers ~0.4 GB resident)",
            "parallelism": "replicas"}


def batched_leg(ctx, n_images=4, frames=4, warm=2):
    """4 orbit views of the config-2 scene at 1920x1080, ReSTIR as in the headline:
    rendered one after another (plain) and as one batched frame (one trace launch
    for all images). Device-synchronised wall time around each leg (the images
    run on several streams); images are identical (tests/test_gpu_batch.py)."""
    import torch
    from hdrestir_b200 import configs
    from hdrestir_b200.context import Context, ris_path_trace_batch
    ris = configs.RIS_CONFIG2
    cams = [configs.orbit_camera(0.9 * k, WIDTH, HEIGHT) for k in range(n_images)]
    ctxs = [Context(device=torch.cuda.current_device(), timings=False) for _ in cams]
    out = {}
    try:
        for c in ctxs:
            c.share_scene(ctx)
        for mode in ("plain", "batched"):
            for c in ctxs:
                c.clear_persistent()

            def frame(k):
                for c, cam in zip(ctxs, cams):
                    c.raycast(cam, k)
                if mode == "batched":
                    ris_path_trace_batch(ctxs, cams, [k] * len(cams), **ris)
                else:
                    for c, cam in zip(ctxs, cams):
                        c.ris_path_trace(cam, k, **ris)
                for c in ctxs:
                    c.accumulate(k)

            for k in range(warm):
                frame(k)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for k in range(warm, warm + frames):
                frame(k)
            torch.cuda.synchronize()
            dt = time.perf_counter() - t0
            out[mode] = {"frames_per_s": n_images * frames / dt, "ms_per_batch_frame": 1000.0 * dt / frames}
    finally:
        for c in ctxs:
            c.close()
    out["workload"] = f"{n_images} views of config 2 at {WIDTH}x{HEIGHT}, {frames} timed frames each"
    return out


def orbit_leg(ctx, frames=8, warm=3):
    """Config 2's orbit run (extensions): the camera circles the terrain by 0.002 rad per
    frame; temporal reuse reprojected from the previous frame, M-cap 20, 5 spatial neighbours
    within 30 px; firefly accumulation restarted at each pose. Device-timed with CUDA events
    around each frame's passes."""
    import torch
    from hdrestir_b200 import configs
    from hdrestir_b200.context import Context
    ris = dict(configs.RIS_CONFIG2, m_cap=20, spatial_neighbors=5, spatial_radius=30.0, reproject=True)
    c = Context(device=torch.cuda.current_device(), timings=False)
    try:
        c.share_scene(ctx)
        ms = []
        for k in range(warm + frames):
            cam = configs.orbit_camera(0.002 * k, WIDTH, HEIGHT)
            c.region_begin(0)
            c.raycast(cam, k)
            c.ris_path_trace(cam, k, **ris)
            c.accumulate(0)
            c.region_end(0)
            c.synchronize()
            if k >= warm:
                ms.append(c.region_elapsed(0))
    finally:
        c.close()
    avg = sum(ms) / len(ms)
    return {"frames_per_s": 1000.0 / avg, "ms_per_frame": avg,
            "workload": f"config 2 orbit at {WIDTH}x{HEIGHT}: reprojected temporal reuse, M-cap 20, "
                        f"5 spatial neighbours within 30 px, {frames} timed frames"}


def config3_leg(reps: int = 2):
    """Config 3: one 3840x2160 frame and 64 frames of 512x512 (orbit views), PathTracer
    maxDepth 16 on the config-2 scene plus a 2048x1024 dome: as 65 PathTracePass launches
    (plain) and as one launch over all tiles (batched). Device-synchronised wall time of the
    integration pass; the primary rays (raycast) run before it, untimed."""
    import torch
    from hdrestir_b200 import configs
    from hdrestir_b200.context import Context, path_trace_batch
    sc, cam, cams = configs.config3()
    cams = [cam] + cams
    paths = sum(c.width * c.height for c in cams)
    ctxs = [Context(device=torch.cuda.current_device(), timings=False) for _ in cams]
    out = {"workload": "config 3: 3840x2160 + 64 x 512x512, PathTracer maxDepth 16, dome 2048x1024",
           "paths": paths}
    try:
        ctxs[0].upload_scene(sc)
        for x in ctxs[1:]:
            x.share_scene(ctxs[0])
        best = {}
        for rep in range(reps + 1):  # the first round warms up
            for mode in ("plain", "batched"):
                for x, c in zip(ctxs, cams):
                    x.raycast(c, rep)
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                if mode == "batched":
                    path_trace_batch(ctxs, cams, [rep] * len(cams), **configs.PT_CONFIG3)
                else:
                    for x, c in zip(ctxs, cams):
                        x.path_trace(c, rep, **configs.PT_CONFIG3)
                torch.cuda.synchronize()
                dt = time.perf_counter() - t0
                if rep > 0:
                    best[mode] = min(best.get(mode, 1e30), dt)
        for mode, dt in best.items():
            out[mode] = {"ms": 1000.0 * dt, "paths_per_s": paths / dt}
    finally:
        for x in ctxs:
            x.close()
    return out


def serving_leg(n_jobs: int, rate: float = 200.0):
    """Config-4 serving: the same Poisson job stream (`rate` jobs/s) through the
    server in serial mode (the plain per-frame pipeline, one job at a time) and
    in served mode (continuous batching). Latency = host wall time from a job's
    arrival to the step that finished it; images are identical in both modes
    (tests/test_gpu_server.py), so the comparison is at equal MSE. At 200 jobs/s
    the jobs arrive faster than any mode serves them and the latencies measure
    the drain of that backlog; at a rate the box sustains they measure service."""
    from hdrestir_b200 import abi, configs
    from hdrestir_b200.server import Server
    jobs = configs.config4_jobs(n_jobs, rate=rate)
    scenes = [configs.config0()[0], configs.config1()[0], configs.config2()[0]]
    cams = [configs.config_camera(j["cfg"], j["width"], j["height"]) for j in jobs]
    mpx_frames = sum(j["width"] * j["height"] * j["frames"] for j in jobs) / 1e6
    out = {"workload": f"config 4: {n_jobs} jobs, Poisson {rate:g} jobs/s, scenes config 0-2, "
                       "256^2..2048x1152, 1-16 frames, ReSTIR (32 cand) or PathTracer (maxDepth 4); "
                       "HBM admission budget 120 GB",
           "mpx_frames": mpx_frames}
    step_px = {"plain": 0, "served_all": 0, "served": 32 << 20}

    def stream(sv, sids):
        lat, pending, nxt = [], {}, 0
        steps = 0
        t0 = time.perf_counter()
        while len(lat) < n_jobs:
            now = time.perf_counter() - t0
            while nxt < n_jobs and jobs[nxt]["arrival"] <= now:
                j = jobs[nxt]
                kw = configs.RIS_CONFIG2 if j["pipeline"] == "ris" else configs.PT_CONFIG4
                jid = sv.submit(sids[j["cfg"]], cams[nxt], j["frames"], j["pipeline"], **kw)
                pending[jid] = j["arrival"]
                nxt += 1
            if not pending:
                time.sleep(max(0.0, jobs[nxt]["arrival"] - now))
                continue
            steps += 1
            if sv.step() == 0:
                continue
            now = time.perf_counter() - t0
            for jid in sv.finished():
                if sv.state(jid)[0] == abi.JOB_FAILED:
                    raise RuntimeError(f"serving job {jid} failed")
                lat.append(now - pending.pop(jid))
                sv.take(jid, keep_image=False)
        return lat, steps, time.perf_counter() - t0

    for mode in ("plain", "served_all", "served"):
        with Server(device=0, hbm_budget=120 << 30, serial=(mode == "plain"), step_pixels=step_px[mode]) as sv:
            sids = [sv.add_scene(s) for s in scenes]
            # untimed warm-up: the same job stream once, so the timed pass sees the server at steady state
            # (kernels loaded, contexts pooled, the frame-buffer pool and batch queues grown)
            stream(sv, sids)
            # two timed passes, the one with the shorter makespan kept (with its latencies): a
            # host-side stall of the driving loop shows in one pass, not in the server's steady state
            lat, steps, makespan = min((stream(sv, sids) for _ in range(2)), key=lambda r: r[2])
        lat.sort()
        out[mode] = {"jobs_per_s": n_jobs / makespan, "mpx_frames_per_s": mpx_frames / makespan,
                     "makespan_s": makespan, "latency_p50_ms": 1000.0 * statistics.median(lat),
                     "latency_p99_ms": 1000.0 * lat[min(len(lat) - 1, int(round(0.99 * (len(lat) - 1))))],
                     "steps": steps}
    out["modes"] = ("plain: one job at a time, each frame rendered alone; served_all: every admitted job "
                    "advances each step; served: least remaining work first less half the work served "
                    "since the job arrived, 32 Mpx per step; each mode "
                    "timed on its second and third passes over the job stream, the shorter kept (the first "
                    "warms the server up)")
    return out


def graph_leg(ctx, cam, ris, world, n_frames=10):
    """Each frame's pass chain submitted eagerly (one call per pass) and as one CUDA
    graph (hdr_graph_*: one frame recorded, then replayed per frame with its frame
    index: a frame-slot store and one graph launch). Device time of n_frames
    consecutive frames (CUDA events around the loop: the stream idles where the host
    submits slower than the device runs) and the host's median submit time per frame,
    for the headline frame and for config 0's 256x256 PathTracer frame (maxDepth 4:
    4 rounds of small wavefront kernels)."""
    from hdrestir_b200 import configs
    from hdrestir_b200.context import Context
    out = {}
    sc0, cam0 = configs.config0()

    def restir(c, k, cam=cam):
        c.raycast(cam, k)
        c.ris_path_trace(cam, k, **ris)
        c.accumulate(k, firefly=True, mode="parity")

    def pt(c, k, cam=cam0):
        c.raycast(cam, k)
        c.path_trace(cam, k, max_depth=4)
        c.accumulate(k, firefly=True, mode="parity")

    for name, passes, scene in (("config2_restir_1080p", restir, None), ("config0_pt_256", pt, sc0)):
        g = Context(device=ctx.device, timings=False)
        try:
            if scene is None:
                g.share_scene(ctx)
            else:
                g.upload_scene(scene)
            res = {}
            k = 0
            for mode in ("eager", "graph"):
                # warm-up: the first frame sizes the buffers; in graph mode the second is recorded
                passes(g, k)
                k += 1
                if mode == "graph":
                    g.record_frame(lambda: passes(g, k))
                else:
                    passes(g, k)
                k += 1
                g.synchronize()
                host = []
                g.region_begin(0)
                for _ in range(n_frames):
                    t0 = time.perf_counter()
                    if mode == "graph":
                        g.graph_launch(k)  # the recorded frame replayed with this frame index
                    else:
                        passes(g, k)
                    host.append(time.perf_counter() - t0)
                    k += 1
                g.region_end(0)
                ms = max_over_ranks(g.region_elapsed(0), world) / n_frames
                res[mode] = {"frames_per_s": world * 1000.0 / ms, "ms_per_frame": ms,
                             "host_submit_us_per_frame": 1e6 * statistics.median(host)}
            res["graph_info"] = g.graph_info()
            out[name] = res
        finally:
            g.close()
    out["note"] = ("graph = the frame's passes recorded with hdr_graph_begin/_end and run with one "
                   "hdr_graph_launch; images identical to eager (tests/test_gpu_graph.py)")
    return out


def run_ours(args, rank, local_rank, world):
    import numpy as np
    import torch
    from hdrestir_b200 import configs
    from hdrestir_b200.context import Context

    torch.cuda.set_device(local_rank)
    if world > 1:
        import torch.distributed as dist
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300),
                                device_id=torch.device("cuda", local_rank))
    ctx = Context(device=local_rank, timings=True)
    scene, cam = configs.config2(WIDTH, HEIGHT)
    ctx.upload_scene(scene)
    ris = dict(candidate_count=CANDIDATES, use_reservoir=True, skip_visibility=False, max_depth=1)

    def frame(k):
        ctx.raycast(cam, k)
        ctx.ris_path_trace(cam, k, **ris)
        ctx.accumulate(k, firefly=True, mode="parity")

    def barrier():
        replica_barrier(world)

    # ---- warm-up (frame indices continue through the timed region: reservoirs persist)
    ctx.clear_persistent()
    for k in range(args.warmup):
        frame(k)
    ctx.synchronize()
    ctx.pass_times(reset=True)

    # ---- device-resident timed region
    clocks = ClockSampler(local_rank)
    clocks.start()
    barrier()
    launches0 = ctx.launch_count()
    frame_ms = []
    ctx.region_begin(0)
    for k in range(args.warmup, args.warmup + args.steps):
        ctx.region_begin(1)
        frame(k)
        ctx.region_end(1)
        frame_ms.append(ctx.region_elapsed(1))
    ctx.region_end(0)
    total_ms = ctx.region_elapsed(0)
    barrier()
    clk = clocks.stop()
    gpu_launches = ctx.launch_count() - launches0
    (t_ray, t_int, t_acc, t_gen, t_closest, t_shadow, t_shade), counts = ctx.pass_times(reset=True, slots=7)
    wave_counts = ctx.download("__wave_counts").view(np.int32)  # [0] closest rays, [1] shadow rays (last frame)
    n_shadow = int(wave_counts[1])
    n_closest = int(wave_counts[0])
    total_ms = max_over_ranks(total_ms, world)
    fps = whole_job_rate(args.steps, world, total_ms)

    # ---- the same frames in the other execution forms (identical images, see the parity tests)
    variants = {}
    for name, kw in (("trace_all_rays", dict(trace_all_rays=True)), ("one_kernel", dict(one_kernel=True))):
        ctx.clear_persistent()
        n_var = max(2, min(args.steps, 5))
        for k in range(2):
            ctx.raycast(cam, k)
            ctx.ris_path_trace(cam, k, **ris, **kw)
            ctx.accumulate(k, firefly=True, mode="parity")
        barrier()
        ctx.region_begin(3)
        for k in range(2, 2 + n_var):
            ctx.raycast(cam, k)
            ctx.ris_path_trace(cam, k, **ris, **kw)
            ctx.accumulate(k, firefly=True, mode="parity")
        ctx.region_end(3)
        ms = max_over_ranks(ctx.region_elapsed(3), world) / n_var
        variants[name] = {"frames_per_s": world * 1000.0 / ms, "ms_per_frame": ms, "frames": n_var}
    graph = graph_leg(ctx, cam, ris, world, n_frames=max(2, min(args.steps, 10)))
    ctx.pass_times(reset=True)
    ctx.clear_persistent()
    for k in range(args.warmup):
        frame(k)

    # ---- end to end through the public API: camera from the host, every frame's image back to
    # pinned memory (two host buffers; each frame's read-back overlaps the next frame's passes)
    color_host = [torch.empty((WIDTH * HEIGHT, 4), dtype=torch.float32, pin_memory=True) for _ in range(2)]
    color_np = [t.numpy() for t in color_host]
    barrier()
    ctx.region_begin(2)
    t0 = time.perf_counter()
    for k in range(args.warmup + args.steps, args.warmup + 2 * args.steps):
        frame(k)
        ctx.download_async("Color", color_np[k % 2])
    ctx.download_wait()
    ctx.region_end(2)
    e2e_ms = ctx.region_elapsed(2)
    wall_e2e = time.perf_counter() - t0
    barrier()
    e2e_ms = max_over_ranks(e2e_ms, world)
    e2e_fps = whole_job_rate(args.steps, world, e2e_ms)
    h2d = 2 * len(bytes(cam.c_desc())) + 64  # camera block per camera-taking pass + pass parameters
    d2h = WIDTH * HEIGHT * 16

    if rank != 0:
        ctx.close()
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()
        return None

    peak, peak_kind = measured_peaks()
    px = WIDTH * HEIGHT
    achieved = SHADOW_BYTES_PER_RAY * n_shadow / (t_shadow / 1000.0) / 1e9
    traffic, traffic_src = ncu_traffic("trace_shadow")
    # rays traced per frame: the primary (raycast) rays and the two queues of the last frame
    rays = px + n_closest + n_shadow
    out = {
        "metric": METRIC, "value": fps, "unit": "frames/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32",
        "data": "synthetic seeded config-2 scene (1.03M triangles, 10k rect lights)",
        "config": config_block(),
        "latency_ms": {"p50": statistics.median(frame_ms), "p99": sorted(frame_ms)[
            min(len(frame_ms) - 1, int(round(0.99 * (len(frame_ms) - 1))))], "max": max(frame_ms)},
        "pass_ms": {"raycast": t_ray, "ris_integrate": t_int, "accumulate": t_acc},
        "kernel_ms": {"ris_generate": t_gen, "trace_closest": t_closest, "trace_shadow": t_shadow,
                      "ris_shade": t_shade},
        "rays_per_frame": {"primary": px, "closest": n_closest, "shadow": n_shadow},
        "rays_per_s": rays / (total_ms / args.steps / 1000.0),
        "rays_per_s_note": "rays traced: primary + closest-hit queue + shadow queue of a frame",
        "roofline": {"kernel": "trace_shadow4_kernel (NEE shadow rays, any-hit, 4-wide SAH shadow BVH)",
                     "bound": "hbm",
                     "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                     "peak_kind": peak_kind, "traffic": traffic, "traffic_source": traffic_src,
                     "algorithmic_bytes": SHADOW_BYTES_PER_RAY * n_shadow, "launch_ms": t_shadow,
                     "shadow_rays_per_s": n_shadow / (t_shadow / 1000.0),
                     "note": "algorithmic bytes = 33 B per shadow ray (queue record + occlusion byte); the "
                             "kernel is issue/divergence bound (software BVH traversal), not HBM bound"},
        "roofline_accumulate": {"bound": "hbm", "achieved": ACCUM_BYTES_PER_PX * px / (t_acc / 1000.0) / 1e9,
                                "peak": peak, "unit": "GB/s",
                                "frac": ACCUM_BYTES_PER_PX * px / (t_acc / 1000.0) / 1e9 / peak},
        "e2e": {"value": e2e_fps, "unit": "frames/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                "wall_s": wall_e2e},
        "gpu_launches": gpu_launches,
        "clocks": clk,
        "variants": variants,
        "cuda_graph": graph,
        "note": "default = wavefront (generate/trace/shade); BSDF-candidate rays are not cast in scenes with no "
                "light geometry and no environment, where their result cannot change the image (bit-identical, "
                "tested); 'trace_all_rays' casts them as the reference does",
    }
    if world == 1 and not args.no_serving:
        out["batched"] = batched_leg(ctx)
        out["orbit"] = orbit_leg(ctx)
        out["serving"] = serving_leg(args.serving_jobs)
        out["serving_sustained"] = serving_leg(max(8, args.serving_jobs // 2), rate=8.0)
        out["config3"] = config3_leg()
    if world == 1 and not args.no_cpu_baseline:
        threads = os.cpu_count() or 1
        secs, kind, cpu_color = cpu_frames(scene, cam, range(3), threads)
        value = 2.0 / sum(secs[1:])
        out["mse"] = mse_block(ctx, cam, cpu_color, 3)
        out["cpu_baseline"] = {"value": value, "unit": "frames/s", "cores": threads, "kind": kind,
                               "sample": cpu_sample_label(HEIGHT, "frames 1 and 2 timed after frame 0")}
        for v in out["variants"].values():  # every execution form against the same CPU baseline
            v["vs_cpu_baseline"] = v["frames_per_s"] / value
        out["vs_cpu_baseline"] = {"value": fps / value, "e2e": e2e_fps / value}
    ctx.close()
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()
    return out


def main():
    global WIDTH, HEIGHT
    args = parse()
    WIDTH, HEIGHT = args.width, args.height
    rank, local_rank, world = dist_env()
    if args.impl == "reference":
        out = run_reference(args, rank, world)
    else:
        out = run_ours(args, rank, local_rank, world)
    if out is not None and rank == 0:
        print(json.dumps(out))


if __name__ == "__main__":
    main()
