"""Frames for which everything but the light candidates' weights fits a context's budget: every
form of a wavefront RIS frame renders without them and gives the frame that has them (spatial
reuse, reprojection, recorded light indices, autotuning, general and lean resampling). The weights
give way to buffers that come after them (accumulation, rays traced for a query)."""
import numpy as np
import pytest

from hdrestir_b200 import abi, configs
from hdrestir_b200.scene import Light

pytestmark = pytest.mark.gpu


def _dome(w, h):
    sc, cam = configs.config1(w, h, n_lights=12)
    tex = np.random.default_rng(5).uniform(0.05, 1.0, (8, 16, 3)).astype(np.float32)
    sc.lights.append(Light(abi.LIGHT_DOME, color=(1.0, 1.0, 1.0), intensity=1.0, texture=tex))
    return sc, cam


SCENES = {"boxes": lambda w, h: configs.config1(w, h, n_lights=40), "dome": _dome,
          "textured": lambda w, h: configs.textured_variant(w, h)}
FORMS = {
    "plain": dict(candidate_count=16, use_reservoir=False),
    "reservoir": dict(candidate_count=32, use_reservoir=True),
    "skip_visibility": dict(candidate_count=16, use_reservoir=True, skip_visibility=True),
    "long_streams": dict(candidate_count=80, use_reservoir=True),
    "reproject": dict(candidate_count=16, use_reservoir=True, reproject=True),
    "spatial": dict(candidate_count=16, use_reservoir=True, spatial_neighbors=3),
    "lights": dict(candidate_count=16, use_reservoir=True),
    "autotune": dict(candidate_count=16, use_reservoir=True),
    "accumulate": dict(candidate_count=16, use_reservoir=True),
    "trace_rays": dict(candidate_count=16, use_reservoir=True),
}


@pytest.mark.parametrize("scene,form", [("boxes", f) for f in FORMS] + [
    ("dome", "plain"), ("dome", "reservoir"), ("dome", "spatial"), ("textured", "spatial")])
def test_frames_without_room_for_the_weights(scene, form):
    from hdrestir_b200.context import Context
    sc, cam = SCENES[scene](48, 40)
    ris = dict(skip_visibility=False, max_depth=1)
    ris.update(FORMS[form])

    def frames(budget):
        out = []
        with Context(device=0, hbm_budget=budget, record_lights=form == "lights") as ctx:
            try:
                ctx.upload_scene(sc)
                for f in range(2):
                    ctx.raycast(cam, f)
                    if form == "autotune":
                        ctx.autotune_frame(cam, f, **ris)
                    else:
                        ctx.ris_path_trace(cam, f, **ris)
                    if form == "accumulate":
                        ctx.accumulate(f, firefly=True, mode="parity")
                    if form == "trace_rays":
                        ctx.trace_rays(np.tile(np.float32([0, 5, 0, 0, -1, 0]), (400, 1)))
                    names = ["Color"] + ["__ris_reservoir"] * ris["use_reservoir"] + ["__ris_nee_lights"] * (form == "lights")
                    out += [ctx.download(n).copy() for n in names]
            except abi.HdrError:
                return None, None
            try:
                return out, ctx.buffer_size("__wave_nee_weight" + "_plain" * (not ris["use_reservoir"]))
            except abi.HdrError:
                return out, 0

    want, weights = frames(0)
    size = 4 if ris["use_reservoir"] else 8
    assert weights >= 48 * 40 * (ris["candidate_count"] // 2) * size
    lo, hi = 1, 1 << 28  # refused, enough
    while hi - lo > 1024:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if frames(mid)[0] is not None else (mid, hi)
    got, held = frames(hi)
    assert held == 0
    for a, b in zip(got, want):
        nan = np.isnan(a) if a.dtype == np.float32 else np.zeros(a.shape, bool)
        assert np.array_equal(a.view(np.uint8 if a.dtype == np.uint8 else np.uint32)[~nan],
                              b.view(np.uint8 if b.dtype == np.uint8 else np.uint32)[~nan])
    assert any(np.nan_to_num(np.abs(a[:, :3])).sum() > 0 for a in want if a.ndim == 2)


def test_replacing_the_weights_themselves_when_they_give_way():
    """A buffer of that name whose larger replacement only fits once the old one is given back."""
    from hdrestir_b200.context import Context
    sc, cam = SCENES["boxes"](48, 40)
    ris = dict(candidate_count=16, use_reservoir=True, max_depth=1)
    done = 0
    for budget in np.linspace(2 << 20, 6 << 20, 60).astype(int):
        with Context(device=0, hbm_budget=int(budget)) as ctx:
            try:
                ctx.upload_scene(sc)
                ctx.raycast(cam, 0)
                ctx.ris_path_trace(cam, 0, **ris)
                held = ctx.buffer_size("__wave_nee_weight")
            except abi.HdrError:
                continue
            try:
                ctx.upload("__wave_nee_weight", np.zeros(held + 4096, np.uint8))
                done += 1
                assert ctx.buffer_size("__wave_nee_weight") == held + 4096
            except abi.HdrError:
                pass
            ctx.ris_path_trace(cam, 1, **ris)
            ctx.synchronize()
    assert done > 0
