"""Resampling from stored light-candidate weights (csrc/wavefront.cu) against the one-kernel
form, which generates and evaluates every candidate in place: images and reservoirs byte for
byte, at the sizes where the two could part: one candidate, odd counts, the last count whose
streams travel between the kernels and the first whose do not, streams past 311 draws, lights
that draw different numbers, the plain form's largest candidate list, odd image sizes."""
import numpy as np
import pytest

from hdrestir_b200 import configs

pytestmark = pytest.mark.gpu

SCENES = {
    "terrain": lambda w, h: configs.small_variant(2, w, h, grid=48, n_spheres=60, n_lights=300),
    "boxes": lambda w, h: configs.config1(w, h, n_lights=40),
    "mixed_lights": lambda w, h: configs.mixed_lights(w, h),
    "textured": lambda w, h: configs.textured_variant(w, h),
}


def _frames(ctx, cam, n, **ris):
    out = []
    ctx.clear_persistent()
    for f in range(n):
        ctx.raycast(cam, f)
        ctx.ris_path_trace(cam, f, max_depth=1, **ris)
        out.append(ctx.download("Color").copy())
        if ris["use_reservoir"]:
            out.append(ctx.download("__ris_reservoir").copy())
    return out


@pytest.mark.parametrize("scene,width,height,candidates,reservoir,skip_visibility", [
    ("terrain", 61, 43, 32, True, False),
    ("terrain", 16, 16, 1, True, False),
    ("terrain", 33, 9, 3, True, True),
    ("terrain", 40, 24, 74, True, False),
    ("terrain", 40, 24, 76, True, False),
    ("terrain", 24, 16, 220, True, False),
    ("boxes", 37, 29, 64, False, False),
    ("boxes", 37, 29, 1, False, True),
    ("boxes", 50, 31, 16, False, True),
    ("mixed_lights", 45, 27, 16, True, False),
    ("mixed_lights", 45, 27, 15, False, False),
    ("textured", 39, 25, 32, True, False),
])
def test_resampling_equals_one_kernel_form(scene, width, height, candidates, reservoir, skip_visibility):
    from hdrestir_b200.context import Context
    sc, cam = SCENES[scene](width, height)
    ris = dict(candidate_count=candidates, use_reservoir=reservoir, skip_visibility=skip_visibility)
    with Context(device=0) as ctx:
        ctx.upload_scene(sc)
        want = _frames(ctx, cam, 3, one_kernel=True, **ris)
        for shape in range(4):
            ctx.set_trace_tuning(12, 16, shape, 0)
            got = _frames(ctx, cam, 3, **ris)
            assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(got, want))
        assert any(np.abs(a[:, :3]).sum() > 0 for a in want if a.ndim == 2)


def test_budget_without_room_for_the_weights():
    """A frame for which everything but the light candidates' weights fits the context's budget
    renders all the same, with the same image; with nothing to spare it is refused."""
    from hdrestir_b200.context import Context
    sc, cam = SCENES["terrain"](64, 48)
    ris = dict(candidate_count=32, use_reservoir=True, skip_visibility=False)

    def frames(budget):
        with Context(device=0, hbm_budget=budget) as ctx:
            try:
                ctx.upload_scene(sc)
                out = _frames(ctx, cam, 2, **ris)
            except RuntimeError:
                return None, None
            try:
                return out, ctx.buffer_size("__wave_nee_weight")
            except RuntimeError:
                return out, 0

    want, weights = frames(0)
    assert weights == 64 * 48 * 16 * 4
    lo, hi = 1, 1 << 28  # refused, enough
    assert frames(lo)[0] is None
    while hi - lo > 1024:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if frames(mid)[0] is not None else (mid, hi)
    for budget, held in ((hi, 0), (hi + weights // 2, 0), (hi + weights, weights)):
        got, have = frames(budget)
        assert have == held
        assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(got, want))


def test_recording_whose_weights_cannot_grow():
    """Recorded after frames with a reservoir, a frame without one needs larger weights, which a
    recording cannot allocate: it is recorded in the one-kernel form."""
    from hdrestir_b200.context import Context
    sc, cam = SCENES["boxes"](40, 24)
    ris = dict(candidate_count=16, max_depth=1, skip_visibility=False)
    with Context(device=0) as ctx, Context(device=0) as plain:
        for c in (ctx, plain):
            c.upload_scene(sc)
            c.raycast(cam, 0)
        ctx.ris_path_trace(cam, 0, use_reservoir=True, **ris)
        ctx.graph_begin()
        ctx.raycast(cam, 1)
        ctx.ris_path_trace(cam, 1, use_reservoir=False, **ris)
        ctx.graph_end()
        ctx.graph_launch(1)
        plain.raycast(cam, 1)
        plain.ris_path_trace(cam, 1, use_reservoir=False, **ris)
        assert np.array_equal(ctx.download("Color").view(np.uint32), plain.download("Color").view(np.uint32))
