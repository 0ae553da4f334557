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
