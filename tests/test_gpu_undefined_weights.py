"""Frames whose candidate weights are infinite or undefined: the wavefront form, which stores a
light candidate's weight before its shadow ray is cast and does not evaluate the path's bounce,
equals the one-kernel form, which evaluates every candidate after its ray. Near-mirror lobes
(a density that is infinite when the half vector rounds to the normal), throughputs and
emissions past the largest float, environments with an infinite or undefined texel, lights whose
density overflows."""
import numpy as np
import pytest

from hdrestir_b200 import abi, configs
from hdrestir_b200.scene import Light

pytestmark = pytest.mark.gpu


def _materials(**values):
    sc, cam = configs.config1(61, 43, n_lights=24)
    for m in sc.materials:
        for field, v in values.items():
            setattr(m, field, v)
    return sc, cam


def _lights(**values):
    sc, cam = configs.config1(61, 43, n_lights=8)
    for light in sc.lights[::2]:
        for field, v in values.items():
            setattr(light, field, v)
    return sc, cam


def _dome(texel):
    sc, cam = configs.config1(61, 43, n_lights=4)
    tex = np.random.default_rng(3).uniform(0.1, 1.0, (8, 16, 3)).astype(np.float32)
    tex[2, 5] = texel
    sc.lights.append(Light(abi.LIGHT_DOME, color=(1.0, 1.0, 1.0), intensity=1.0, texture=tex))
    return sc, cam


SCENES = {
    "mirror_0.005": lambda: _materials(metallic=1.0, roughness=0.005),
    "mirror_0.012": lambda: _materials(metallic=1.0, roughness=0.012),
    "coat_0.005": lambda: _materials(coat=1.0, coat_roughness=0.005, coat_ior=3.0),
    "sheen_0.004": lambda: _materials(sheen=1.0, sheen_roughness=0.004),
    "colour_3e38": lambda: _materials(diffuse_color=(3e38, 1.0, 1.0)),
    "dome_inf": lambda: _dome(np.inf),
    "dome_nan": lambda: _dome(np.nan),
    "dome_3e38": lambda: _dome(3e38),
    "light_inf": lambda: _lights(intensity=np.inf),
    "light_3e38": lambda: _lights(intensity=3e38),
    "light_tiny": lambda: _lights(width=1e-20, height=1e-20),
    "light_huge": lambda: _lights(width=3e19, height=3e19),
}


def _frames(ctx, cam, **ris):
    out = []
    ctx.clear_persistent()
    for f in range(3):
        ctx.raycast(cam, f)
        ctx.ris_path_trace(cam, f, max_depth=1, **ris)
        out.append(ctx.download("Color").copy())
        if ris["use_reservoir"]:
            out.append(ctx.download("__ris_reservoir").copy())
    return out


@pytest.mark.parametrize("scene", SCENES)
def test_undefined_weights_equal_one_kernel_form(scene):
    from hdrestir_b200.context import Context
    sc, cam = SCENES[scene]()
    with Context(device=0) as ctx:
        ctx.upload_scene(sc)
        for candidates, reservoir in ((1, True), (1, False), (2, True), (2, False), (16, True), (16, False), (76, True)):
            for skip_visibility in (False, True):
                ris = dict(candidate_count=candidates, use_reservoir=reservoir, skip_visibility=skip_visibility)
                want = _frames(ctx, cam, one_kernel=True, **ris)
                got = _frames(ctx, cam, **ris)
                for a, b in zip(got, want):
                    nan = np.isnan(a)
                    assert np.array_equal(nan, np.isnan(b)), ris
                    assert np.array_equal(a.view(np.uint32)[~nan], b.view(np.uint32)[~nan]), ris
