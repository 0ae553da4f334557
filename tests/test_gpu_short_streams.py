"""Streams whose draws end before word 156 of the generator's first block take a form of their
own (MtShort, csrc/device/rng.cuh). Around the sizes where the general form takes over, and with
a lens and materials that draw the most (coat, sheen, roughness), the images equal those of the
one-thread forms, which always use the general stream, byte for byte."""
import numpy as np
import pytest

from hdrestir_b200 import configs

pytestmark = pytest.mark.gpu

LENS = dict(enable_dof=1, focal_length=50.0, f_stop=1.4, focus_distance=12.0, bokeh_blades=6)


def _scene(w, h, lens, box=False):
    sc, cam = configs.config0(w, h) if box else configs.small_variant(2, w, h, grid=48, n_spheres=60, n_lights=80)
    for m in sc.materials:
        m.coat, m.coat_roughness, m.sheen, m.sheen_roughness, m.roughness = 0.5, 0.3, 0.5, 0.4, 0.4
    if lens:
        cam.params = LENS
    return sc, cam


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("lens", [False, True])
@pytest.mark.parametrize("candidates", [2, 32, 35, 36, 37, 38])  # 36: 154 draws at most, 37: 159
def test_candidate_generation(candidates, lens):
    from hdrestir_b200.context import Context
    sc, cam = _scene(45, 27, lens)
    with Context(device=0) as ctx:
        ctx.upload_scene(sc)
        for f in range(2):
            ctx.raycast(cam, f)
            images = []
            for one in (True, False):
                ctx.clear_persistent()
                ctx.ris_path_trace(cam, f, max_depth=1, candidate_count=candidates, use_reservoir=True, one_kernel=one)
                images.append(ctx.download("Color").copy())
            assert _same(*images)


@pytest.mark.parametrize("lens", [False, True])
@pytest.mark.parametrize("depth", [1, 14, 15, 16, 17, 20])
def test_path_rounds(depth, lens):
    from hdrestir_b200.context import Context
    sc, cam = _scene(33, 21, lens, box=True)  # closed: paths reach their last vertex
    with Context(device=0) as a, Context(device=0, pt_one_kernel=True) as b:
        for f in range(2):
            images = []
            for ctx in (a, b):
                if f == 0:
                    ctx.upload_scene(sc)
                ctx.raycast(cam, f)
                ctx.path_trace(cam, f, max_depth=depth, max_reflection_bounces=64, roulette_aggressiveness=1000.0)
                images.append(ctx.download("Color").copy())
            assert _same(*images)
