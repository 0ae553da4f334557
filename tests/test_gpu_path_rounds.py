"""The wavefront PathTracePass, whose rounds connect a vertex and sample the next in one kernel
and trace both ray queues in one launch, against the one-thread form, byte for byte: depth 1,
depths of either parity (the active lists and their counters swap every round), streams that
are finished in a thread, scenes whose last bounce cannot meet light and scenes where it can."""
import numpy as np
import pytest

from hdrestir_b200 import configs
from hdrestir_b200.scene import Material

pytestmark = pytest.mark.gpu


def _scene(kind, w, h):
    if kind == "box":
        return configs.config0(w, h)
    if kind == "dome":
        sc, cam, _ = configs.config3(w, h, n_small=1, small=8, grid=48, n_spheres=40, n_lights=50, dome_size=(64, 32))
        return sc, cam
    sc, cam = configs.small_variant(2, w, h, grid=48, n_spheres=40, n_lights=50)
    if kind == "emissive":
        sc.materials[1] = Material(emission=3.0, emission_color=(1.0, 0.5, 0.2))
    return sc, cam


@pytest.mark.parametrize("kind,w,h,depth", [
    ("box", 33, 17, 1), ("box", 64, 48, 2), ("box", 65, 31, 3), ("box", 40, 30, 32), ("terrain", 57, 23, 4),
    ("terrain", 16, 1, 5), ("emissive", 40, 24, 2), ("emissive", 40, 24, 3), ("dome", 45, 28, 1), ("dome", 45, 28, 16),
])
def test_rounds_equal_one_thread_form(kind, w, h, depth):
    from hdrestir_b200.context import Context, path_trace_batch
    sc, cam = _scene(kind, w, h)
    with Context(device=0) as a, Context(device=0, pt_one_kernel=True) as b, Context(device=0) as c:
        a.upload_scene(sc)
        b.upload_scene(sc)
        c.share_scene(a)
        want = []
        for f in (0, 7):
            for ctx in (a, b):
                ctx.raycast(cam, f)
                ctx.path_trace(cam, f, max_depth=depth)
            want.append(b.download("Color").copy())
            assert np.array_equal(a.download("Color").view(np.uint32), want[-1].view(np.uint32))
        a.raycast(cam, 0)
        c.raycast(cam, 7)
        path_trace_batch([a, c], [cam, cam], [0, 7], max_depth=depth)
        for ctx, img in zip((a, c), want):
            assert np.array_equal(ctx.download("Color").view(np.uint32), img.view(np.uint32))


@pytest.mark.parametrize("depth", [63, 64, 65, 66, 130])
def test_many_rounds(depth):
    """A lightless box of mirrors with one glowing material: two draws a vertex, so paths live
    for 122 rounds, past the rounds' last block of counters."""
    from hdrestir_b200.context import Context
    sc, cam = configs.config0(24, 17)
    sc.lights = []
    for k, m in enumerate(sc.materials):
        m.metallic, m.roughness, m.diffuse_color = 1.0, 0.0, (1.0, 1.0, 1.0)
        m.emission = 0.5 if k == 0 else 0.0
    images = []
    for one in (False, True):
        with Context(device=0, pt_one_kernel=one) as ctx:
            ctx.upload_scene(sc)
            ctx.raycast(cam, 3)
            for _ in range(2):  # the counters a frame leaves are the next frame's start
                ctx.path_trace(cam, 3, max_depth=depth, max_reflection_bounces=1000, roulette_aggressiveness=1e6)
            images.append(ctx.download("Color").copy())
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
    assert np.abs(images[0][:, :3]).sum() > 0
