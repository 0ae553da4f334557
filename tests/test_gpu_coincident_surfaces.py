"""Closest hits where surfaces coincide or nearly do: doubled instances, exactly and a few units
in the last place apart, in both orders. The SAH-tree walk with its check gives the reference
walk's hits (every field of them), for rays of every kind the kernels trace."""
import copy

import numpy as np
import pytest

from hdrestir_b200 import configs

pytestmark = pytest.mark.gpu

SCENES = {
    "box": lambda w, h: configs.config0(w, h),
    "boxes": lambda w, h: configs.config1(w, h, n_lights=16),
    "terrain": lambda w, h: configs.small_variant(2, w, h, grid=40, n_spheres=30, n_lights=40),
}


def _doubled(sc, scale, first):
    sc = copy.deepcopy(sc)
    more = copy.deepcopy(sc.instances)
    for i in more:
        t = np.asarray(i.transform, np.float32).copy()
        t[:3, :3] *= np.float32(scale)
        t[3, :3] *= np.float32(scale)
        i.transform = t
    sc.instances = more + sc.instances if first else sc.instances + more
    return sc


def _rays(ctx, cam, n):
    """Rays between surface points that the camera sees, towards random directions, and down axes."""
    ctx.raycast(cam, 0)
    g = ctx.download("GBuffer")
    p = g["position"][g["hit"] == 1]
    rng = np.random.default_rng(11)
    a, b = p[rng.integers(0, len(p), n)], p[rng.integers(0, len(p), n)]
    o = (a + g["normal"][g["hit"] == 1][rng.integers(0, len(p), n)] * 1e-4).astype(np.float32)
    d = np.where(rng.random((n, 1)) < 0.5, b - a, rng.normal(size=(n, 3))).astype(np.float32)
    axis = rng.random(n) < 0.2
    d[axis] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, axis.sum())] * rng.choice([-1.0, 1.0], (axis.sum(), 1))
    d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), np.float32(1e-20))
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.mark.parametrize("first", [False, True])
@pytest.mark.parametrize("ulps", [0, 1, 2, 4, 12, 40])
@pytest.mark.parametrize("scene", SCENES)
def test_coincident_surfaces_give_the_reference_hits(scene, ulps, first):
    from hdrestir_b200.context import Context
    sc, cam = SCENES[scene](96, 64)
    sc = _doubled(sc, 1.0 + ulps * 2.0 ** -23, first)
    with Context(device=0, reference_closest=True) as ref, Context(device=0) as ctx:
        for c in (ref, ctx):
            c.upload_scene(sc)
        rays = _rays(ref, cam, 60_000)
        want, got = ref.trace_rays(rays), ctx.trace_rays(rays)
        assert (want["hit"] == 1).sum() > 10_000
        assert want.tobytes() == got.tobytes()
        ref.raycast(cam, 0), ctx.raycast(cam, 0)
        assert np.array_equal(ref.download("GBuffer").view(np.uint8), ctx.download("GBuffer").view(np.uint8))
        images = []
        for c in (ref, ctx):
            c.path_trace(cam, 0, max_depth=3)
            images.append(c.download("Color").view(np.uint32).copy())
            c.ris_path_trace(cam, 0, candidate_count=8, use_reservoir=True, max_depth=1, trace_all_rays=True)
            images.append(c.download("Color").view(np.uint32).copy())
        assert np.array_equal(images[0], images[2]) and np.array_equal(images[1], images[3])
