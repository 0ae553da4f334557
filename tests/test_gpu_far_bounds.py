"""Scenes near and past the coordinates that the 4-wide SAH trees serve (kSh4MaxBound,
csrc/host/shadow_bvh.cpp): rays along an axis, whose other two slabs the walk tests with the
reciprocal of the smallest direction, get the reference walk's answers."""
import numpy as np
import pytest

from hdrestir_b200.scene import Instance, Material, Mesh, Scene

pytestmark = pytest.mark.gpu


def _ground(extent):
    h = extent / 2
    points = np.float32([[-h, 0, -h], [-h, 0, h], [h, 0, h], [h, 0, -h]])
    return Scene(meshes=[Mesh(points, np.int32([[0, 1, 2], [0, 2, 3]]))], materials=[Material()],
                 instances=[Instance(0, np.eye(4), 0)])


def _rays(extent):
    at = np.stack(np.meshgrid(np.linspace(-0.499, 0.499, 16), np.linspace(-0.499, 0.499, 16)), -1).reshape(-1, 2) * extent
    o = np.stack([at[:, 0], np.full(len(at), 1e3), at[:, 1]], 1)
    down = np.concatenate([o, np.tile([0.0, -1.0, 0.0], (len(at), 1))], 1)
    slant = np.concatenate([o, np.tile([1e-12, -1.0, -1e-12], (len(at), 1))], 1)
    return np.concatenate([down, slant]).astype(np.float32)


@pytest.mark.parametrize("extent", [2.0, 1e12, 1.9e16, 1.99e16, 2.01e16] + list(np.linspace(2.58e16, 2.68e16, 11)) + [1e19])
def test_axis_rays_over_a_far_ground(extent):
    from hdrestir_b200.context import Context
    sc, rays = _ground(extent), _rays(extent)
    limit = np.full(len(rays), 1e30, np.float32)
    answers = []
    for flags in (dict(reference_shadows=True, reference_closest=True), {}, dict(sah_closest=True)):
        with Context(device=0, **flags) as ctx:
            ctx.upload_scene(sc)
            answers.append((ctx.trace_rays(rays), ctx.trace_rays(rays, limit, any_hit=True)))
    want = answers[0]
    assert (want[0]["hit"] == 1).all() or extent > 1e18  # past it the triangle test itself overflows
    for got in answers[1:]:
        for a, b in zip(got, want):
            assert np.array_equal(a["hit"], b["hit"])
        assert np.array_equal(got[0]["depth"], want[0]["depth"])
