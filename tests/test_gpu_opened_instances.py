"""Instances whose nodes are opened into the SAH trees' top level (host/shadow_bvh.h): the
walks' answers against the reference walk of the reference's trees, on scenes where opening
meets its edges: meshes with one triangle or none, several instances of one mesh of which
only some have the identity transform, flat meshes, coordinates far from the origin, more
nodes than are opened, and instances that become or stop being the identity by moving.
Closest hits must equal the reference walk's byte for byte. Shadow answers must equal an
exhaustive test of every triangle: IntersectTriangle (bvh.cpp:8-30) in float32 on the
instance-space ray, which is what the walk promises (the reference's own walk also misses
hits that its rounded box tests cull, and many of these rays run through vertices and faces)."""
import numpy as np
import pytest

from hdrestir_b200 import configs
from hdrestir_b200.scene import Instance, Material, Mesh, Scene

pytestmark = pytest.mark.gpu


def _tri(k, shift=0.0):
    rng = np.random.default_rng(k)
    p = rng.uniform(-1, 1, (3, 3)) + np.array([shift, 0.0, 0.0])
    return Mesh(p.astype(np.float32), np.array([[0, 1, 2]], np.int32))


def _move(t, scale=1.0):
    m = np.eye(4) * scale
    m[3] = [*t, 1.0]
    return m


def _scene(kind):
    sc = Scene(name=kind)
    sc.materials.append(Material())

    def add(mesh, *transforms):
        sc.meshes.append(mesh)
        for t in transforms:
            sc.instances.append(Instance(len(sc.meshes) - 1, t, 0))

    if kind == "one_triangle":
        add(_tri(1), np.eye(4))
    elif kind == "single_triangles":  # every mesh one triangle, all opened
        for k in range(40):
            add(_tri(k, shift=0.2 * (k % 7)), np.eye(4))
    elif kind == "empty_meshes":
        add(Mesh(np.zeros((3, 3), np.float32), np.zeros((0, 3), np.int32)), np.eye(4), _move((1, 0, 0)))
        add(configs.sphere_mesh(8, 5), np.eye(4))
        add(Mesh(np.zeros((3, 3), np.float32), np.zeros((0, 3), np.int32)), np.eye(4))
    elif kind == "shared_mesh":  # the first identity instance is opened, its twin and the moved ones are not
        add(configs.sphere_mesh(), _move((2.0, 0, 0), 0.5), np.eye(4), np.eye(4), _move((-2.0, 0.5, 0), 0.7))
        add(configs.box_mesh((-1, -1.5, -1), (1, -1, 1)), np.eye(4), _move((0, 2.5, 0)))
    elif kind == "flat":  # zero extents, coplanar with each other
        p, i = configs.quad((-3, 0, -3), (-3, 0, 3), (3, 0, 3), (3, 0, -3))
        add(Mesh(p, i), np.eye(4), _move((0, 1, 0)))
        add(configs.box_mesh((-1, 0, -1), (1, 1, 1)), np.eye(4))
    elif kind == "far":  # large coordinates, small extents
        s = configs.sphere_mesh(12, 7)
        add(Mesh(s.points * 0.3 + np.array([3000.0, -2000.0, 500.0], np.float32), s.indices), np.eye(4))
        add(s, _move((3000.5, -2000.0, 500.0), 0.2))
    else:  # more nodes than are opened
        h = configs.value_noise(160, np.random.default_rng(3)) * 2.0
        add(configs.grid_mesh(160, 6.0, h), np.eye(4))
        rng = np.random.default_rng(4)
        add(configs.sphere_mesh(8, 5), *[_move(rng.uniform(-5, 5, 3) * [1, 0.2, 1] + [0, 2, 0], 0.3) for _ in range(30)])
    return sc


def _rays(sc, n, rng):
    pts = []
    for inst in sc.instances:
        p = sc.meshes[inst.mesh].points
        if len(sc.meshes[inst.mesh].indices):
            pts.append((np.concatenate([p, np.ones((len(p), 1))], 1) @ np.asarray(inst.transform, np.float64))[:, :3])
    pts = np.concatenate(pts)
    lo, hi = pts.min(0), pts.max(0)
    ext = np.maximum(hi - lo, 0.5)
    o = rng.uniform(lo - ext, hi + ext, (n, 3))
    to = pts[rng.integers(0, len(pts), n)] + rng.normal(scale=0.15, size=(n, 3)) * ext
    to[: n // 8] = pts[rng.integers(0, len(pts), n // 8)]  # through vertices
    d = to - o
    d[n // 8: n // 5, 1] = 0.0
    d[n // 5: n // 4, ::2] = 0.0
    length = np.linalg.norm(d, axis=1, keepdims=True)
    d /= np.maximum(length, 1e-9)
    return (np.concatenate([o, d], 1).astype(np.float32),
            (length[:, 0] * rng.uniform(0.5, 1.5, n)).astype(np.float32))


def _blocked(ctx, sc, rays, lim):
    """Any triangle with t < limit, every triangle of every instance tested."""
    f = np.float32
    records = ctx.scene_array("instances").view(f).reshape(-1, 32)
    out = np.zeros(len(rays), bool)
    o, d = rays[:, :3], rays[:, 3:]

    def dot(a, b):
        return (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]) + a[..., 2] * b[..., 2]

    def cross(a, b):
        return np.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1], a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                         a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)

    for inst, rec in zip(sc.instances, records):
        mesh = sc.meshes[inst.mesh]
        if not len(mesh.indices):
            continue
        m = rec[:16].reshape(4, 4)
        q = [((o[:, 0] * m[0, c] + o[:, 1] * m[1, c]) + o[:, 2] * m[2, c]) + m[3, c] for c in range(4)]
        inv_w = f(1.0) / q[3]
        oo = np.stack([inv_w * q[c] for c in range(3)], 1)
        od = np.stack([(d[:, 0] * m[0, c] + d[:, 1] * m[1, c]) + d[:, 2] * m[2, c] for c in range(3)], 1)
        v0, v1, v2 = (mesh.points[mesh.indices[:, k]] for k in range(3))
        e1, e2 = v1 - v0, v2 - v0
        for at in range(0, len(e1), 4096):
            a0, a1, a2 = v0[None, at:at + 4096], e1[None, at:at + 4096], e2[None, at:at + 4096]
            p = cross(od[:, None], a2)
            det = dot(a1, p)
            with np.errstate(all="ignore"):
                inv = f(1.0) / det
                t = oo[:, None] - a0
                u = dot(t, p) * inv
                r = cross(t, a1)
                v = dot(od[:, None], r) * inv
                dist = dot(a2, r) * inv
            out |= ((np.abs(det).astype(np.float64) >= 1e-8) & ~((u < 0) | (u > 1)) & ~((v < 0) | (u + v > 1))
                    & (dist > f(1e-4)) & (dist < lim[:, None])).any(1)
    return out


def _compare(ctx, ref, sc, rays, lim):
    got, want = ctx.trace_rays(rays), ref.trace_rays(rays)
    assert np.array_equal(got.view(np.uint8), want.view(np.uint8))
    few = slice(None, None, 60)
    rays, lim = np.ascontiguousarray(rays[few]), np.ascontiguousarray(lim[few])
    assert np.array_equal(ctx.trace_stats(rays, 4, lim)[:, 3] != 0, _blocked(ctx, sc, rays, lim))
    return int((want["hit"] == 1).sum())


KINDS = ["one_triangle", "single_triangles", "empty_meshes", "shared_mesh", "flat", "far", "many_nodes"]


@pytest.mark.parametrize("kind", KINDS)
def test_answers_equal_the_reference_walk(kind):
    from hdrestir_b200.context import Context
    sc = _scene(kind)
    rays, lim = _rays(sc, 60_000, np.random.default_rng(11))
    with Context(device=0) as ctx, Context(device=0, reference_closest=True) as ref:
        ctx.upload_scene(sc)
        ref.upload_scene(sc)
        assert _compare(ctx, ref, sc, rays, lim) > 0


def test_instances_that_become_and_stop_being_the_identity():
    from hdrestir_b200.context import Context
    sc = _scene("shared_mesh")
    rng = np.random.default_rng(12)
    here = [np.asarray(i.transform, np.float32) for i in sc.instances]
    swapped = [here[1], here[0], _move((0.3, 0, 1.5), 0.6), np.eye(4), _move((0, 0.1, 0)), np.eye(4)]
    none = [_move((0.1 * k, 0, 0), 0.9) for k in range(len(here))]
    with Context(device=0) as ctx, Context(device=0, reference_closest=True) as ref:
        ctx.upload_scene(sc)
        ref.upload_scene(sc)
        for transforms in (swapped, none, here):
            xf = np.stack([np.asarray(t, np.float32) for t in transforms])
            ctx.set_instance_transforms(xf)
            ref.set_instance_transforms(xf)
            for inst, t in zip(sc.instances, transforms):
                inst.transform = np.asarray(t, np.float64)
            rays, lim = _rays(sc, 40_000, rng)
            assert _compare(ctx, ref, sc, rays, lim) > 0
