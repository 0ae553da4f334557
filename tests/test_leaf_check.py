"""The closest-hit check tests a hit's boxes only at the two leaves that hold it
(ref_reaches, csrc/device/traverse.cuh). That equals testing every box on the way down
because a box that contains another passes the reference's slab test wherever the inner one
does, and no farther along the ray: IntersectAABB (scene.cpp:16-47, bvh.cpp:32-64) restated
in float32, as the kernels evaluate it, on nested boxes and rays that graze their faces."""
import numpy as np
import pytest

f32 = np.float32


def slab(o, d, lo, hi, double_thresholds):
    a = np.abs(d)
    small = (a.astype(np.float64) < 1e-8) if double_thresholds else (a < f32(1e-8))
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        inv = (f32(1.0) / d).astype(f32)
        t1 = ((lo - o).astype(f32) * inv).astype(f32)
        t2 = ((hi - o).astype(f32) * inv).astype(f32)
    near = np.where(small, f32(-1e30), np.minimum(t1, t2)).max(1)
    far = np.where(small, f32(1e30), np.maximum(t1, t2)).min(1)
    near, far = np.maximum(near, f32(-1e30)), np.minimum(far, f32(1e30))
    outside = (small & ((o < lo) | (o > hi))).any(1)
    return ~outside & ~(near > far) & (far > f32(1e-4)), near


def cases(kind, n, rng):
    lo = rng.uniform(-20, 20, (n, 3)).astype(f32)
    hi = (lo + rng.exponential(1.0, (n, 3)).astype(f32)).astype(f32)
    if kind == "flat":  # leaves of axis-aligned faces
        hi[:, 0] = lo[:, 0]
    o = rng.uniform(-25, 25, (n, 3)).astype(f32)
    target = (lo + (hi - lo) * rng.uniform(0, 1, (n, 3)).astype(f32)).astype(f32)
    if kind == "graze":  # rays through corners and edges, and starting on faces
        pick = rng.integers(0, 3, (n, 3))
        target = np.where(pick == 0, lo, np.where(pick == 1, hi, target)).astype(f32)
        o[: n // 2, 1] = target[: n // 2, 1]
    if kind == "parallel":  # origins inside the slabs that the parallel axes below only compare
        o[: n // 2, 1] = target[: n // 2, 1]
        o[n // 3:, 2] = target[n // 3:, 2]
    d = (target - o).astype(f32)
    d = (d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), f32(1e-20))).astype(f32)
    if kind == "parallel":  # one or two axes at or near the threshold
        d[: n // 2, 1] = 0.0
        d[n // 3:, 2] = rng.choice([0.0, 9e-9, -1e-8, 1.1e-8, 1e-12], len(d) - n // 3).astype(f32)
    # ancestors: the exact union with other boxes, each side grown or kept
    grow = np.where(rng.random((n, 6)) < 0.5, 0.0, rng.exponential(2.0, (n, 6))).astype(f32)
    return o, d, lo, hi, (lo - grow[:, :3]).astype(f32), (hi + grow[:, 3:]).astype(f32)


@pytest.mark.parametrize("double_thresholds", [False, True])
@pytest.mark.parametrize("kind", ["plain", "flat", "graze", "parallel"])
def test_an_ancestor_passes_where_the_leaf_passes(kind, double_thresholds):
    rng = np.random.default_rng([len(kind), int(double_thresholds)])
    o, d, lo, hi, plo, phi = cases(kind, 400_000, rng)
    leaf, t_leaf = slab(o, d, lo, hi, double_thresholds)
    parent, t_parent = slab(o, d, plo, phi, double_thresholds)
    assert leaf.sum() > 10_000
    assert parent[leaf].all()
    assert (t_parent[leaf] <= t_leaf[leaf]).all()
