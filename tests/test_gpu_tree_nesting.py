"""The trees that the closest-hit check reads (ref_reaches, csrc/device/traverse.cuh): it tests a
hit's boxes at the two leaves alone, which stands for the whole path because every inner node's
box is the exact union of its children's. Read back from the resident scene: host and device
BLAS builds, and the TLAS as uploaded and as rebuilt on the device after instances moved."""
import numpy as np
import pytest

from hdrestir_b200 import configs
from hdrestir_b200.context import Context

pytestmark = pytest.mark.gpu

SCENES = {
    "box": lambda: configs.config0(32, 32),
    "boxes": lambda: configs.config1(32, 32, n_lights=8),
    "terrain": lambda: configs.small_variant(2, 32, 32, grid=128, n_spheres=80, n_lights=8),
    "textured": lambda: configs.textured_variant(32, 32),
}


def _nested(nodes, root):
    """Walks the tree at `root`: the inner nodes, whose boxes are their children's union bit for bit."""
    inner, todo = 0, [root]
    while todo:
        n = todo.pop()
        left = nodes[n, 3:4].view(np.int32)[0]
        if left < 0:
            continue
        kids = nodes[root + left: root + left + 2] if root else nodes[left: left + 2]
        lo, hi = kids[:, :3].min(0), kids[:, 4:7].max(0)
        assert np.array_equal(nodes[n, :3], lo) and np.array_equal(nodes[n, 4:7], hi), n
        inner += 1
        todo += [root + left, root + left + 1]
    return inner


def _check(ctx):
    tlas = ctx.scene_array("tlas_nodes").view(np.float32).reshape(-1, 8)
    blas = ctx.scene_array("blas_nodes").view(np.float32).reshape(-1, 8)
    inst = ctx.scene_array("instances").view(np.int32).reshape(-1, 32)
    inner = _nested(tlas, 0)
    for base in sorted({int(r[19]) for r in inst if r[29]}):
        inner += _nested(blas, base)
    return inner


@pytest.mark.parametrize("device_build", [False, True])
@pytest.mark.parametrize("scene", SCENES)
def test_every_box_is_the_union_of_its_childrens(scene, device_build):
    sc, _ = SCENES[scene]()
    with Context(device=0, device_build=device_build) as ctx:
        ctx.upload_scene(sc)
        inner = _check(ctx)
        assert inner > 0
        rng = np.random.default_rng(2)
        xf = np.stack([np.asarray(i.transform, np.float32).reshape(4, 4) for i in sc.instances])
        for move in range(3):
            x = xf.copy()
            x[:, 3, :3] += rng.uniform(-2, 2, (len(x), 3)).astype(np.float32)
            x[:, :3, :3] *= rng.uniform(0.5, 2.0, (len(x), 1, 1)).astype(np.float32)
            if move == 2:
                x[::3, :, 1] = 0.0  # flattened instances
                x[::3, 3, 3] = 1.0
            ctx.set_instance_transforms(x)
            assert _check(ctx) > 0
