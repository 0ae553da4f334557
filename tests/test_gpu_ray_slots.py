"""Frames with 2^31 ray slots or more (pixels times light candidates): the queues number them
with ints, so such a frame takes the one-kernel form, and what has no such form is refused."""
import numpy as np
import pytest

from hdrestir_b200 import abi, configs

pytestmark = pytest.mark.gpu

SIDE, CANDIDATES = 1024, 4096  # 2^20 pixels, 2^11 light candidates each


def test_frames_of_too_many_ray_slots():
    from hdrestir_b200.context import Context
    sc, _ = configs.config1(64, 48, n_lights=8)
    away = configs.make_camera((0.0, 6.0, 9.0), (0.0, 6.02, 18.0), SIDE, SIDE, fov=70.0)
    assert SIDE * SIDE * (CANDIDATES // 2) == 2 ** 31
    ris = dict(candidate_count=CANDIDATES, use_reservoir=True, max_depth=1)
    with Context(device=0, hbm_budget=1 << 30) as ctx:
        ctx.upload_scene(sc)
        ctx.raycast(away, 0)
        ctx.ris_path_trace(away, 0, **ris)
        got = ctx.download("Color").copy()
        ctx.ris_path_trace(away, 0, one_kernel=True, **ris)
        assert np.array_equal(got.view(np.uint32), ctx.download("Color").view(np.uint32))
        with pytest.raises(abi.HdrError, match="2\\^31 ray slots"):
            ctx.ris_path_trace(away, 0, spatial_neighbors=2, **ris)
        with pytest.raises(abi.HdrError, match="2\\^31 ray slots"):
            ctx.autotune_frame(away, 0, **ris)
    with Context(device=0, hbm_budget=1 << 30, record_lights=True) as ctx:
        ctx.upload_scene(sc)
        ctx.raycast(away, 0)
        with pytest.raises(abi.HdrError, match="2\\^31 ray slots"):
            ctx.ris_path_trace(away, 0, **ris)
