"""The resampling kernel's launch shape: frames that the general kernel shades have none to
choose, so autotuning them leaves the chosen one; setting only the schedule leaves it too."""
import numpy as np
import pytest

from hdrestir_b200 import abi, configs
from hdrestir_b200.scene import Light

pytestmark = pytest.mark.gpu


def test_shade_shape_stays():
    from hdrestir_b200.context import Context
    sc, cam = configs.config1(64, 48, n_lights=8)
    sc.lights.append(Light(abi.LIGHT_DOME, texture=np.full((4, 8, 3), 0.5, np.float32)))
    with Context(device=0) as ctx:
        ctx.upload_scene(sc)
        ctx.raycast(cam, 0)
        first = ctx.trace_tuning()
        ctx.set_trace_tuning(first["node_quorum"], 6)
        assert ctx.trace_tuning() == {**first, "blocks_per_sm": 6}
        for shape in (0, 1, 2, 3, 1, 0):
            ctx.set_trace_tuning(12, 8, shape)
            best = ctx.autotune_frame(cam, 0, candidate_count=8, use_reservoir=True, max_depth=1)
            assert best["shade_ms"] > 0.0
            assert best["shade_shape"] == ctx.trace_tuning()["shade_shape"] == shape
