"""hdr_autotune_trace runs the trace kernels on the last wavefront frame's queues. A frame that
is refused after some of those queues were replaced leaves none to run on."""
import numpy as np
import pytest

from hdrestir_b200 import abi, configs

pytestmark = pytest.mark.gpu

RIS = dict(candidate_count=16, use_reservoir=True, max_depth=1)


def test_autotune_after_a_frame_that_replaced_queues_and_failed():
    from hdrestir_b200.context import Context
    sc, small = configs.config1(48, 32, n_lights=40)
    large = configs.config_camera(1, 160, 120)
    with Context(device=0) as ctx:  # the budgets between "no larger frame" and "all of it"
        ctx.upload_scene(sc)
        ctx.raycast(small, 0)
        ctx.ris_path_trace(small, 0, **RIS)
        before = ctx.buffer_size("__wave_q_shadow")
        ctx.autotune_trace()
    refused = 0
    for budget in np.linspace(2 << 20, 40 << 20, 96).astype(int):
        with Context(device=0, hbm_budget=int(budget)) as ctx:
            try:
                ctx.upload_scene(sc)
                ctx.raycast(small, 0)
                ctx.ris_path_trace(small, 0, **RIS)
            except abi.HdrError:
                continue
            try:
                ctx.raycast(large, 0)
                ctx.ris_path_trace(large, 0, **RIS)
            except abi.HdrError:
                if ctx.buffer_size("__wave_q_shadow") == before:
                    continue  # refused before a queue was replaced
                refused += 1
                with pytest.raises(abi.HdrError, match="previous wavefront"):
                    ctx.autotune_trace()
                continue
            ctx.autotune_trace()
    assert refused > 0
