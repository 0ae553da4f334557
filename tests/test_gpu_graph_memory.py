"""A recorded graph and the memory it uses: eager frames that share none of the recorded buffers
leave it as it was, and once one of its buffers or its scene has been replaced hdr_graph_launch
refuses instead of running on freed memory."""
import numpy as np
import pytest

from hdrestir_b200 import abi, configs

pytestmark = pytest.mark.gpu

RIS = dict(candidate_count=16, max_depth=1, skip_visibility=False)


def _frame(ctx, cam, f, reservoir):
    ctx.raycast(cam, f)
    ctx.ris_path_trace(cam, f, use_reservoir=reservoir, **RIS)


def _bits(ctx, name="Color"):
    return ctx.download(name).view(np.uint32).copy()


@pytest.mark.parametrize("recorded", [True, False])
def test_a_frame_of_the_other_kind_leaves_the_recording_valid(recorded):
    """Weights of 4 bytes with a reservoir, 8 without: an eager frame of either kind between a
    recording of the other and its launch."""
    from hdrestir_b200.context import Context
    sc, cam = configs.config1(61, 43, n_lights=40)
    with Context(device=0) as ctx, Context(device=0) as plain:
        for c in (ctx, plain):
            c.upload_scene(sc)
            _frame(c, cam, 0, recorded)
        ctx.graph_begin()
        _frame(ctx, cam, 1, recorded)
        ctx.graph_end()
        ctx.graph_launch(1)
        _frame(plain, cam, 1, recorded)
        assert np.array_equal(_bits(ctx), _bits(plain))
        for c in (ctx, plain):
            _frame(c, cam, 2, not recorded)
        assert np.array_equal(_bits(ctx), _bits(plain))
        ctx.graph_launch(3)
        _frame(plain, cam, 3, recorded)
        assert np.array_equal(_bits(ctx), _bits(plain))
        assert np.array_equal(_bits(ctx, "__ris_reservoir"), _bits(plain, "__ris_reservoir"))


def _recorded(ctx, sc, cam):
    ctx.upload_scene(sc)
    _frame(ctx, cam, 0, True)
    ctx.accumulate(0)
    ctx.graph_begin()
    _frame(ctx, cam, 1, True)
    ctx.accumulate(1)
    ctx.graph_end()
    ctx.graph_launch(1)


def _larger_frame(ctx, sc, cam):
    _frame(ctx, configs.config_camera(1, 90, 70), 0, True)


def _more_candidates(ctx, sc, cam):
    ctx.ris_path_trace(cam, 1, use_reservoir=True, candidate_count=32, max_depth=1)


def _cleared(ctx, sc, cam):
    ctx.clear_persistent()


def _new_scene(ctx, sc, cam):
    ctx.upload_scene(configs.config1(61, 43, n_lights=8)[0])


@pytest.mark.parametrize("change", [_larger_frame, _more_candidates, _cleared, _new_scene])
def test_a_recording_whose_memory_was_replaced_is_refused(change):
    from hdrestir_b200.context import Context
    sc, cam = configs.config1(61, 43, n_lights=40)
    with Context(device=0) as ctx:
        _recorded(ctx, sc, cam)
        change(ctx, sc, cam)
        with pytest.raises(abi.HdrError, match="record it again"):
            ctx.graph_launch(2)
        _recorded(ctx, sc, cam)  # and can be recorded anew
        ctx.synchronize()


def test_other_buffers_leave_the_recording_valid():
    from hdrestir_b200.context import Context
    sc, cam = configs.config1(61, 43, n_lights=40)
    with Context(device=0) as ctx:
        _recorded(ctx, sc, cam)
        for n in (1000, 3000):  # a buffer of the user's, replaced
            ctx.upload("mine", np.zeros(n, np.float32))
        out = np.empty((61 * 43, 4), np.float32)
        ctx.download_async("Color", out)
        ctx.download_wait()
        ctx.graph_launch(2)
        ctx.synchronize()
