"""The exact in-place firefly clamp (csrc/accumulate.cu, firefly_sequential) against the oracle
around the rows where it hands over from one set of rows to the next (1022 at a time), for
narrow and short frames, and over several frames with the sums it leaves."""
import numpy as np
import pytest

from hdrestir_b200 import configs
from oracle.oracle import accumulate_frame
from tests.accum_frames import same_or_both_nan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (1, 5), (2, 3), (3, 1022), (5, 1023), (4, 1024), (1, 2100), (70, 1030), (300, 7),
                                 (33, 2047), (1100, 3)])
def test_exact_clamp_equals_the_oracle(gpu_ctx, w, h):
    sc, _ = configs.small_variant(0, 8, 8)
    gpu_ctx.upload_scene(sc)
    gpu_ctx.raycast(configs.config_camera(0, w, h), 0)
    gpu_ctx.clear_persistent()
    rng = np.random.default_rng(w * 10_000 + h)
    acc = np.zeros((w * h, 4), np.float32)
    exact = 0
    for f in range(3):
        img = rng.uniform(0.0, 0.4, (h, w, 4)).astype(np.float32)
        bright = rng.random((h, w)) < 0.15
        img[bright, :3] = np.exp(rng.uniform(0, 8, (bright.sum(), 1)))
        # infinite pixels: a sprinkle, and beside every hand-over, each with a bright later neighbour
        for y in {0, h - 1, *range(1019, h, 1022), *range(1020, h, 1022), *range(1021, h, 1022), *range(1022, h, 1022),
                  *rng.integers(0, h, 3)}:
            for x in rng.integers(0, w, 2):
                img[y, x, :3] = (np.inf, 1.0, 1.0) if f != 1 or x % 2 else (np.nan, 2.0, -np.inf)
                img[y, min(x + 1, w - 1), :3] = 40.0
                img[min(y + 1, h - 1), max(x - 1, 0), :3] = 60.0
        frame = np.ascontiguousarray(img.reshape(-1, 4))
        gpu_ctx.upload("Color", frame)
        gpu_ctx.accumulate(f, firefly=True)
        want, shader, acc2 = frame.copy(), frame.copy(), acc.copy()
        accumulate_frame(shader, acc2, w, h, f, firefly=True, mode="shader")
        accumulate_frame(want, acc, w, h, f, firefly=True)
        exact += not same_or_both_nan(want, shader)
        assert same_or_both_nan(gpu_ctx.download("Color"), want), f
        assert same_or_both_nan(gpu_ctx.download("__accum_color"), acc), f
    assert exact > 0 or w <= 4  # of so narrow a frame hardly a pixel can be clamped
