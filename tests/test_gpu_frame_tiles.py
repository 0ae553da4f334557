"""Edges of the tiled frame kernels: the accumulation's 32 x 32 tiles with their margin of two
(csrc/accumulate.cu) around tile borders, with and without luminances that are not finite, and
the whole-pixel render-buffer conversion (csrc/resolve.cu) around its 1024-pixel blocks and
from destinations that are not aligned to a pixel."""
import numpy as np
import pytest

from hdrestir_b200 import abi, configs
from oracle import render_buffer as rb
from oracle.oracle import accumulate_frame
from tests.accum_frames import crafted_frames, same_or_both_nan

pytestmark = pytest.mark.gpu


def _at_size(ctx, w, h):
    sc, _ = configs.small_variant(0, 8, 8)
    ctx.upload_scene(sc)
    ctx.raycast(configs.config_camera(0, w, h), 0)
    ctx.clear_persistent()


@pytest.mark.parametrize("mode", ["parity", "shader"])
@pytest.mark.parametrize("w,h", [(31, 33), (32, 32), (33, 31), (34, 65), (63, 2), (96, 64), (129, 35)])
def test_accumulation_at_tile_borders(gpu_ctx, mode, w, h):
    _at_size(gpu_ctx, w, h)
    frames = crafted_frames(w, h, 3, seed=w + h)
    frames[1] = np.nan_to_num(frames[1], nan=1.0, posinf=3.0, neginf=0.0)  # every luminance finite
    # an infinite pixel and a bright later neighbour across every tile border of the first rows
    img = frames[2].reshape(h, w, 4)
    for x in range(31, w - 1, 32):
        img[0, x - 1:x + 2, :3] = 0.05
        img[0, x, :3] = (np.inf, 1.0, 1.0)
        img[0, x + 1, :3] = 40.0
    acc = np.zeros((w * h, 4), np.float32)
    for f, fr in enumerate(frames):
        gpu_ctx.upload("Color", fr)
        gpu_ctx.accumulate(f, firefly=True, mode=mode)
        want = fr.copy()
        accumulate_frame(want, acc, w, h, f, firefly=True, mode=mode)
        assert same_or_both_nan(gpu_ctx.download("Color"), want), f
        assert same_or_both_nan(gpu_ctx.download("__accum_color"), acc), f


@pytest.mark.parametrize("fmt", [rb.FLOAT16, rb.UNORM8, rb.SNORM8])
@pytest.mark.parametrize("pixels", [1, 255, 1024, 1025, 5000])
@pytest.mark.parametrize("offset", [0, 1, 2, 4])
def test_whole_pixel_conversion(gpu_ctx, fmt, pixels, offset):
    import torch
    _at_size(gpu_ctx, pixels, 1)
    rng = np.random.default_rng(pixels)
    vals = (rng.normal(0.0, 2.0, (pixels, 4)) * 10.0 ** rng.uniform(-6, 4, (pixels, 1))).astype(np.float32)
    gpu_ctx.upload("Color", vals)
    want = rb.copy_from_frame_buffer(vals, fmt, 4)
    size = np.dtype(abi.FMT_DTYPES[fmt]).itemsize
    if offset % size:
        pytest.skip("a component's own alignment")
    dev = torch.zeros(want.nbytes + 64, dtype=torch.uint8, device="cuda:0")
    torch.cuda.synchronize()
    gpu_ctx.resolve("Color", 4, fmt, 4, device_ptr=dev.data_ptr() + 16 + offset)
    gpu_ctx.synchronize()
    got = dev.cpu().numpy()
    assert np.array_equal(got[16 + offset:16 + offset + want.nbytes], want.reshape(-1).view(np.uint8))
    assert not got[:16 + offset].any() and not got[16 + offset + want.nbytes:].any()


@pytest.mark.parametrize("magnitude", [1e3, 1e10, 1e13])
def test_accumulation_of_cancelling_channels(gpu_ctx, magnitude):
    """Finite channels of both signs whose luminance is mostly rounding error: a clamped pixel
    can change its later neighbours too (from 1e9 on some of these rows have one)."""
    n = 1500
    rng = np.random.default_rng(1)
    img = np.full((4 * n, 6, 4), 0.05, np.float32)
    a = (magnitude * rng.uniform(1, 2, n)).astype(np.float32)
    b = -(0.2126 * a.astype(np.float64)) / 0.7152 * (1 - rng.uniform(0, 16, n) * 2.0 ** -24)
    img[1::4, 2, :3] = np.stack([a, b.astype(np.float32), np.zeros(n, np.float32)], 1)
    img[1::4, 3, :3] = np.exp(rng.uniform(0, 12, n))[:, None]
    _at_size(gpu_ctx, 6, 4 * n)
    frame = np.ascontiguousarray(img.reshape(-1, 4))
    gpu_ctx.upload("Color", frame)
    gpu_ctx.accumulate(0, firefly=True)
    want, acc = frame.copy(), np.zeros_like(frame)
    accumulate_frame(want, acc, 6, 4 * n, 0, firefly=True)
    shader, acc2 = frame.copy(), np.zeros_like(frame)
    accumulate_frame(shader, acc2, 6, 4 * n, 0, firefly=True, mode="shader")
    assert np.array_equal(want.view(np.uint32), shader.view(np.uint32)) == (magnitude < 1e9)
    assert same_or_both_nan(gpu_ctx.download("Color"), want)
    assert same_or_both_nan(gpu_ctx.download("__accum_color"), acc)
