// Per-pixel prologue of the wavefront RIS kernels: the pixel's stream, jittered
// camera ray, wavelengths and GBuffer hit (integration_pass.cpp:210-233).
#pragma once

#include "camera.cuh"
#include "integrator.cuh"

namespace hdr {

struct PixelStart {
    size_t i;
    RayF ray;
    SpectralCtx sc;
    Hit hit;
    bool has_hit;
    uint64_t s156;  // the stream's word 156 (MtStream::init_from)
};

__device__ __forceinline__ uint32_t pixel_seed(size_t i, int frame_index) {
    return (uint32_t)i ^ (uint32_t)((unsigned long long)frame_index * 12345ULL);
}
// Pixel (x, y), ps.i set. kSeeded: ps.s156 is known from the pixel's first kernel.
template <bool kSeeded, class Rng>
__device__ __forceinline__ void pixel_start_at(const DeviceScene &s, const CameraD &cam, int frame_index,
                                               const GBufferView &gb, int x, int y, Rng &rng, uint64_t *spill,
                                               PixelStart &ps) {
    const uint32_t seed = pixel_seed(ps.i, frame_index);
    if constexpr (kSeeded) {
        rng.init_from(seed, ps.s156, spill);
    } else {
        rng.init(seed, spill);
        ps.s156 = rng.c;
    }
    const float px = (float)x + rng.next_float();
    const float py = (float)y + rng.next_float();
    ps.ray = camera_ray(cam, px, py, rng);
    ps.sc = make_spectral_ctx(rng.next_float());
    ps.has_hit = load_gbuffer_hit(s, gb, ps.i, ps.hit);
}
template <int kThreads = 256, class Rng>
__device__ __forceinline__ bool pixel_start(const DeviceScene &s, const CameraD &cam, int frame_index,
                                            const GBufferView &gb, Rng &rng, uint64_t *spill, PixelStart &ps) {
    int x, y;
    if (!tile_pixel<kThreads>(cam.width, cam.height, x, y)) return false;
    ps.i = (size_t)y * (size_t)cam.width + (size_t)x;
    pixel_start_at<false>(s, cam, frame_index, gb, x, y, rng, spill, ps);
    return true;
}

}  // namespace hdr
