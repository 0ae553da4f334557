// HdRestirRenderBuffer::CopyFromFrameBuffer / _WriteOutput on the device
// (hydra/hd_restir_render_buffer.cpp:46-73,113-148): a float frame buffer
// ("Color", "Depth", "Albedo", "Normal") converted to the render buffer's
// component format, so the renderer's resolve can take the image from HBM
// instead of a host frame buffer. (A source pixel of the destination pixel's
// size is copied as bytes by the caller, as CopyFromFrameBuffer does.) Per
// component c of a pixel:
//   c >= the source's components : 0
//   Float32 : the value
//   Float16 : GfHalf(value) (round to nearest even)
//   UNorm8  : (uint8_t)clamp(value * 255, 0, 255)   (truncating)
//   SNorm8  : (int8_t)clamp(value * 127, -128, 127)  (truncating)
//   Int32   : (int32_t)value                          (truncating)
// std::clamp(v, lo, hi) is (v < lo) ? lo : (hi < v) ? hi : v. Values the
// reference converts with undefined behaviour (NaN, Int32 out of range) are
// not part of the contract.
#include <cuda_fp16.h>

#include "device/frame.cuh"

namespace hdr {
namespace {

__device__ __forceinline__ float ref_clamp(float v, float lo, float hi) { return (v < lo) ? lo : ((hi < v) ? hi : v); }

__device__ __forceinline__ unsigned short to_half(float v) { return __half_as_ushort(__float2half_rn(v)); }
__device__ __forceinline__ unsigned char to_unorm8(float v) {
    return (unsigned char)ref_clamp(v * 255.0f, 0.0f, 255.0f);
}
__device__ __forceinline__ signed char to_snorm8(float v) { return (signed char)ref_clamp(v * 127.0f, -128.0f, 127.0f); }

template <int kFormat>
__global__ void resolve_kernel(const float *__restrict__ src, int src_comps, void *__restrict__ dst, int dst_comps,
                               size_t pixels) {
    const size_t n = pixels * (size_t)dst_comps;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const size_t px = k / (size_t)dst_comps;
        const int c = (int)(k - px * (size_t)dst_comps);
        const bool have = c < src_comps;
        const float v = have ? src[px * (size_t)src_comps + c] : 0.0f;
        if (kFormat == kResolveFloat32) {
            ((float *)dst)[k] = v;
        } else if (kFormat == kResolveFloat16) {
            ((unsigned short *)dst)[k] = have ? to_half(v) : (unsigned short)0;
        } else if (kFormat == kResolveUNorm8) {
            ((unsigned char *)dst)[k] = have ? to_unorm8(v) : (unsigned char)0;
        } else if (kFormat == kResolveSNorm8) {
            ((signed char *)dst)[k] = have ? to_snorm8(v) : (signed char)0;
        } else {
            ((int *)dst)[k] = have ? (int)v : 0;
        }
    }
}

// Four components to four ("Color" into a half or 8-bit buffer) with dst aligned to a pixel: a
// thread takes pixels whole, four loads in flight, where the general kernel takes a component
// with a 64-bit division each (3840 x 2160 to half: 82 us, now 25 for
// its 199 MB, of which the colours are partly still in L2).
template <int kFormat, class Pixel>
__global__ void __launch_bounds__(256) resolve4_kernel(const float4 *__restrict__ src, Pixel *__restrict__ dst,
                                                       size_t pixels) {
    constexpr int kPer = 4;
    const size_t base = (size_t)blockIdx.x * (256 * kPer) + threadIdx.x;
    float4 v[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k)
        if (base + 256 * k < pixels) v[k] = src[base + 256 * k];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        if (base + 256 * k >= pixels) break;
        Pixel p;
        if constexpr (kFormat == kResolveFloat16)
            p = make_ushort4(to_half(v[k].x), to_half(v[k].y), to_half(v[k].z), to_half(v[k].w));
        else if constexpr (kFormat == kResolveUNorm8)
            p = make_uchar4(to_unorm8(v[k].x), to_unorm8(v[k].y), to_unorm8(v[k].z), to_unorm8(v[k].w));
        else
            p = make_char4(to_snorm8(v[k].x), to_snorm8(v[k].y), to_snorm8(v[k].z), to_snorm8(v[k].w));
        dst[base + 256 * k] = p;
    }
}

template <int kFormat, class Pixel>
bool try_resolve4(const float *src, int src_comps, int dst_comps, void *dst, size_t pixels, cudaStream_t st) {
    const size_t blocks = (pixels + 1023) / 1024;
    if (src_comps != 4 || dst_comps != 4 || (uintptr_t)src % sizeof(float4) || (uintptr_t)dst % sizeof(Pixel) ||
        blocks > 0x7fffffffu)
        return false;
    resolve4_kernel<kFormat><<<(unsigned)blocks, 256, 0, st>>>((const float4 *)src, (Pixel *)dst, pixels);
    return true;
}

}  // namespace

int launch_resolve(const float *src, int src_comps, int format, int dst_comps, void *dst, size_t pixels,
                   int sm_count, cudaStream_t st) {
    const size_t n = pixels * (size_t)dst_comps;
    if (n == 0) return 0;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, (size_t)sm_count * 8);
    if ((format == kResolveFloat16 &&
         try_resolve4<kResolveFloat16, ushort4>(src, src_comps, dst_comps, dst, pixels, st)) ||
        (format == kResolveUNorm8 && try_resolve4<kResolveUNorm8, uchar4>(src, src_comps, dst_comps, dst, pixels, st)) ||
        (format == kResolveSNorm8 && try_resolve4<kResolveSNorm8, char4>(src, src_comps, dst_comps, dst, pixels, st)))
        return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
    switch (format) {
        case kResolveFloat32: resolve_kernel<kResolveFloat32><<<blocks, 256, 0, st>>>(src, src_comps, dst, dst_comps, pixels); break;
        case kResolveFloat16: resolve_kernel<kResolveFloat16><<<blocks, 256, 0, st>>>(src, src_comps, dst, dst_comps, pixels); break;
        case kResolveUNorm8: resolve_kernel<kResolveUNorm8><<<blocks, 256, 0, st>>>(src, src_comps, dst, dst_comps, pixels); break;
        case kResolveSNorm8: resolve_kernel<kResolveSNorm8><<<blocks, 256, 0, st>>>(src, src_comps, dst, dst_comps, pixels); break;
        case kResolveInt32: resolve_kernel<kResolveInt32><<<blocks, 256, 0, st>>>(src, src_comps, dst, dst_comps, pixels); break;
        default: return -1;
    }
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

}  // namespace hdr
