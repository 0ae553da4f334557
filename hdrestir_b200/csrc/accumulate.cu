// AccumulationPass::_execute (passes/accumulation_pass.cpp:64-139) and
// GpuAccumulationPass (gpu_functions/shaders/accumulation.slang:39-97):
// optional 3x3 firefly clamp (luminance > 4 x neighbourhood max + 0.5), then
// accum += Color, Color = accum * (1 / (frameIndex + 1)).
//
// The CPU pass clamps in place in row-major order, so a pixel sees its four
// earlier neighbours already clamped; the shader clamps against the unclamped
// input. For finite colours the two agree: the neighbourhood maximum starts at
// 0, so every threshold is >= 0.5 and a clamped pixel q keeps a luminance of
// about its threshold 4 max_n(q) + 0.5 >= 4 lum(p) + 0.5 for every later
// neighbour p. Such a p would need lum(p) > 4 lum(q') + 0.5 for its clamped
// neighbour q' as well, which no positive luminance satisfies, so a clamped
// pixel never changes a neighbour's decision or threshold. Two things break
// this: an infinite luminance (its clamp scale is 0 and inf * 0 is NaN, which the
// neighbour maximum then skips), and channels of both signs that all but cancel in
// the luminance, whose clamped luminance is then rounding error.
//
// Parity mode therefore runs the parallel clamp, checks on the device whether any
// pixel's result changes under the in-place order (only in tiles that hold such a
// pixel, breaks_order), and clamps the frame exactly (firefly_sequential) only when one
// does. The kernel of the mean reads the check's flag itself, so no mode reads anything back
// to the host or waits for the stream.
//
// The clamp, its check and the sum are one pass over the frame (firefly_sum_kernel), the
// mean a second one: neighbours still read the unclamped colour while the first runs.
// 96 bytes per pixel in parity mode (the sums go to a scratch plane, so that the exact clamp
// can still start from the unchanged ones), 80 in shader mode, instead of 128 and 96 in four
// and two passes: 3840 x 2160 takes 80 + 64 us where the clamp, its check and the sum took
// 2 x 77 + 79.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>

#include "device/gf.cuh"

namespace hdr {

__device__ __forceinline__ float lum4(float4 c) { return 0.2126f * c.x + 0.7152f * c.y + 0.0722f * c.z; }

// Could clamping this pixel change what a later neighbour does? Not with a finite luminance
// that keeps 12 of its 24 bits when it is taken again from the scaled channels.
__device__ __forceinline__ bool breaks_order(float4 c, float lum) {
    const float terms = 0.2126f * fabsf(c.x) + 0.7152f * fabsf(c.y) + 0.0722f * fabsf(c.z);
    return !(terms <= FLT_MAX) || (lum > 0.5f && terms > 1024.0f * lum);  // below 0.5 nothing is clamped
}

__device__ __forceinline__ bool same_bits(float4 a, float4 b) {
    return __float_as_int(a.x) == __float_as_int(b.x) && __float_as_int(a.y) == __float_as_int(b.y) &&
           __float_as_int(a.z) == __float_as_int(b.z) && __float_as_int(a.w) == __float_as_int(b.w);
}

// A tile of kTileW x kTileH pixels per block: a thread has kRows rows of one column, a warp
// kRows rows. The luminances of the tile and of the two pixels around it are in shared memory: a
// pixel's neighbours, and theirs for the in-place check, are clamped coordinates of the frame,
// which stay inside that margin.
constexpr int kTileW = 32, kTileH = 32, kRows = 4, kMargin = 2;
constexpr int kTileThreads = kTileW * kTileH / kRows;
constexpr int kLumW = kTileW + 2 * kMargin, kLumH = kTileH + 2 * kMargin;
constexpr int kMarginRows = 2 * kMargin * kLumW, kMarginPixels = kMarginRows + 2 * kMargin * kTileH;

// Tile coordinates (from lum[0]) of pixel m of the margin: the rows above and below, then the sides.
__device__ __forceinline__ void margin_pixel(int m, int &lx, int &ly) {
    if (m < kMarginRows) {
        ly = m / kLumW;
        lx = m - ly * kLumW;
        if (ly >= kMargin) ly += kTileH;
    } else {
        const int k = m - kMarginRows;
        ly = kMargin + k / (2 * kMargin);
        lx = k % (2 * kMargin);
        if (lx >= kMargin) lx += kTileW;
    }
}

struct LumTile {
    const float *lum;
    int x0, y0, width, height;  // frame coordinates of lum[0]; the frame
    __device__ __forceinline__ float at(int x, int y) const {
        return lum[(sclampi(y, 0, height - 1) - y0) * kLumW + (sclampi(x, 0, width - 1) - x0)];
    }
    __device__ __forceinline__ float threshold(int x, int y) const {
        float max_n = 0.0f;
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx)
                if (dx != 0 || dy != 0) max_n = smaxf(max_n, at(x + dx, y + dy));
        return max_n * 4.0f + 0.5f;
    }
};

__device__ __forceinline__ float4 firefly_clamp(float4 c, float lum, float thr) {
    if (lum > thr && lum > 0.0f) {
        const float scale = thr / lum;
        c.x *= scale;
        c.y *= scale;
        c.z *= scale;
    }
    return c;
}

// sums = accum + clamped colour for the frame (sums may be accum itself when nothing needs the
// old sums: kParity false). kParity: *changed is set when some pixel's clamp would come out
// differently with its earlier neighbours already clamped. Bound by memory: all of a thread's
// loads are issued before the first luminance, and a column's maxima of three are shared by the
// rows above and below (a maximum from 0 up that skips NaN has no order). 3840 x 2160: 80 us for
// 398 MB; with the colours read a second time after the luminances, eight loads for each
// threshold and a thread's rows eight apart it took 112.
template <bool kParity>
__global__ void __launch_bounds__(kTileThreads)
    firefly_sum_kernel(const float4 *__restrict__ color, const float4 *accum, float4 *sums, int width, int height,
                       int *changed) {
    __shared__ float lum[kLumH * kLumW];
    const int tiles_x = (width + kTileW - 1) / kTileW;
    const int tx = (int)(blockIdx.x % (unsigned)tiles_x) * kTileW, ty = (int)(blockIdx.x / (unsigned)tiles_x) * kTileH;
    const int t = threadIdx.x, x = tx + t % kTileW, y0 = ty + t / kTileW * kRows;
    float4 c[kRows], a[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        c[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (x < width && y0 + r < height) {
            c[r] = color[(size_t)(y0 + r) * width + x];
            a[r] = accum[(size_t)(y0 + r) * width + x];
        }
    }
    bool odd = false;
    for (int m = t; m < kMarginPixels; m += kTileThreads) {
        int lx, ly;
        margin_pixel(m, lx, ly);
        const int mx = tx - kMargin + lx, my = ty - kMargin + ly;
        float l = 0.0f;
        if (mx >= 0 && my >= 0 && mx < width && my < height) {
            const float4 v = color[(size_t)my * width + mx];
            l = lum4(v);
            if (kParity) odd |= breaks_order(v, l);
        }
        lum[ly * kLumW + lx] = l;
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const float l = lum4(c[r]);
        lum[(y0 - ty + r + kMargin) * kLumW + kMargin + t % kTileW] = l;
        if (kParity) odd |= breaks_order(c[r], l);
    }
    const bool check = kParity ? __syncthreads_or(odd) : (__syncthreads(), false);
    if (x >= width || y0 >= height) return;
    const LumTile tile{lum, tx - kMargin, ty - kMargin, width, height};
    float side[kRows + 2], mid[kRows + 2];  // rows y0 - 1 .. y0 + kRows: the columns beside x; x
#pragma unroll
    for (int r = 0; r < kRows + 2; ++r) {
        const int yr = smini(y0 + r - 1, height);  // rows past the frame's edge repeat it (at())
        side[r] = smaxf(smaxf(0.0f, tile.at(x - 1, yr)), tile.at(x + 1, yr));
        mid[r] = tile.at(x, yr);
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        if (y0 + r >= height) break;
        const float sides = smaxf(smaxf(side[r], side[r + 1]), side[r + 2]);
        const float thr = smaxf(smaxf(sides, mid[r]), mid[r + 2]) * 4.0f + 0.5f;
        const float4 k = firefly_clamp(c[r], lum4(c[r]), thr);
        const size_t p = (size_t)(y0 + r) * width + x;
        if (check) {  // ApplyFireflySuppression's body with the earlier neighbours clamped
            float max_n = 0.0f;
            for (int dy = -1; dy <= 1; ++dy)
                for (int dx = -1; dx <= 1; ++dx) {
                    if (dx == 0 && dy == 0) continue;
                    const int nx = sclampi(x + dx, 0, width - 1), ny = sclampi(y0 + r + dy, 0, height - 1);
                    const size_t q = (size_t)ny * width + nx;
                    float4 v = color[q];
                    if (q < p) v = firefly_clamp(v, lum4(v), tile.threshold(nx, ny));
                    max_n = smaxf(max_n, lum4(v));
                }
            if (!same_bits(firefly_clamp(c[r], lum4(c[r]), max_n * 4.0f + 0.5f), k)) atomicOr(changed, 1);
        }
        sums[p] = make_float4(a[r].x + k.x, a[r].y + k.y, a[r].z + k.z, a[r].w + k.w);
    }
}

__device__ __forceinline__ float4 mean_of(float4 a, float inv_n) {
    return make_float4(a.x * inv_n, a.y * inv_n, a.z * inv_n, a.w * inv_n);
}

// The row-major in-place clamp, exactly, with the sum and the mean in the colour's place, by one
// block of 1024 threads. Pixel (x, y) depends on its earlier neighbours (x-1, y), (x-1, y-1),
// (x, y-1), (x+1, y-1), so a thread walks a row two pixels behind the row above, with a barrier
// after each step, and the rows pass their luminances on in shared memory: the clamped one of a
// pixel when it is clamped, the unclamped one four steps earlier, when the row above comes to need
// it (at time t thread k is at x and reads x-1 .. x+1 of k-1, which clamps x+2, and of k+1, which
// publishes x+2: rings of four have the slots apart). Rows are taken kWalkRows at a time: thread 0
// publishes the last row of the rows before, kept in last_row, the thread past the last row the
// unclamped row below. Bounded: w + 2 kWalkRows + 6 steps for each kWalkRows rows.
//
// Uncoalesced by its nature (a warp's lanes are in 32 rows): what bounds it is the count of
// accesses, three loads and two stores a pixel: 1.43, 9.55 and 35.3 ms for a frame of 640 x 360,
// 1920 x 1080 and 3840 x 2160 (1.64, 10.8 and 47.0 with the eight neighbours' colours from memory
// and the sum and mean in a pass of this block's own).
constexpr int kWalkRows = 1022;
__device__ __noinline__ void firefly_sequential(float4 *color, float *last_row, float4 *accum, int width, int height,
                                                float inv_n) {
    __shared__ float unclamped[4][1024], clamped[4][1024];
    const int k = threadIdx.x;
    for (int y0 = 0; y0 < height; y0 += kWalkRows) {
        const int rows = smini(kWalkRows, height - y0), y = y0 - 1 + k;
        const bool own = k >= 1 && k <= rows, ahead = k >= 1 && k <= rows + 1 && y < height;
        const size_t row = (size_t)smaxi(y, 0) * width;
        const int steps = width + 4 + 2 * (rows + 1);
        for (int t = 0; t < steps; ++t) {
            const int x = t - 4 - 2 * k;
            if (ahead && x + 4 >= 0 && x + 4 < width) unclamped[x & 3][k] = lum4(color[row + x + 4]);
            if (x >= 0 && x < width && k == 0 && y0 > 0) clamped[x & 3][0] = last_row[x];
            if (x >= 0 && x < width && own) {
                const float4 c = color[row + x], b = accum[row + x];
                const float lum = lum4(c);
                const int l = (x - 1) & 3, m = x & 3, r = (x + 1) & 3;
                const bool left = x > 0, right = x + 1 < width, up = y > 0, down = y + 1 < height;
                // (a clamped coordinate at the border names the pixel itself)
                float max_n = left && right && up && down ? 0.0f : smaxf(0.0f, lum);
                if (left) max_n = smaxf(max_n, clamped[l][k]);
                if (right) max_n = smaxf(max_n, unclamped[r][k]);
                if (up) {
                    if (left) max_n = smaxf(max_n, clamped[l][k - 1]);
                    max_n = smaxf(max_n, clamped[m][k - 1]);
                    if (right) max_n = smaxf(max_n, clamped[r][k - 1]);
                }
                if (down) {
                    if (left) max_n = smaxf(max_n, unclamped[l][k + 1]);
                    max_n = smaxf(max_n, unclamped[m][k + 1]);
                    if (right) max_n = smaxf(max_n, unclamped[r][k + 1]);
                }
                const float4 f = firefly_clamp(c, lum, max_n * 4.0f + 0.5f);
                const float4 a = make_float4(b.x + f.x, b.y + f.y, b.z + f.z, b.w + f.w);
                clamped[m][k] = lum4(f);
                if (k == rows) last_row[x] = lum4(f);
                accum[row + x] = a;
                color[row + x] = mean_of(a, inv_n);
            }
            __syncthreads();
        }
    }
}

// The mean, and the sums in their place (kParity; else sums is accum itself). From the last
// pixel down: the sums written last are still in L2. kParity: where the check set *changed the
// first block does the frame's exact clamp, sums and mean from the unchanged accum and colours
// (`out` still holds them), and the others have nothing to do; a kernel of its own for that,
// which almost always only read the flag, took 2.6 us of every frame.
template <bool kParity>
__global__ void __launch_bounds__(1024, 2) mean_kernel(float4 *sums, float4 *accum, float4 *out, int width, int height,
                                                       float inv_n, const int *frame_slot, const int *changed) {
    if (frame_slot) inv_n = 1.0f / (float)(*frame_slot + 1);
    const size_t count = (size_t)width * height;
    if (kParity && *changed) {  // the same for every thread
        if (blockIdx.x == 0) firefly_sequential(out, (float *)sums, accum, width, height, inv_n);
        return;
    }
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < count; k += (size_t)gridDim.x * blockDim.x) {
        const size_t i = count - 1 - k;
        const float4 a = sums[i];
        if (kParity) accum[i] = a;
        out[i] = mean_of(a, inv_n);
    }
}

__global__ void __launch_bounds__(256) accumulate_kernel(const float4 *in, float4 *__restrict__ accum, float4 *out, size_t count, float inv_n,
                                                         const int *frame_slot) {
    // a recorded pass reads its frame index from the slot (the same float division the host does)
    if (frame_slot) inv_n = 1.0f / (float)(*frame_slot + 1);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        const float4 c = in[i];
        float4 a = accum[i];
        a.x += c.x;
        a.y += c.y;
        a.z += c.z;
        a.w += c.w;
        accum[i] = a;
        out[i] = make_float4(a.x * inv_n, a.y * inv_n, a.z * inv_n, a.w * inv_n);
    }
}

// Enqueues the pass on `st`; nothing waits for the device. Returns the number
// of kernels launched, or -1 with the CUDA error in *err.
// scratch holds one float4 plane of width*height (only used with firefly);
// flag_dev one int, zeroed on the stream before each parity-mode check.
int launch_accumulate(float4 *color, float4 *accum, float4 *scratch, int *flag_dev, int width, int height,
                      int frame_index, int firefly, int mode, cudaStream_t st, cudaError_t *err,
                      const int *frame_slot) {
    const size_t count = (size_t)width * height;
    const float inv_n = 1.0f / (float)(frame_index + 1);
    int launches = 0;
    cudaError_t e = cudaSuccess;
    const int blocks = (int)std::max<size_t>(1, std::min<size_t>((count + 255) / 256, (size_t)148 * 8));
    if (firefly) {
        const int mean_blocks = (int)std::max<size_t>(1, std::min<size_t>((count + 1023) / 1024, (size_t)148 * 2));
        const unsigned grid =
            (unsigned)((size_t)((width + kTileW - 1) / kTileW) * (size_t)((height + kTileH - 1) / kTileH));
        if (mode == 0) {
            if ((e = cudaMemsetAsync(flag_dev, 0, sizeof(int), st)) != cudaSuccess) {
                if (err) *err = e;
                return -1;
            }
            firefly_sum_kernel<true><<<grid, kTileThreads, 0, st>>>(color, accum, scratch, width, height, flag_dev);
            mean_kernel<true><<<mean_blocks, 1024, 0, st>>>(scratch, accum, color, width, height, inv_n, frame_slot,
                                                            flag_dev);
        } else {
            firefly_sum_kernel<false><<<grid, kTileThreads, 0, st>>>(color, accum, accum, width, height, nullptr);
            mean_kernel<false><<<mean_blocks, 1024, 0, st>>>(accum, accum, color, width, height, inv_n, frame_slot,
                                                             nullptr);
        }
        launches += 2;
    } else {
        accumulate_kernel<<<blocks, 256, 0, st>>>(color, accum, color, count, inv_n, frame_slot);
        ++launches;
    }
    if ((e = cudaGetLastError()) != cudaSuccess) {
        if (err) *err = e;
        return -1;
    }
    return launches;
}

}  // namespace hdr
