// RISPathTracePass as a wavefront (maxDepth 1, opaque materials): the same
// per-pixel integrator as the one-thread-per-pixel kernel, with its rays cast
// by dedicated traversal kernels instead of inside the shading code.
//
//   generate : per pixel, draws exactly the numbers IntegrationPass::_execute
//              and RisDirectLightIntegrator draw while building the candidate
//              list (integration_pass.cpp:210-226, ris_direct_light_integrator.cpp:
//              230-262), and appends the rays those draws define to two
//              compacted queues: closest-hit (the bounce ray, BSDF candidates)
//              and shadow (one per NEE candidate that passes the early-outs of
//              _evaluateLightSample, :628-658). It saves the stream state at the
//              end of generation: the reservoir-update numbers start there.
//   trace    : one thread per queued ray; closest hit or "occluded before the
//              light" for the ray's slot.
//   shade    : per pixel, repeats the same draws, reads the slot results instead
//              of tracing, and runs the reference's resampling, temporal merge and
//              colour write-back with the saved stream state supplying the
//              update numbers.
// The shade kernel checks that its own stream ends where generate's did
// whenever it replays every candidate.
//
// Rays whose result cannot reach the image are not queued unless the caller
// asks for them: a generated BSDF candidate contributes only when its ray hits
// light geometry or escapes to an environment, so a scene with neither makes
// every such candidate an empty one whatever the ray hits; without emissive
// materials either, the path's bounce ray cannot change the connection
// candidate's weight. Generate then only advances the stream past those
// candidates, and shade counts them as misses and continues from the stream
// state generate saved.
// Compiled twice: here (namespace hdr) with closures that leave the texture code
// out, for scenes without textures, and in wavefront_tex.cu (namespace
// hdr::textured) with it. Untextured frames keep the registers they had.
#ifndef HDR_WAVE_TEXTURED
#define HDR_TEXTURES 0
#endif
#define HDR_SKY 0        // the launchers never take a scene under the physical sky
#define HDR_BLACKBODY 0  // nor one with blackbody lights (extension)
#define HDR_CANDIDATE_INLINE __forceinline__
#define HDR_BOUNCE_INLINE __forceinline__

#include "device/integrator.cuh"
#include "device/pixel.cuh"

namespace hdr {
#ifdef HDR_WAVE_TEXTURED
namespace textured {
#endif

__device__ __forceinline__ int queue_append(int *counter, bool want) {
    const unsigned active = __activemask();
    const unsigned mask = __ballot_sync(active, want);
    if (!want) return -1;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(mask));
    base = __shfl_sync(mask, base, leader);
    return base + __popc(mask & ((1u << lane) - 1u));
}

// Kernel parameters of struct type are __grid_constant__: code that takes their
// address (a reference kept in a struct, a call) reads the parameter space
// instead of a per-thread copy in local memory (a few hundred bytes written per
// thread).
__global__ void __launch_bounds__(256)
    ris_generate_kernel(const __grid_constant__ DeviceScene s, const __grid_constant__ CameraD cam, int frame_arg,
                        const __grid_constant__ PathRun pr, const __grid_constant__ RisRun ris,
                        const __grid_constant__ GBufferView gb, const __grid_constant__ WaveBuffers wb, float4 *color,
                        int trace_level, unsigned *err) {
    uint64_t spill[312];
    MtStream rng;
    PixelStart ps;
    if (!pixel_start(s, cam, live_frame(cam, frame_arg), gb, rng, spill, ps)) return;
    const size_t i = ps.i;
    if (!ps.has_hit) {  // PathIntegrator::Li without a hit: background only, no reservoir access
        V3 rgb = v3s(0.0f);
        if (env_present(s) && pr.render_ibl_background)
            rgb = spectrum_to_rgb(rgb_to_spectrum(env_radiance(s, ps.ray.d), ps.sc.up), ps.sc.cie);
        if (cam.p.has_params && cam.p.enable_exposure) rgb = rgb * cam.p.exposure_mult;
        color[i] = make_float4(rgb.x, rgb.y, rgb.z, 1.0f);
        wb.done[i] = 1;
        if (wb.nee_light)
            for (int j = 0; j < wb.n_shadow; ++j) wb.nee_light[i * (size_t)wb.n_shadow + j] = -1;
        return;
    }
    wb.done[i] = 0;
    Closure c = get_closure(s, ps.hit);
    if (!pr.enable_subsurface) c.subsurface = 0.0f;
    const bool inside = dot(c.normal, ps.ray.d) > 0.0f;
    const Surface sf = make_surface(s, ps.ray.o, ps.ray.d, ps.hit, c, inside);
    const size_t cbase = i * (size_t)wb.n_closest, sbase = i * (size_t)wb.n_shadow;
    // the path's bounce ray (_li, path_integrator.cpp:104-111)
    BounceState st{0, 0};
    const Bounce fb = sample_bounce(c, sf.sn, inside, ps.hit.position, ps.ray.d, pr.max_refl, pr.max_refr, st, ps.sc,
                                    rng);
    {
        const int q = queue_append(&wb.counts[0], fb.ok && trace_level >= kTraceBounceRay);
        if (q >= 0) {
            wb.q_closest[2 * (size_t)q] =
                make_float4(fb.origin.x, fb.origin.y, fb.origin.z, __int_as_float(wb.slot_base_closest + (int)cbase));
            wb.q_closest[2 * (size_t)q + 1] = make_float4(fb.dir.x, fb.dir.y, fb.dir.z, 0.0f);
        }
    }
    // technique split and NEE candidates (:239-246, :553-589)
    const int N = ris.candidate_count;
    const int n_nee = smaxi(1, N / 2), n_bsdf = smaxi(0, N - n_nee);
    for (int j = 0; j < n_nee; ++j) {
        int li;
        LightSampleD ls;
        V3 o, d;
        float lim = 0.0f;
        const bool proposed = propose_candidate(s, ps.hit.position, rng, li, ls);
        if (wb.nee_light) wb.nee_light[sbase + j] = proposed ? li : -1;
        const bool want = proposed && ris_nee_shadow_ray(s, sf, li, ls, ris.skip_vis, o, d, lim);
        const int q = queue_append(&wb.counts[1], want);
        if (q >= 0) {
            wb.q_shadow[2 * (size_t)q] =
                make_float4(o.x, o.y, o.z, __int_as_float(wb.slot_base_shadow + (int)(sbase + j)));
            wb.q_shadow[2 * (size_t)q + 1] = make_float4(d.x, d.y, d.z, lim);
        }
    }
    // generated BSDF candidates (:442-450)
    const int n_fresh = n_bsdf - ((fb.ok && fb.pdf > 0.0f) ? 1 : 0);
    if (trace_level < kTraceAllBsdfRays) {  // their rays are not cast: only the stream has to advance
        const BounceDraws bd = bounce_draws_of(c, sf.sn, inside, ps.ray.d, ps.sc);
        for (int k = 0; k < n_fresh; ++k) {
            BounceState st2{0, 0};
            bounce_draws(bd, 1, 1, st2, rng);
        }
        store_stream(wb.rng_state, i, wb.pixels, rng);
        return;
    }
    for (int k = 0; k < n_fresh; ++k) {
        BounceState st2{0, 0};
        const Bounce b = sample_bounce(c, sf.sn, inside, ps.hit.position, ps.ray.d, 1, 1, st2, ps.sc, rng);
        const int q = queue_append(&wb.counts[0], b.ok);
        if (q >= 0) {
            wb.q_closest[2 * (size_t)q] = make_float4(b.origin.x, b.origin.y, b.origin.z,
                                                      __int_as_float(wb.slot_base_closest + (int)(cbase + 1 + k)));
            wb.q_closest[2 * (size_t)q + 1] = make_float4(b.dir.x, b.dir.y, b.dir.z, 0.0f);
        }
    }
    store_stream(wb.rng_state, i, wb.pixels, rng);
}

template <int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    ris_shade_kernel(const __grid_constant__ DeviceScene s, const __grid_constant__ CameraD cam, int frame_arg,
                     const __grid_constant__ PathRun pr, const __grid_constant__ RisRun ris,
                     const __grid_constant__ GBufferView gb, const __grid_constant__ ReservoirView rv,
                     const __grid_constant__ WaveBuffers wb, float4 *color, int trace_level, unsigned *err) {
    uint64_t spill[312];
    MtStream rng;
    PixelStart ps;
    if (!pixel_start<kThreads>(s, cam, live_frame(cam, frame_arg), gb, rng, spill, ps)) return;
    const size_t i = ps.i;
    if (wb.done[i]) return;
    unsigned e = 0;
    const TracedResults tr{&s, wb.hits + i * (size_t)wb.n_closest, wb.hit_v + i * (size_t)wb.n_closest,
                           wb.occ + i * (size_t)wb.n_shadow, trace_level, wb.q_winner, wb.counts + 4, (int)i};
    const MtStream gen_end = load_stream(wb.rng_state, i, wb.pixels);
    // past 311 draws the state lives in local memory only: replay instead
    const MtStream *gen_end_ptr = gen_end.k < 312 ? &gen_end : nullptr;
    // the wavefront form runs only for maxDepth 1 and opaque scenes
    const Spec L =
        path_li<true, TracedResults, true>(s, tr, ps.ray.o, ps.ray.d, true, ps.hit, ps.sc, rng, pr, ris, rv, i, gen_end_ptr, e);
    V3 rgb = spectrum_to_rgb(L, ps.sc.cie);
    if (cam.p.has_params && cam.p.enable_exposure) rgb = rgb * cam.p.exposure_mult;
    color[i] = make_float4(rgb.x, rgb.y, rgb.z, 1.0f);
    if (e) atomicOr(err, e);
}

namespace {
PathRun path_run(const RisParamsD &p) {
    PathRun pr;
    pr.max_depth = p.max_depth;
    pr.enable_subsurface = p.enable_subsurface != 0;
    pr.max_refl = p.max_refl;
    pr.max_refr = p.max_refr;
    pr.render_ibl_background = p.render_ibl_background != 0;
    pr.roulette = p.roulette;
    return pr;
}
RisRun ris_run(const RisParamsD &p) {
    RisRun ris;
    ris.candidate_count = p.candidate_count;
    ris.use_reservoir = p.use_reservoir != 0;
    ris.skip_vis = p.skip_visibility != 0;
    ris.m_cap = p.m_cap;
    ris.reproj = p.reproj;
    return ris;
}
}  // namespace

int launch_ris_generate(const DeviceScene &s, const CameraD &cam, int frame_index, const RisParamsD &p,
                        GBufferView gb, WaveBuffers wb, float4 *color, int trace_level, unsigned *err,
                        cudaStream_t st) {
    ris_generate_kernel<<<tile_blocks(cam.width, cam.height), 256, 0, st>>>(s, cam, frame_index, path_run(p),
                                                                             ris_run(p), gb, wb, color, trace_level,
                                                                             err);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_ris_shade(const DeviceScene &s, const CameraD &cam, int frame_index, const RisParamsD &p,
                     GBufferView gb, ReservoirView rv, WaveBuffers wb, float4 *color, int trace_level, unsigned *err,
                     cudaStream_t st, const TraceTuning &tune) {
    const PathRun pr = path_run(p);
    const RisRun ris = ris_run(p);
    const int blocks = tile_blocks(cam.width, cam.height);
    switch (tune.shade_shape) {
        case 1:
            ris_shade_kernel<256, 2><<<blocks, 256, 0, st>>>(s, cam, frame_index, pr, ris, gb, rv, wb, color,
                                                             trace_level, err);
            break;
        case 2:
            ris_shade_kernel<128, 3><<<tile_blocks<128>(cam.width, cam.height), 128, 0, st>>>(
                s, cam, frame_index, pr, ris, gb, rv, wb, color, trace_level, err);
            break;
        case 3:
            ris_shade_kernel<128, 4><<<tile_blocks<128>(cam.width, cam.height), 128, 0, st>>>(
                s, cam, frame_index, pr, ris, gb, rv, wb, color, trace_level, err);
            break;
        default:
            ris_shade_kernel<256, 1><<<blocks, 256, 0, st>>>(s, cam, frame_index, pr, ris, gb, rv, wb, color,
                                                             trace_level, err);
    }
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

// After the queued winner shadow rays: a pixel whose winner turned out occluded
// gets what the test on the spot would have given it, throughput 0 (so the
// direct term is 0) and Color = Beer * emission of its surface.
__global__ void __launch_bounds__(256) ris_winner_fixup_kernel(DeviceScene s, CameraD cam, int frame_arg, PathRun pr,
                                                              GBufferView gb, ReservoirView rv, const float4 *q,
                                                              const int *count, const unsigned char *occ,
                                                              float4 *color) {
    const int frame_index = live_frame(cam, frame_arg);
    const int n = *count;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int px = __float_as_int(q[2 * (size_t)k].w);
        if (!occ[px]) continue;
        const int x = px % cam.width, y = px / cam.width;
        MtStream rng;
        rng.init((uint32_t)px ^ (uint32_t)((unsigned long long)frame_index * 12345ULL), nullptr);
        const float fx = (float)x + rng.next_float();
        const float fy = (float)y + rng.next_float();
        const RayF ray = camera_ray(cam, fx, fy, rng);
        const SpectralCtx sc = make_spectral_ctx(rng.next_float());
        Hit h;
        if (!load_gbuffer_hit(s, gb, (size_t)px, h)) continue;
        Closure c = get_closure(s, h);
        if (!pr.enable_subsurface) c.subsurface = 0.0f;
        const bool inside = dot(c.normal, ray.d) > 0.0f;
        Spec tp = spec(1.0f);
        beer_absorption(tp, c, h.depth, inside, sc);
        if (rv.throughput) rv.throughput[px] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const Spec L = tp * (rgb_to_spectrum(c.emission, sc.up) + spec(0.0f));
        V3 rgb = spectrum_to_rgb(L, sc.cie);
        if (cam.p.has_params && cam.p.enable_exposure) rgb = rgb * cam.p.exposure_mult;
        color[px] = make_float4(rgb.x, rgb.y, rgb.z, 1.0f);
    }
}

int launch_winner_visibility(const DeviceScene &s, const CameraD &cam, int frame_index, const RisParamsD &p,
                             GBufferView gb, ReservoirView rv, WaveBuffers wb, float4 *color, unsigned *err,
                             cudaStream_t st, const TraceTuning &tune) {
    if (hdr::launch_shadow_queue(s, wb.q_winner, wb.counts + 4, wb.counts + 5, wb.occ_winner, tune, err, st) < 0)
        return -1;
    ris_winner_fixup_kernel<<<tune.sm_count * 4, 256, 0, st>>>(s, cam, frame_index, path_run(p), gb, rv, wb.q_winner,
                                                               wb.counts + 4, wb.occ_winner, color);
    return cudaPeekAtLastError() == cudaSuccess ? 2 : -1;
}

int launch_ris_wavefront(const DeviceScene &s, const CameraD &cam, int frame_index, const RisParamsD &p,
                         GBufferView gb, ReservoirView rv, WaveBuffers wb, float4 *color, int trace_level,
                         unsigned *err, cudaStream_t st, const TraceTuning &tune, cudaEvent_t *ev_begin,
                         cudaEvent_t *ev_end) {
    // [0] closest rays queued, [1] shadow rays queued, [2] / [3] shadow / closest rays handed out,
    // [4] / [5] winner shadow rays queued / handed out
    if (cudaMemsetAsync(wb.counts, 0, (wb.q_winner ? 6 : 4) * sizeof(int), st) != cudaSuccess) return -1;
    auto mark = [&](cudaEvent_t *ev, int k) { return !ev || cudaEventRecord(ev[k], st) == cudaSuccess; };
    if (!mark(ev_begin, 0)) return -1;
    // callee names in parentheses: no argument-dependent lookup, so the hdr::textured build
    // calls its own launchers, not hdr::'s
    if ((launch_ris_generate)(s, cam, frame_index, p, gb, wb, color, trace_level, err, st) < 0) return -1;
    if (!mark(ev_end, 0)) return -1;
    const int traced =
        hdr::launch_wave_trace(s, wb, tune, err, st, ev_begin ? ev_begin + 1 : nullptr, ev_end ? ev_end + 1 : nullptr);
    if (traced < 0) return -1;
    if (!mark(ev_begin, 3)) return -1;
    if ((launch_ris_shade)(s, cam, frame_index, p, gb, rv, wb, color, trace_level, err, st, tune) < 0) return -1;
    int launches = 2 + traced;
    if (wb.q_winner) {  // the winners' shadow rays, then the pixels they found occluded
        if ((launch_winner_visibility)(s, cam, frame_index, p, gb, rv, wb, color, err, st, tune) < 0) return -1;
        launches += 2;
    }
    if (!mark(ev_end, 3)) return -1;
    return launches;
}

#ifdef HDR_WAVE_TEXTURED
}  // namespace textured
#endif
}  // namespace hdr
