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
//              _evaluateLightSample, :628-658). A light candidate's resampling
//              weight, should its ray be unoccluded, is computed and stored here,
//              while its sample is at hand. It saves the stream state at the
//              end of generation: the reservoir-update numbers start there.
//   trace    : closest hit or "occluded before the light" for the ray's slot (trace.cu).
//   resample : per pixel, the reference's choice among the stored weights, the
//              temporal merge and the colour write-back, the saved stream state
//              supplying the update numbers; the chosen light candidate alone is
//              evaluated again. Where BSDF rays matter, the general form (shade)
//              also replays the draws of the BSDF candidates.
// The general form checks that its own stream ends where generate's did
// whenever it replays every candidate.
//
// Rays whose result cannot reach the image are not queued unless the caller
// asks for them: a generated BSDF candidate contributes only when its ray hits
// light geometry or escapes to an environment, so a scene with neither makes
// every such candidate an empty one whatever the ray hits; without emissive
// materials either, the path's bounce ray cannot change the connection
// candidate's weight. Generate then only advances the stream past those
// candidates, and resampling counts them as misses and continues from the stream
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

// WaveBuffers::done of a pixel
constexpr int kPixelMiss = 1;     // no GBuffer hit: its colour is written
constexpr int kPixelConn = 2;     // the path's bounce is a candidate (its pdf is above 0)
constexpr int kPixelConnNan = 4;  // and its pdf squared overflows: its weight is a NaN (power_heuristic3
                                  // with a count of 0 in front of it is 0)

// Kernel parameters of struct type are __grid_constant__: code that takes their
// address (a reference kept in a struct, a call) reads the parameter space
// instead of a per-thread copy in local memory (a few hundred bytes written per
// thread).
//
// Bound by instruction issue (16 light candidates per 1080p terrain pixel, weights included: about
// 900 instructions per candidate, a quarter of them the stream). A stream of at most 155 draws
// takes no branch per draw and needs no spill block: 1.64 -> 1.42 ms, 512 x 512 boxes with 8
// candidates 0.119 -> 0.105, textured 960 x 540 0.417 -> 0.368.
//
// Shape: four blocks of 128 (128 registers, nothing spilled). Five (96 registers): 1.45, 0.115,
// 0.416 ms; six (80): 1.41, 0.117, 0.415.
constexpr int kGenerateThreads = 128;
template <class Rng, bool kWeights>  // MtShort where draws_to_generation_end is at most 155
__global__ void __launch_bounds__(kGenerateThreads, 4)
    ris_generate_kernel(const __grid_constant__ DeviceScene s, const __grid_constant__ CameraD cam, int frame_arg,
                        const __grid_constant__ PathRun pr, const __grid_constant__ RisRun ris,
                        const __grid_constant__ GBufferView gb, const __grid_constant__ WaveBuffers wb, float4 *color,
                        int trace_level, unsigned *err) {
    uint64_t spill[312];
    Rng rng;
    PixelStart ps;
    if (!pixel_start<kGenerateThreads>(s, cam, live_frame(cam, frame_arg), gb, rng, spill, ps)) return;
    const size_t i = ps.i;
    if (!ps.has_hit) {  // PathIntegrator::Li without a hit: background only, no reservoir access
        V3 rgb = v3s(0.0f);
        if (env_present(s) && pr.render_ibl_background)
            rgb = spectrum_to_rgb(rgb_to_spectrum(env_radiance(s, ps.ray.d), ps.sc.up), ps.sc.cie);
        if (cam.p.has_params && cam.p.enable_exposure) rgb = rgb * cam.p.exposure_mult;
        color[i] = make_float4(rgb.x, rgb.y, rgb.z, 1.0f);
        wb.done[i] = kPixelMiss;
        if (wb.nee_light)
            for (int j = 0; j < wb.n_shadow; ++j) wb.nee_light[i * (size_t)wb.n_shadow + j] = -1;
        return;
    }
    Closure c = get_closure(s, ps.hit);
    if (!pr.enable_subsurface) c.subsurface = 0.0f;
    const bool inside = dot(c.normal, ps.ray.d) > 0.0f;
    const Surface sf = make_surface(s, ps.ray.o, ps.ray.d, ps.hit, c, inside);
    const size_t cbase = i * (size_t)wb.n_closest;
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
    const bool conn = fb.ok && fb.pdf > 0.0f;
    wb.done[i] = (unsigned char)((conn ? kPixelConn : 0) | (conn && n_bsdf > 0 && isinf(fb.pdf * fb.pdf) ? kPixelConnNan : 0));
    const uint32_t k0 = rng.k;
    const RisStrategy strat{n_nee, 0, n_bsdf, ris.skip_vis};
    for (int j = 0; j < n_nee; ++j) {
        int li;
        LightSampleD ls;
        RisNeeRay ray;
        ray.cast = ray.stays = false;
        ray.weight = 0.0;
        const bool proposed = propose_candidate(s, ps.hit.position, rng, li, ls);
        if (wb.nee_light) wb.nee_light[i * (size_t)wb.n_shadow + j] = proposed ? li : -1;
        if (proposed) ray = ris_nee_ray(s, sf, li, ls, strat, ps.sc, kWeights);
        const size_t slot = (size_t)j * wb.pixels + i;
        if (kWeights) {
            if (ris.use_reservoir)
                ((float *)wb.nee_weight)[slot] = nee_weight_bits<float>(ray.weight, ray.stays);
            else
                ((double *)wb.nee_weight)[slot] = nee_weight_bits<double>(ray.weight, ray.stays);
        }
        const int q = queue_append(&wb.counts[1], ray.cast);
        if (q >= 0) {
            wb.q_shadow[2 * (size_t)q] =
                make_float4(ray.o.x, ray.o.y, ray.o.z, __int_as_float(wb.slot_base_shadow + (int)slot));
            wb.q_shadow[2 * (size_t)q + 1] = make_float4(ray.d.x, ray.d.y, ray.d.z, ray.limit);
        }
    }
    // generated BSDF candidates (:442-450)
    const int n_fresh = n_bsdf - (conn ? 1 : 0);
    if (trace_level < kTraceAllBsdfRays) {  // their rays are not cast: only the stream has to advance
        const BounceDraws bd = bounce_draws_of(c, sf.sn, inside, ps.ray.d, ps.sc);
        for (int k = 0; k < n_fresh; ++k) {
            BounceState st2{0, 0};
            bounce_draws(bd, 1, 1, st2, rng);
        }
        store_stream_from(wb.rng_state, i, wb.pixels, whole_stream(rng), ps.s156, k0);
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
    store_stream_from(wb.rng_state, i, wb.pixels, whole_stream(rng), ps.s156, k0);
}

template <bool kWeights>
__device__ __forceinline__ TracedResults<kWeights> traced_results(const DeviceScene &s, const RisRun &ris,
                                                                  const WaveBuffers &wb, int trace_level, size_t i) {
    return TracedResults<kWeights>{
        &s, wb.hits + i * (size_t)wb.n_closest, wb.hit_v + i * (size_t)wb.n_closest, wb.occ + i,
        (const char *)wb.nee_weight + i * (ris.use_reservoir ? sizeof(float) : sizeof(double)),
        wb.pixels, ris.skip_vis, trace_level, wb.q_winner, wb.counts + 4, (int)i};
}

// The general form of a pixel's resampling: every candidate that is not a light's is replayed,
// without stored weights the lights' too.
template <bool kWeights>
__device__ __forceinline__ void shade_general(const DeviceScene &s, const CameraD &cam, int frame_index,
                                              const PathRun &pr, const RisRun &ris, const GBufferView &gb,
                                              const ReservoirView &rv, const WaveBuffers &wb, float4 *color,
                                              int trace_level, int x, int y, unsigned &e) {
    const size_t i = (size_t)y * (size_t)cam.width + (size_t)x;
    uint64_t spill[312];
    MtStream rng;
    PixelStart ps;
    uint32_t k0;
    const MtStream gen_end =
        load_stream_from(wb.rng_state, i, wb.pixels, pixel_seed(i, frame_index), ps.s156, k0);
    ps.i = i;
    pixel_start_at<true>(s, cam, frame_index, gb, x, y, rng, spill, ps);
    const auto tr = traced_results<kWeights>(s, ris, wb, trace_level, i);
    // past 311 draws the state lives in local memory only: replay instead
    const MtStream *gen_end_ptr = gen_end.k < 312 ? &gen_end : nullptr;
    // the wavefront form runs only for maxDepth 1 and opaque scenes
    const Spec L =
        path_li<true, TracedResults<kWeights>, true>(s, tr, ps.ray.o, ps.ray.d, true, ps.hit, ps.sc, rng, pr, ris, rv, i, gen_end_ptr, e);
    V3 rgb = spectrum_to_rgb(L, ps.sc.cie);
    if (cam.p.has_params && cam.p.enable_exposure) rgb = rgb * cam.p.exposure_mult;
    color[i] = make_float4(rgb.x, rgb.y, rgb.z, 1.0f);
}

template <bool kWeights>
__global__ void __launch_bounds__(256, 2)
    ris_shade_kernel(const __grid_constant__ DeviceScene s, const __grid_constant__ CameraD cam, int frame_arg,
                     const __grid_constant__ PathRun pr, const __grid_constant__ RisRun ris,
                     const __grid_constant__ GBufferView gb, const __grid_constant__ ReservoirView rv,
                     const __grid_constant__ WaveBuffers wb, float4 *color, int trace_level, unsigned *err) {
    int x, y;
    if (!tile_pixel(cam.width, cam.height, x, y)) return;
    if (wb.done[(size_t)y * (size_t)cam.width + (size_t)x] & kPixelMiss) return;
    unsigned e = 0;
    shade_general<kWeights>(s, cam, live_frame(cam, frame_arg), pr, ris, gb, rv, wb, color, trace_level, x, y, e);
    if (e) atomicOr(err, e);
}

// A light candidate (or a history's sample) as the reservoir holds it: target function and
// throughput of a sample that is not dropped and not occluded (ris_nee_candidate,
// _reEvaluateForTemporalReuse :675-691).
__device__ __forceinline__ Spec light_throughput(const DeviceScene &s, const Surface &sf, int li,
                                                 const LightSampleD &ls, const SpectralCtx &sc) {
    const V3 bval = ggx_eval_f(sf.g, sf.sn, -sf.ray_d, ls.dir);
    return light_emission(s, li, ls.color, sc) * rgb_to_spectrum(bval * dot(sf.sn, ls.dir), sc.up);
}

// Resampling of a pixel none of whose BSDF rays matter (trace level kTraceNoBsdfRays: no light
// geometry, no environment, no emission). Its BSDF candidates, the path's bounce among them,
// weigh 0 and only count, so no bounce is sampled: the light candidates' weights choose, and
// only the winner is evaluated, from its own draws (found by index: no draw before it is
// replayed). Evaluating the candidates here, as the general form's kernel did, took 2.15 ms of a
// 1080p terrain frame, most of it local memory and draws repeated; weights from the generate
// kernel, where the candidate is in registers anyway, and this kernel take 0.42 ms next to 0.59
// ms more in generate. More resident warps pay against spills: 0.60 ms at 128 registers, 0.53
// at 96, 0.43 at 64 in blocks of 256, 0.42 in blocks of 128.
// ris_direct_li with the loops that cannot matter left out, for frames whose streams
// stay below draw 312 during generation (launch_ris_shade).
template <int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    ris_resample_kernel(const __grid_constant__ DeviceScene s, const __grid_constant__ CameraD cam, int frame_arg,
                        const __grid_constant__ PathRun pr, const __grid_constant__ RisRun ris,
                        const __grid_constant__ GBufferView gb, const __grid_constant__ ReservoirView rv,
                        const __grid_constant__ WaveBuffers wb, float4 *color, unsigned *err) {
    int x, y;
    if (!tile_pixel<kThreads>(cam.width, cam.height, x, y)) return;
    const size_t i = (size_t)y * (size_t)cam.width + (size_t)x;
    const int done = wb.done[i];
    if (done & kPixelMiss) return;
    const int frame_index = live_frame(cam, frame_arg);
    unsigned e = 0;
    uint64_t spill[312];
    PixelStart ps;
    uint32_t k0;
    MtStream upd = load_stream_from(wb.rng_state, i, wb.pixels, pixel_seed(i, frame_index), ps.s156, k0);
    upd.spill = spill;
    const auto tr = traced_results<true>(s, ris, wb, kTraceNoBsdfRays, i);
    const int N = ris.candidate_count;
    const int n_nee = smaxi(1, N / 2), n_bsdf = smaxi(0, N - n_nee), conn = (done & kPixelConn) ? 1 : 0;
    const int n_total = n_nee + conn + smaxi(0, n_bsdf - conn);

    // the light candidates' choice
    int winner = -1;
    float wsum = 0.0f;
    double wsum_d = 0.0;
    if (ris.use_reservoir) {
        for (int j = 0; j < n_nee; ++j) {
            const float w = tr.nee_weight<float>(j);
            if (w <= 0.0f) continue;
            wsum += w;
            if (upd.next_float() <= w / wsum) winner = j;
        }
        if (done & kPixelConnNan) {  // not <= 0: it enters the sum and draws, and is never chosen
            wsum += __int_as_float(0x7fffffff);
            (void)upd.next_raw();
        }
    } else if (n_total > kMaxPlainRisCandidates) {
        e |= kErrRisCapacity;
    } else {
        for (int j = 0; j < n_nee; ++j) {
            const double w = tr.nee_weight<double>(j);
            if (w > 0.0) wsum_d += w;
        }
        if (wsum_d > 0.0) {
            double remaining = (double)upd.next_float() * wsum_d;
            for (int j = 0; j < n_nee && winner < 0; ++j) {
                const double w = tr.nee_weight<double>(j);
                if (w <= 0.0) continue;
                remaining -= w;
                if (remaining <= 0.0) winner = j;
            }
        }
    }

    MtStream rng;
    ps.i = i;
    pixel_start_at<true>(s, cam, frame_index, gb, x, y, rng, spill, ps);
    Closure c = get_closure(s, ps.hit);
    if (!pr.enable_subsurface) c.subsurface = 0.0f;
    const bool inside = dot(c.normal, ps.ray.d) > 0.0f;
    Spec beer = spec(1.0f);
    beer_absorption(beer, c, ps.hit.depth, inside, ps.sc);
    const Surface sf = make_surface(s, ps.ray.o, ps.ray.d, ps.hit, c, inside);
    const Spec emitted = rgb_to_spectrum(sf.c.emission, ps.sc.up);

    Reservoir r;
    r.chosen = cand_none();
    r.wsum = wsum;
    r.m = n_total;
    r.w = 0.0f;
    if (ris.use_reservoir) {  // temporal reuse (:284-305)
        Reservoir prev;
        bool have_prev = true;
        if (ris.reproj.mode == 0)
            reservoir_load(rv, i, prev);
        else
            have_prev = reprojected_history(ris.reproj, sf.hit.position, prev);
        if (have_prev && prev.chosen.valid && prev.chosen.has_lc && prev.chosen.target > 0.0f) {
            const float phat_gen = prev.chosen.target;
            const Spec reeval = ris_reevaluate(s, sf, prev.chosen.light, prev.chosen.ls, ps.sc);
            const float phat_curr = spectrum_luminance(reeval, ps.sc.cie);
            if (ris.m_cap > 0) {  // extension: bound the history (M-cap)
                const int cap = ris.m_cap * n_total;
                if (prev.m > cap) {
                    prev.wsum *= (float)cap / (float)prev.m;
                    prev.m = cap;
                }
            }
            const float mw = prev.wsum * (phat_curr / phat_gen);
            r.m += prev.m;  // Merge (:157-166)
            if (mw > 0.0f) {
                r.wsum += mw;
                if (upd.next_float() <= mw / r.wsum) {
                    r.chosen = prev.chosen;
                    r.chosen.target = phat_curr;
                    r.chosen.tp = reeval;
                    winner = -1;
                }
            }
        }
    }
    if (winner >= 0) {
        rng.skip(k0 - rng.k);
        skip_candidates(s, winner, rng);
        Cand &k = r.chosen;
        k.valid = k.has_lc = propose_candidate(s, ps.hit.position, rng, k.light, k.ls);
        k.tp = light_throughput(s, sf, k.light, k.ls, ps.sc);
        k.target = spectrum_luminance(k.tp, ps.sc.cie);
        k.vis_tested = !ris.skip_vis;
    }
    float W = 0.0f;
    if (ris.use_reservoir)
        reservoir_finalize(r, n_total);
    else if (r.chosen.valid)
        W = (float)(wsum_d / (double)r.chosen.target);
    if (r.chosen.valid && !r.chosen.vis_tested && r.chosen.has_lc) {  // winner visibility (:309-321)
        const RisContrib nee =
            ris_evaluate_light_sample(s, tr, -1, sf, r.chosen.light, r.chosen.ls, false, ps.sc, e);
        r.chosen.tp = nee.emission * nee.tmul;
        r.chosen.vis_tested = true;
    }
    Spec direct = spec(0.0f);
    if (ris.use_reservoir) {
        reservoir_store(rv, i, r);
        if (r.chosen.valid && !(r.w <= 0.0f)) direct = r.chosen.tp * r.w;
    } else if (r.chosen.valid) {
        direct = r.chosen.tp * W;
    }
    V3 rgb = spectrum_to_rgb(beer * (emitted + direct), ps.sc.cie);
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
    ris.trace_all = p.trace_all != 0;
    ris.reproj = p.reproj;
    return ris;
}
}  // namespace

int launch_ris_generate(const DeviceScene &s, const CameraD &cam, int frame_index, const RisParamsD &p,
                        GBufferView gb, WaveBuffers wb, float4 *color, int trace_level, unsigned *err,
                        cudaStream_t st) {
    const bool few = draws_to_generation_end(p) <= 155;
    auto k = wb.nee_weight ? (few ? ris_generate_kernel<MtShort, true> : ris_generate_kernel<MtStream, true>)
                           : (few ? ris_generate_kernel<MtShort, false> : ris_generate_kernel<MtStream, false>);
    k<<<tile_blocks<kGenerateThreads>(cam.width, cam.height), kGenerateThreads, 0, st>>>(
        s, cam, frame_index, path_run(p), ris_run(p), gb, wb, color, trace_level, err);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_ris_shade(const DeviceScene &s, const CameraD &cam, int frame_index, const RisParamsD &p,
                     GBufferView gb, ReservoirView rv, WaveBuffers wb, float4 *color, int trace_level, unsigned *err,
                     cudaStream_t st, const TraceTuning &tune) {
    const PathRun pr = path_run(p);
    const RisRun ris = ris_run(p);
    if (lean_resampling(p, wb, trace_level)) {
        const bool wide = tune.shade_shape < 2;  // 256 threads per block, else 128
        const int blocks = wide ? tile_blocks<256>(cam.width, cam.height) : tile_blocks<128>(cam.width, cam.height);
        auto k = tune.shade_shape == 0   ? ris_resample_kernel<256, 2>
                 : tune.shade_shape == 1 ? ris_resample_kernel<256, 4>
                 : tune.shade_shape == 2 ? ris_resample_kernel<128, 5>
                                         : ris_resample_kernel<128, 8>;
        k<<<blocks, wide ? 256 : 128, 0, st>>>(s, cam, frame_index, pr, ris, gb, rv, wb, color, err);
    } else {
        auto k = wb.nee_weight ? ris_shade_kernel<true> : ris_shade_kernel<false>;
        k<<<tile_blocks(cam.width, cam.height), 256, 0, st>>>(s, cam, frame_index, pr, ris, gb, rv, wb, color,
                                                              trace_level, err);
    }
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

// After the queued winner shadow rays: a pixel whose winner turned out occluded
// gets what the test on the spot would have given it, throughput 0 (so the
// direct term is 0) and Color = Beer * emission of its surface.
__global__ void __launch_bounds__(256) ris_winner_fixup_kernel(DeviceScene s, CameraD cam, int frame_arg, PathRun pr,
                                                              GBufferView gb, ReservoirView rv,
                                                              const uint4 *rng_state, const float4 *q,
                                                              const int *count, const unsigned char *occ,
                                                              float4 *color) {
    const int frame_index = live_frame(cam, frame_arg);
    const int n = *count;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int px = __float_as_int(q[2 * (size_t)k].w);
        if (!occ[px]) continue;
        const int x = px % cam.width, y = px / cam.width;
        MtShort rng;
        rng.init_from(pixel_seed((size_t)px, frame_index), stored_s156(rng_state, (size_t)px));
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
    if (hdr::launch_shadow_queue(s, wb.q_winner, wb.pixels, wb.counts + 4, wb.counts + 5, wb.occ_winner, tune, err, st) < 0)
        return -1;
    ris_winner_fixup_kernel<<<tune.sm_count * 4, 256, 0, st>>>(s, cam, frame_index, path_run(p), gb, rv, wb.rng_state,
                                                               wb.q_winner, wb.counts + 4, wb.occ_winner, color);
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
