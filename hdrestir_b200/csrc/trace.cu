// Ray-queue kernels of the wavefront passes: the closest-hit and shadow queries over
// the queues the generate / sample kernels fill, one answer per ray in its slot.
#include <algorithm>
#include <type_traits>

#include "device/frame.cuh"

namespace hdr {

// Trace kernels. Rays of a warp take very different numbers of steps (shadow
// rays towards random lights: 43 % of lane-steps did work when each lane
// traced a fixed ray), so the default form is persistent: a lane whose ray is
// finished takes the next queued ray (one atomic per warp for all its idle
// lanes) and every lane steps its own walk, one stack entry per iteration,
// until the queue is drained. fetch_at counts the rays handed out.
constexpr unsigned kFullMask = 0xffffffffu;

__device__ __forceinline__ int fetch_ray(int *fetch_at, int n, bool need, bool &drained) {
    const unsigned want = __ballot_sync(kFullMask, need);
    if (!want || drained) return -1;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(want) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(fetch_at, __popc(want));
    base = __shfl_sync(kFullMask, base, leader);
    if (base + __popc(want) >= n) drained = true;  // warp-uniform
    const int k = base + __popc(want & ((1u << lane) - 1));
    return (need && k < n) ? k : -1;
}

// Stack entries below kSharedDepth live in the block's shared memory (one
// column per thread), deeper ones in local memory.
constexpr int kTraceThreads = 128;
constexpr int kSharedDepth = 24;
static_assert(kTraceStack == kWideStack, "one spill size for both walks");

template <bool kWide, bool kAnyHit>
struct TraceWalk {
    using Entry = typename std::conditional<kWide, int2, int>::type;
    using Stack = SplitStack<Entry, kSharedDepth, kTraceThreads>;
    using type = typename std::conditional<kWide, WideWalk<kAnyHit, Stack>, BinaryWalk<kAnyHit, Stack>>::type;
};

// Phased schedule (PhasedWalk): node steps run while at least `quorum` lanes
// of the warp are stepping nodes; then the parked leaves, instance entries and
// finished rays of all lanes are served, and finished lanes take the next
// queued rays.
// Shared-memory stack entries per thread of the phased wide walk (8-byte
// entries: the same 12 KB per block as the binary walk's 24 four-byte ones).
constexpr int kSharedDepthWide = 12;

// kShallow (binary walk only): the scene's trees fit a kShallowStack-entry
// stack, which then lives wholly in shared memory (20 KB per block).
template <bool kWide, bool kAnyHit, bool kShallow>
struct PhasedTraceWalk {
    static_assert(!(kWide && kShallow), "the shallow stack serves the binary walk");
    using Entry = typename std::conditional<kWide, int2, int>::type;
    static constexpr int kShared = kShallow ? kShallowStack : (kWide ? kSharedDepthWide : kSharedDepth);
    using Stack = typename std::conditional<kShallow, ColumnStack<Entry, kShared, kTraceThreads>,
                                            SplitStack<Entry, kShared, kTraceThreads>>::type;
    using type = typename std::conditional<kWide, PhasedWideWalk<kAnyHit, Stack>, PhasedWalk<kAnyHit, Stack>>::type;
};

template <class Stk, class Entry>
__device__ __forceinline__ void bind_deep(Stk &, Entry *) {}
template <class Entry, int kDepth, int kThreads>
__device__ __forceinline__ void bind_deep(SplitStack<Entry, kDepth, kThreads> &st, Entry *deep) {
    st.deep = deep;
}

template <bool kWide, bool kShallow, bool kAnyHit, class Put>
__device__ __forceinline__ void phased_trace(const DeviceScene &s, const float4 *__restrict__ q,
                                             int n, int *fetch_at, int quorum, Put put, unsigned &e) {
    using PW = PhasedTraceWalk<kWide, kAnyHit, kShallow>;
    __shared__ typename PW::Entry col[PW::kShared * kTraceThreads];
    typename PW::Entry deep[kShallow ? 1 : kTraceStack - PW::kShared];
    typename PW::type w;
    w.stack.col = col + threadIdx.x;
    bind_deep(w.stack, deep);
    w.mode = kModeDone;
    NoStats ns;
    int slot = -1;
    bool drained = false;
    for (;;) {
        const bool done = w.mode == kModeDone;
        if (done && slot >= 0) {
            put(slot, w);
            slot = -1;
        }
        const int k = fetch_ray(fetch_at, n, done, drained);
        if (done) {
            if (k >= 0) {
                const float4 a = q[2 * (size_t)k], b = q[2 * (size_t)k + 1];
                w.start(s, V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, kAnyHit ? b.w : 0.0f);
                slot = __float_as_int(a.w);
            } else {
                w.mode = kModeIdle;
            }
        }
        if (!__any_sync(kFullMask, w.mode != kModeIdle)) break;
        do {
            if (w.mode == kModeNode) {
                if (w.regular(s))
                    w.template node_step<true>(s, e, ns);
                else
                    w.template node_step<false>(s, e, ns);
            }
        } while (__popc(__ballot_sync(kFullMask, w.mode == kModeNode)) >= quorum);
        if (w.mode == kModeLeaf) w.leaf(s, ns);
        if (w.mode == kModeInst) w.inst(s);
    }
}

// Resident blocks per SM the phased kernels are compiled for (64 registers for
// the binary walk, 80 for the wide one).
template <bool kWide>
constexpr int phased_min_blocks() {
    return kWide ? 6 : 8;
}

// Closest hits on the reference's trees, fetch counting the entries handed out.
template <bool kWide, bool kShallow>
__global__ void __launch_bounds__(kTraceThreads, phased_min_blocks<kWide>()) trace_closest_phased_kernel(DeviceScene s, const float4 *__restrict__ q,
                                                                             const int *count, int *fetch, float4 *hits, float *hit_v,
                                                                             int quorum, unsigned *err) {
    unsigned e = 0;
    phased_trace<kWide, kShallow, false>(
        s, q, *count, fetch, quorum,
        [&](int slot, const auto &w) {
            hits[slot] = make_float4(w.hit.t, __int_as_float(w.hit.inst), __int_as_float(w.hit.tri), w.hit.u);
            hit_v[slot] = w.hit.v;
        },
        e);
    if (e) atomicOr(err, e);
}

template <bool kWide, bool kShallow>
__global__ void __launch_bounds__(kTraceThreads, phased_min_blocks<kWide>()) trace_shadow_phased_kernel(DeviceScene s, const float4 *__restrict__ q,
                                                                            const int *count, int *fetch,
                                                                            unsigned char *occ, int quorum,
                                                                            unsigned *err) {
    unsigned e = 0;
    phased_trace<kWide, kShallow, true>(
        s, q, *count, fetch, quorum,
        [&](int slot, const auto &w) { occ[slot] = w.shadow_answer() ? 1 : 0; }, e);
    if (e) atomicOr(err, e);
}

// Walks of the shadow BVH (DeviceScene::sh4) over a ray queue: persistent lanes, each on
// its own ray's 4-wide walk. Node steps run while at least `quorum` lanes of
// the warp are on node entries; then the parked leaves (triangle tests) and
// ray switches of all lanes are served, and finished lanes take new rays.
//
// A warp takes the rays it hands out in chunks of consecutive entries: one atomic per
// chunk instead of one whenever some of its lanes finish (2.4 M atomics on one address
// for the 14.5 M shadow rays of a 1080p frame).
constexpr int kSh4Shared = 24;

struct RayChunk {
    unsigned at, end;  // entries in hand
    unsigned size;     // entries taken at a time
    bool drained;  // the queue has no more
    __device__ __forceinline__ void init(unsigned n) {
        at = end = 0;
        drained = false;
        // a few chunks per warp, so that the warps finish together
        const unsigned warps = (gridDim.x * blockDim.x) >> 5;
        size = min(128u, max(32u, (n / (4 * warps)) & ~31u));
    }
    // an entry for every lane with `need` (warp-uniform state); -1: none in this chunk
    __device__ __forceinline__ int take(int *fetch_at, unsigned n, bool need) {
        const unsigned want = __ballot_sync(kFullMask, need);
        if (!want) return -1;
        const int lane = threadIdx.x & 31;
        if (at >= end && !drained) {
            unsigned base = 0;
            if (lane == 0) base = (unsigned)atomicAdd(fetch_at, (int)size);
            at = __shfl_sync(kFullMask, base, 0);
            end = min(n, at + size);
            drained = at + size >= n;
        }
        const unsigned k = at + __popc(want & ((1u << lane) - 1u));
        const bool got = need && k < end;
        at = min(max(at, end), at + __popc(want));
        return got ? (int)k : -1;
    }
    __device__ __forceinline__ bool empty() const { return drained && at >= end; }
};

// W: the walk; start(w, entry a, entry b) gives it a ray; put(slot, w) stores its answer.
template <class W, class Start, class Put>
__device__ __forceinline__ void walk4_queue(const DeviceScene &s, W &w, const float4 *__restrict__ q, int n, int *fetch,
                                            int quorum, int *col, Start start, Put put, unsigned &e) {
    int deep[kSh4Stack - kSh4Shared];
    w.stack.bind(col + threadIdx.x, deep);
    w.cur = kSh4Done;
    NoStats ns;
    RayChunk chunk;
    chunk.init((unsigned)n);
    int slot = -1;
    for (;;) {
        const bool over = sh4_is_over(w.cur);
        if (over && slot >= 0) {
            put(slot, w);
            slot = -1;
        }
        const int k = chunk.take(fetch, (unsigned)n, over);
        if (k >= 0) {
            const float4 *at = q + 2 * (size_t)k;
            const float4 a = __ldg(at), b = __ldg(at + 1);
            w.src.at = at;
            start(w, a, b);
            slot = __float_as_int(a.w);
        } else if (over && chunk.empty()) {
            w.cur = kSh4Idle;
        }
        if (!__any_sync(kFullMask, w.cur != kSh4Idle)) break;
        do {
            if (sh4_is_node(w.cur)) w.node_step(s, e, ns);
        } while (__popc(__ballot_sync(kFullMask, sh4_is_node(w.cur))) >= quorum);
        if (sh4_is_leaf(w.cur)) w.leaf(s, ns);
        if (sh4_is_switch(w.cur)) w.switch_ray(s, ns);
    }
}

using Sh4QueueStack = Sh4SplitStack<kSh4Shared, kTraceThreads>;

__device__ __forceinline__ void shadow4_queue(const DeviceScene &s, const float4 *__restrict__ q, int n, int *fetch,
                                              unsigned char *occ, int quorum, int *col, unsigned &e) {
    Shadow4Walk<Sh4QueueStack, Sh4RayRecord> w;
    walk4_queue(
        s, w, q, n, fetch, quorum, col,
        [&](auto &x, float4 a, float4 b) { x.start(s, V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, b.w); },
        [&](int slot, const auto &x) { occ[slot] = x.blocked() ? 1 : 0; }, e);
}

// Closest hits (DeviceScene::sh4_closest). With sh4_closest == 2 the hits are then checked by
// check_closest_kernel, for which the triangle's upper bits carry the walk's bound (hit_pack).
__device__ __forceinline__ void closest4_queue(const DeviceScene &s, const float4 *__restrict__ q, int n, int *fetch,
                                               float4 *hits, float *hit_v, int quorum, int *col, unsigned &e) {
    Closest4Walk<Sh4QueueStack, Sh4RayRecord> w;
    walk4_queue(
        s, w, q, n, fetch, quorum, col,
        [&](auto &x, float4 a, float4 b) { x.start(s, V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}); },
        [&](int slot, const auto &x) {
            hits[slot] = make_float4(x.best_t, __int_as_float(x.hit_inst(s)),
                                     __int_as_float(x.found() ? hit_pack(x.hit_tri(s), x.bound_ulps()) : -1), x.best_u);
            hit_v[slot] = x.best_v;
        },
        e);
}

template <int kMinBlocks>
__global__ void __launch_bounds__(kTraceThreads, kMinBlocks) trace_shadow4_kernel(const __grid_constant__ DeviceScene s,
                                                                       const float4 *__restrict__ q, const int *count,
                                                                       int *fetch, unsigned char *occ, int quorum,
                                                                       unsigned *err) {
    __shared__ int col[kSh4Shared * kTraceThreads];
    unsigned e = 0;
    shadow4_queue(s, q, *count, fetch, occ, quorum, col, e);
    if (e) atomicOr(err, e);
}

template <int kMinBlocks>
__global__ void __launch_bounds__(kTraceThreads, kMinBlocks) trace_closest4_kernel(const __grid_constant__ DeviceScene s,
                                                                                 const float4 *__restrict__ q,
                                                                                 int *counts, float4 *hits,
                                                                                 float *hit_v, int quorum,
                                                                                 unsigned *err) {
    __shared__ int col[kSh4Shared * kTraceThreads];
    unsigned e = 0;
    closest4_queue(s, q, counts[0], &counts[3], hits, hit_v, quorum, col, e);
    if (e) atomicOr(err, e);
}

// Both queues in one launch: even blocks take the closest hits first, odd ones the shadow rays,
// each then helps with what is left of the other. A path tracer's late rounds have few rays, and
// the last of them are waited for once instead of twice.
template <int kMinBlocks>
__global__ void __launch_bounds__(kTraceThreads, kMinBlocks) trace_both4_kernel(const __grid_constant__ DeviceScene s,
                                                                              const float4 *__restrict__ q_closest,
                                                                              const float4 *__restrict__ q_shadow,
                                                                              int *counts, float4 *hits, float *hit_v,
                                                                              unsigned char *occ, int quorum,
                                                                              unsigned *err) {
    __shared__ int col[kSh4Shared * kTraceThreads];
    unsigned e = 0;
    for (int pass = 0; pass < 2; ++pass) {
        if ((pass ^ blockIdx.x) & 1)
            shadow4_queue(s, q_shadow, counts[1], &counts[2], occ, quorum, col, e);
        else
            closest4_queue(s, q_closest, counts[0], &counts[3], hits, hit_v, quorum, col, e);
    }
    if (e) atomicOr(err, e);
}

// The check of the SAH walk's closest hits (sh4_closest == 2), one thread per queue entry: an
// entry whose hit ref_reaches cannot vouch for walks the reference's trees here. Few do (of
// 500,000 random rays the unchecked walk answers 19 differently among coplanar boxes, none over
// the terrain), so they get no list and no kernel of their own: the two kernels took 208 us of
// the four rounds of a 256 x 256 path-traced box, this one takes 23. Surfaces within a few units
// in the last place of each other reject more: a room's walls four times over, 0 to 3 units
// apart, 1080p: RIS with all rays 7.5 ms (6.85 with the list), path tracing at depth 4 5.95 (7.4);
// walls twice over are no slower than with it. Walking a block's rejected entries side by side
// was slower still (8.46). A miss needs no check: the SAH trees' boxes hold every triangle, so
// the reference walk finds no hit either.
__global__ void __launch_bounds__(256) check_closest_kernel(const __grid_constant__ DeviceScene s,
                                                            const float4 *__restrict__ q, const int *count,
                                                            float4 *hits, float *hit_v, unsigned *err) {
    const int n = *count;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const float4 a = q[2 * (size_t)k];
        const int slot = __float_as_int(a.w);
        const float4 h = hits[slot];
        const int inst = __float_as_int(h.y), tri = __float_as_int(h.z);
        if (inst < 0) continue;
        const float4 b = q[2 * (size_t)k + 1];
        const V3 o{a.x, a.y, a.z}, d{b.x, b.y, b.z};
        const float bound = __int_as_float(__float_as_int(h.x) + hit_bound_ulps(tri));
        if (ref_reaches(s.dev, o, d, inst, hit_tri(tri), bound)) continue;
        const RefClosest r = reference_closest(s.dev, o, d);
        hits[slot] = make_float4(r.hit.t, __int_as_float(r.hit.inst), __int_as_float(r.hit.tri), r.hit.u);
        hit_v[slot] = r.hit.v;
        if (r.err) atomicOr(err, r.err);
    }
}

// Blocks of a persistent launch over a queue of at most `slots` entries.
int grid_for(int most, size_t slots, int threads) {
    return (int)std::max<size_t>(1, std::min<size_t>((size_t)most, (slots + (size_t)threads - 1) / (size_t)threads));
}

// The shadow-ray queue q (count / fetch counters on the device, answers into occ).
int launch_shadow_queue(const DeviceScene &s, const float4 *q, size_t slots, const int *count, int *fetch,
                        unsigned char *occ, const TraceTuning &tune, unsigned *err, cudaStream_t st) {
    const int tgrid = grid_for(tune.sm_count * tune.blocks_per_sm, slots, kTraceThreads);
    if (s.sh4) {
        // register budget: 64 (8 resident blocks), 80 (6) or 90 (5) per thread
        auto k = tune.shadow_shape == 0 ? trace_shadow4_kernel<8>
                                        : (tune.shadow_shape == 1 ? trace_shadow4_kernel<6> : trace_shadow4_kernel<5>);
        k<<<tgrid, kTraceThreads, 0, st>>>(s, q, count, fetch, occ, tune.node_quorum, err);
    } else {
        const bool shallow = s.shallow && (tune.mode & kTraceSplitStack) == 0;
        auto shadow = s.wide ? trace_shadow_phased_kernel<true, false>
                             : (shallow ? trace_shadow_phased_kernel<false, true>
                                        : trace_shadow_phased_kernel<false, false>);
        shadow<<<tgrid, kTraceThreads, 0, st>>>(s, q, count, fetch, occ, tune.node_quorum, err);
    }
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

template <bool kWide, bool kRefill>
__global__ void __launch_bounds__(kTraceThreads) trace_closest_kernel(DeviceScene s, const float4 *__restrict__ q,
                                                                      int *counts, float4 *hits, float *hit_v,
                                                                      unsigned *err) {
    using TW = TraceWalk<kWide, false>;
    __shared__ typename TW::Entry col[kSharedDepth * kTraceThreads];
    typename TW::Entry deep[kTraceStack - kSharedDepth];
    typename TW::type w;
    w.stack.col = col + threadIdx.x;
    w.stack.deep = deep;
    const int n = counts[0];
    unsigned e = 0;
    NoStats ns;
    if (!kRefill) {
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
            const float4 a = q[2 * (size_t)k], b = q[2 * (size_t)k + 1];
            w.start(s, V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, 0.0f);
            while (w.step(s, e, ns)) {
            }
            const int slot = __float_as_int(a.w);
            hits[slot] = make_float4(w.hit.t, __int_as_float(w.hit.inst), __int_as_float(w.hit.tri), w.hit.u);
            hit_v[slot] = w.hit.v;
        }
    } else {
        int slot = -1;
        bool drained = false;
        for (;;) {
            const int k = fetch_ray(&counts[3], n, slot < 0, drained);
            if (k >= 0) {
                const float4 a = q[2 * (size_t)k], b = q[2 * (size_t)k + 1];
                w.start(s, V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, 0.0f);
                slot = __float_as_int(a.w);
            }
            if (!__any_sync(kFullMask, slot >= 0)) break;
            if (slot >= 0 && !w.step(s, e, ns)) {
                hits[slot] = make_float4(w.hit.t, __int_as_float(w.hit.inst), __int_as_float(w.hit.tri), w.hit.u);
                hit_v[slot] = w.hit.v;
                slot = -1;
            }
        }
    }
    if (e) atomicOr(err, e);
}

template <bool kWide, bool kRefill>
__global__ void __launch_bounds__(kTraceThreads) trace_shadow_kernel(DeviceScene s, const float4 *__restrict__ q,
                                                                     int *counts, unsigned char *occ, unsigned *err) {
    using TW = TraceWalk<kWide, true>;
    __shared__ typename TW::Entry col[kSharedDepth * kTraceThreads];
    typename TW::Entry deep[kTraceStack - kSharedDepth];
    typename TW::type w;
    w.stack.col = col + threadIdx.x;
    w.stack.deep = deep;
    const int n = counts[1];
    unsigned e = 0;
    NoStats ns;
    if (!kRefill) {
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
            const float4 a = q[2 * (size_t)k], b = q[2 * (size_t)k + 1];
            w.start(s, V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, b.w);
            while (w.step(s, e, ns)) {
            }
            occ[__float_as_int(a.w)] = w.shadow_answer() ? 1 : 0;
        }
    } else {
        int slot = -1;
        bool drained = false;
        for (;;) {
            const int k = fetch_ray(&counts[2], n, slot < 0, drained);
            if (k >= 0) {
                const float4 a = q[2 * (size_t)k], b = q[2 * (size_t)k + 1];
                w.start(s, V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, b.w);
                slot = __float_as_int(a.w);
            }
            if (!__any_sync(kFullMask, slot >= 0)) break;
            if (slot >= 0 && !w.step(s, e, ns)) {
                occ[slot] = w.shadow_answer() ? 1 : 0;
                slot = -1;
            }
        }
    }
    if (e) atomicOr(err, e);
}

int launch_wave_trace(const DeviceScene &s, WaveBuffers wb, const TraceTuning &tune, unsigned *err, cudaStream_t st,
                      cudaEvent_t *ev_begin, cudaEvent_t *ev_end) {
    auto mark = [&](cudaEvent_t *ev, int k) { return !ev || cudaEventRecord(ev[k], st) == cudaSuccess; };
    const bool refill = (tune.mode & kTraceLanePerRay) == 0;
    // a lane that keeps its ray has its share of the queue fixed by the grid: smaller shares
    const int most = tune.sm_count * tune.blocks_per_sm * (refill ? 1 : 2);
    const int cgrid = grid_for(most, wb.closest_slots, kTraceThreads);
    const int sgrid = grid_for(most, wb.shadow_slots, kTraceThreads);
    const bool phased = refill && (tune.mode & kTraceUnphased) == 0;
    const bool shallow = s.shallow && (tune.mode & kTraceSplitStack) == 0;
    const bool both = s.sh4 && s.sh4_closest && wb.closest_slots > 0 && !ev_begin;  // not timed one by one
    if (!mark(ev_begin, 0)) return -1;
    int launches = 0;
    if (both) {
        const int grid = grid_for(most, wb.closest_slots + wb.shadow_slots, kTraceThreads);
        auto k = tune.shadow_shape == 0 ? trace_both4_kernel<8>
                                        : (tune.shadow_shape == 1 ? trace_both4_kernel<6> : trace_both4_kernel<5>);
        k<<<grid, kTraceThreads, 0, st>>>(s, wb.q_closest, wb.q_shadow, wb.counts, wb.hits, wb.hit_v, wb.occ,
                                          tune.node_quorum, err);
        ++launches;
    } else if (wb.closest_slots == 0) {
        // no closest-hit queue (kTraceNoBsdfRays)
    } else if (s.sh4_closest) {
        auto closest = tune.shadow_shape == 0 ? trace_closest4_kernel<8>
                                              : (tune.shadow_shape == 1 ? trace_closest4_kernel<6>
                                                                        : trace_closest4_kernel<5>);
        closest<<<cgrid, kTraceThreads, 0, st>>>(s, wb.q_closest, wb.counts, wb.hits, wb.hit_v, tune.node_quorum, err);
        ++launches;
    } else if (phased) {
        auto closest = s.wide    ? trace_closest_phased_kernel<true, false>
                       : shallow ? trace_closest_phased_kernel<false, true>
                                 : trace_closest_phased_kernel<false, false>;
        closest<<<cgrid, kTraceThreads, 0, st>>>(s, wb.q_closest, wb.counts, wb.counts + 3, wb.hits, wb.hit_v,
                                                 tune.node_quorum, err);
        ++launches;
    } else {
        auto closest = s.wide ? (refill ? trace_closest_kernel<true, true> : trace_closest_kernel<true, false>)
                              : (refill ? trace_closest_kernel<false, true> : trace_closest_kernel<false, false>);
        closest<<<cgrid, kTraceThreads, 0, st>>>(s, wb.q_closest, wb.counts, wb.hits, wb.hit_v, err);
        ++launches;
    }
    if (wb.closest_slots > 0 && s.sh4_closest == 2) {
        check_closest_kernel<<<grid_for(tune.sm_count * 8, wb.closest_slots, 256), 256, 0, st>>>(
            s, wb.q_closest, wb.counts, wb.hits, wb.hit_v, err);
        ++launches;
    }
    if (!mark(ev_end, 0) || !mark(ev_begin, 1)) return -1;
    if (both) {
    } else if (phased || s.sh4) {
        if (launch_shadow_queue(s, wb.q_shadow, wb.shadow_slots, wb.counts + 1, wb.counts + 2, wb.occ, tune, err, st) < 0)
            return -1;
        ++launches;
    } else {
        auto shadow = s.wide ? (refill ? trace_shadow_kernel<true, true> : trace_shadow_kernel<true, false>)
                             : (refill ? trace_shadow_kernel<false, true> : trace_shadow_kernel<false, false>);
        shadow<<<sgrid, kTraceThreads, 0, st>>>(s, wb.q_shadow, wb.counts, wb.occ, err);
        ++launches;
    }
    if (!mark(ev_end, 1)) return -1;
    return cudaPeekAtLastError() == cudaSuccess ? launches : -1;
}

}  // namespace hdr
