// Shadow-ray walk over the shadow BVH (host/shadow_bvh.h): "is there a hit
// nearer than the limit", the visibility query of _evaluateLightSample
// (ris_direct_light_integrator.cpp:628-658) and of the MIS integrator's NEE.
//
// The answer is the reference's: a triangle blocks the ray exactly when
// IntersectTriangle (bvh.cpp:8-30, restated in tri_test) returns t < limit for
// it in its instance's space, which is the same arithmetic on the same records
// whatever tree finds it. The trees only cull, so their box tests are made
// conservative: bounds are rounded outward on the node's grid, the near and far slab
// distances are computed with the reciprocal direction shrunk and grown by 2^-20 and
// offset by 2^-20 of the origin term, which covers the rounding of
// t = bound * (1/d) - o * (1/d), so a box is never skipped when a ray hits a
// triangle inside it. (The reference culls with its own rounded slab tests on
// its own boxes; it can miss a hit that grazes a box face by an ulp, which no
// tree change reproduces. Such rays are counted by the tests.)
//
// What bounds the walk, on the 14.5 M shadow rays of a 1080p terrain frame (1.03 M
// triangles, 2001 instances; 6.93 ms before, 3.47 ms now):
//  * L1's data stage. A divergent load takes a pass for nearly every line it touches.
//    112-byte float nodes in seven 128-bit loads kept the stage 62 % busy next to an issue
//    rate of 63 % (93 % once the instructions were halved); 64-byte nodes of byte bounds in
//    two 256-bit loads leave it at 60 %.
//  * Instructions: 379 warp instructions per ray before, 200 now. The ray's own order of the
//    children does not shorten a shadow walk (22.9 steps either way), so children are tried as
//    they stand; entries need no decoding; near and far bounds share the two halves of
//    packed multiply-adds; three-operand min and max; an end marker instead of a test at
//    every pop.
//  * Registers: one ray at a time (the world ray is read again after an instance) fits 64
//    without spills in the loop, 8 resident blocks of 128 instead of 6.
#pragma once

#include "gf.cuh"
#include "sh4_layout.h"

namespace hdr {

constexpr unsigned kErrShadowStack = 16u;

// The walk's entry in hand: a child entry of sh4_layout.h, or one of these (their
// instance bit is set, so one comparison tells a node from everything else).
constexpr int kSh4World = 0x7ffffffb;  // back from an instance to the world ray
constexpr int kSh4Hit = 0x7ffffffc;    // shadow walk over: a triangle blocks the ray
constexpr int kSh4Done = 0x7ffffffd;   // walk over
constexpr int kSh4Idle = 0x7ffffffe;   // lane without a ray

__device__ __forceinline__ bool sh4_is_node(int e) { return (unsigned)e < (unsigned)kSh4InstBit; }
__device__ __forceinline__ bool sh4_is_leaf(int e) { return e < 0; }
__device__ __forceinline__ bool sh4_is_switch(int e) { return e >= kSh4InstBit && e <= kSh4World; }
__device__ __forceinline__ bool sh4_is_over(int e) { return e == kSh4Hit || e == kSh4Done; }

// Two floats in one 64-bit register: fma.rn.f32x2 and add.rn.f32x2 work on both in one
// instruction, each half rounded as the scalar form rounds it.
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_get(F2 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// A ray prepared for the 4-child box tests: near and far values side by side.
struct Sh4Axis {
    F2 inv;         // 1/d shrunk by 2^-20 | grown by 2^-20
    F2 off;         // -o/d, conservatively lowered | raised
    unsigned pick;  // byte selector of the near bounds in (minima, maxima): the minima, or the
                    // maxima where the direction is negative
};
struct Sh4Ray {
    Sh4Axis x, y, z;
};

__device__ __forceinline__ Sh4Axis sh4_axis(float o, float d) {
    const float dd = fabsf(d) > 1e-20f ? d : copysignf(1e-20f, d);
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(dd));  // within one unit in the last place
    const float in = inv * (1.0f - 9.5367431640625e-07f), inf = inv * (1.0f + 9.5367431640625e-07f);
    const float e = fabsf(o * inv) * 9.5367431640625e-07f;
    Sh4Axis a;
    a.inv = f2(in, inf);
    a.off = f2(-o * in - e, -o * inf + e);
    a.pick = dd < 0.0f ? 0x7654u : 0x3210u;
    return a;
}

__device__ __forceinline__ Sh4Ray sh4_ray(V3 o, V3 d) {
    return Sh4Ray{sh4_axis(o.x, d.x), sh4_axis(o.y, d.y), sh4_axis(o.z, d.z)};
}

// max(a, b, c) / min(a, b, c) in one instruction, NaN operands ignored like fmaxf / fminf
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// 32 bytes in one load (as four 64-bit words: the assembler of CUDA 12.9 crashes on the form
// with eight 32-bit words in the larger kernels)
__device__ __forceinline__ void load_256(unsigned long long at, unsigned v[8]) {
    unsigned long long w[4];
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3]) : "l"(at));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[2 * k] = (unsigned)w[k];
        v[2 * k + 1] = (unsigned)(w[k] >> 32);
    }
}

// Entry and exit distances of the four children along one axis: a bound is 1 + byte / 32768
// (the byte put into a float's mantissa) times scale, plus origin. Near and far go through
// each instruction together.
__device__ __forceinline__ void sh4_slabs(unsigned minima, unsigned maxima, unsigned origin, unsigned scale,
                                          const Sh4Axis &a, float near[4], float far[4]) {
    const float s = __uint_as_float(scale), o = __uint_as_float(origin);
    const F2 s2 = f2_mul(f2(s, s), a.inv), o2 = f2_fma(f2(o, o), a.inv, a.off);
    const unsigned n = __byte_perm(minima, maxima, a.pick), f = __byte_perm(maxima, minima, a.pick);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const unsigned at = 0x7604u | (unsigned)k << 4;
        const F2 q = f2(__uint_as_float(__byte_perm(n, 0x3f800000u, at)),
                        __uint_as_float(__byte_perm(f, 0x3f800000u, at)));
        f2_get(f2_fma(q, s2, o2), near[k], far[k]);
    }
}

// The four child boxes of a node against the ray: child k's box overlaps [0, limit]
// along the ray exactly when t0[k] <= t1[k]; t0[k] is its entry distance.
__device__ __forceinline__ void sh4_children(const float4 *nodes, int idx, const Sh4Ray &r, float limit, float t0[4],
                                             float t1[4], int code[4]) {
    const unsigned long long node = (unsigned long long)nodes + 64ull * (unsigned)idx;
    const unsigned turn = ((unsigned)idx << 4) & 32u;  // sh4_slot_of
    unsigned a[8], b[8];
    load_256(node | turn, a);
    load_256(node | (turn ^ 32u), b);
    float nx[4], ny[4], nz[4], fx[4], fy[4], fz[4];
    sh4_slabs(a[6], a[7], a[0], a[3], r.x, nx, fx);
    sh4_slabs(b[0], b[1], a[1], a[4], r.y, ny, fy);
    sh4_slabs(b[2], b[3], a[2], a[5], r.z, nz, fz);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        code[k] = (int)b[4 + k];
        t0[k] = fmaxf(max3f(nx[k], ny[k], nz[k]), 0.0f);
        t1[k] = fminf(min3f(fx[k], fy[k], fz[k]), limit);
    }
}

// IntersectTriangle (bvh.cpp:8-30) on a tri_geo record, as tri_test.
__device__ __forceinline__ bool sh4_tri_blocks(V3 o, V3 d, const float4 *g, float limit) {
    const float4 g0 = __ldg(g), g1 = __ldg(g + 1), g2 = __ldg(g + 2);
    const V3 v0{g0.x, g0.y, g0.z};
    const V3 e1{g0.w, g1.x, g1.y};
    const V3 e2{g1.z, g1.w, g2.x};
    const V3 pvec = cross(d, e2);
    const float det = dot(e1, pvec);
    if (fabsf(det) <= 9.99999993922529e-09f) return false;  // std::abs(det) < 1e-8 (double)
    const float inv_det = 1.0f / det;
    const V3 tvec = o - v0;
    const float u = dot(tvec, pvec) * inv_det;
    if (u < 0.0f || u > 1.0f) return false;
    const V3 qvec = cross(tvec, e1);
    const float v = dot(d, qvec) * inv_det;
    if (v < 0.0f || u + v > 1.0f) return false;
    const float t = dot(e2, qvec) * inv_det;
    return t > 1e-4f && t < limit;
}

// Where a walk finds its world ray again when it leaves an instance.
struct Sh4RayValue {
    V3 o, d;
    __device__ __forceinline__ void get(V3 &wo, V3 &wd) const { wo = o, wd = d; }
};
struct Sh4RayRecord {  // a ray queue entry: origin.xyz, slot | direction.xyz, limit
    const float4 *at;
    __device__ __forceinline__ void get(V3 &wo, V3 &wd) const {
        const float4 a = __ldg(at), b = __ldg(at + 1);
        wo = V3{a.x, a.y, a.z}, wd = V3{b.x, b.y, b.z};
    }
};

// What both walks share: a resumable state machine over one ray at a time, the world
// ray or, inside an instance, its object-space ray (keeping both cost 19 registers and
// spills). `cur` is the entry in hand; the caller serves it by kind: a node step tests
// the node's four child boxes, takes one hit child into hand and pushes the others;
// leaves and ray switches (into an instance, or back) are served in their own phases,
// so that the node steps of a warp stay in step.
template <class Stk, class Src>
struct Walk4Base {
    V3 oo, od;
    Sh4Ray r;
    int cur;
    Stk stack;
    Src src;

    // an end marker stands at the bottom of the stack, so popping needs no test
    __device__ __forceinline__ void begin(const DeviceScene &s, V3 o, V3 d) {
        oo = o;
        od = d;
        r = sh4_ray(o, d);
        stack.reset(kSh4Done);
        cur = s.has_tlas ? 0 : kSh4Done;
    }
    __device__ __forceinline__ void next() { cur = stack.pop(); }

    // the hit children in order: the first in hand, the others pushed so that the next comes out first
    template <class Hit>
    __device__ __forceinline__ void take(const int code[4], Hit hit, unsigned &err) {
        int in_hand = kSh4Done;
        bool any = false;
        if (stack.fast(4)) {  // the pushes and the pop stay in the fast part of the stack
#pragma unroll
            for (int k = 3; k >= 0; --k) {
                const bool h = hit(k);
                stack.push_fast_if(h && any, in_hand);
                if (h) in_hand = code[k];
                any = any || h;
            }
            cur = any ? in_hand : stack.pop_fast();
            return;
        }
        if (!stack.room(4)) {
            err |= kErrShadowStack;
            cur = kSh4Done;
            return;
        }
#pragma unroll
        for (int k = 3; k >= 0; --k)
            if (hit(k)) {
                if (any) stack.push(in_hand);
                in_hand = code[k];
                any = true;
            }
        cur = any ? in_hand : stack.pop();
    }

    // enter an instance (returns its index), or go back to the world ray (-1)
    __device__ __forceinline__ int switch_ray(const DeviceScene &s) {
        const int e = cur;
        V3 o, d;
        src.get(o, d);
        int ii = -1;
        if (e != kSh4World) {
            ii = e & (kSh4InstBit - 1);
            const float4 *ip = s.instances + 8 * (size_t)ii;
            const float4 m0 = __ldg(ip), m1 = __ldg(ip + 1), m2 = __ldg(ip + 2), m3 = __ldg(ip + 3);
            const float inv[16] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w,
                                   m2.x, m2.y, m2.z, m2.w, m3.x, m3.y, m3.z, m3.w};
            // GfMatrix4f::Transform divides by w; an affine matrix makes it 1 and the division exact
            if (m0.w == 0.0f && m1.w == 0.0f && m2.w == 0.0f && m3.w == 1.0f)
                oo = m4f_transform_affine(inv, o);
            else
                oo = m4f_transform(inv, o);
            od = m4f_transform_dir(inv, d);
            if (!stack.bottom()) stack.push(kSh4World);
            cur = __ldg(&s.sh4_inst_root[ii]);
        } else {
            oo = o;
            od = d;
            next();
        }
        r = sh4_ray(oo, od);
        return ii;
    }
};

// The shadow walk. The children of a node stand in the order they are tried.
template <class Stk, class Src>
struct Shadow4Walk : Walk4Base<Stk, Src> {
    using B = Walk4Base<Stk, Src>;
    float limit;

    __device__ __forceinline__ void start(const DeviceScene &s, V3 o, V3 d, float lim) {
        limit = lim;
        B::begin(s, o, d);
    }
    __device__ __forceinline__ bool blocked() const { return B::cur == kSh4Hit; }

    // one node entry
    template <class St>
    __device__ __forceinline__ void node_step(const DeviceScene &s, unsigned &err, St &st) {
        st.pop();
        float t0[4], t1[4];
        int code[4];
        sh4_children(s.sh4_nodes, B::cur, B::r, limit, t0, t1, code);
        B::take(code, [&](int k) { return t0[k] <= t1[k]; }, err);
    }

    // a leaf's triangles
    template <class St>
    __device__ __forceinline__ void leaf(const DeviceScene &s, St &st) {
        const int p = ~B::cur, first = p >> 2, cnt = (p & 3) + 1;
        st.leaf();
        for (int q = 0; q < cnt; ++q) {
            st.tri();
            if (sh4_tri_blocks(B::oo, B::od, s.sh4_tris + 3 * (size_t)(first + q), limit)) {
                B::cur = kSh4Hit;
                return;
            }
        }
        B::next();
    }

    template <class St>
    __device__ __forceinline__ void switch_ray(const DeviceScene &s, St &st) {
        if (B::cur != kSh4World) st.leaf();
        (void)B::switch_ray(s);
    }
};

// Entries below kShared in this thread's column of a shared-memory array, the
// rest (up to kSh4Stack) in a per-thread local array. The stack pointer of the
// column is its shared-memory address.
template <int kShared, int kThreads>
struct Sh4SplitStack {
    static constexpr unsigned kStride = 4u * kThreads;
    unsigned base, sp;  // address of entry 0, of the next free entry
    int *deep;
    __device__ __forceinline__ void bind(int *col, int *deep_entries) {
        base = (unsigned)__cvta_generic_to_shared(col);
        sp = base;
        deep = deep_entries;
    }
    __device__ __forceinline__ int depth() const { return (int)((sp - base) / kStride); }
    __device__ __forceinline__ bool fast(int n) const { return sp <= base + (unsigned)(kShared - n) * kStride; }
    __device__ __forceinline__ bool room(int n) const { return depth() + n <= kSh4Stack; }
    __device__ __forceinline__ bool bottom() const { return sp == base + kStride; }
    __device__ __forceinline__ void push_fast_if(bool want, int v) {
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p st.shared.s32 [%0], %1;\n}" ::"r"(sp), "r"(v),
                     "r"((int)want));
        sp += want ? kStride : 0u;
    }
    __device__ __forceinline__ int pop_fast() {
        sp -= kStride;
        int v;
        asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(sp));
        return v;
    }
    __device__ __forceinline__ void push(int v) {
        if (fast(1))
            push_fast_if(true, v);
        else {
            deep[depth() - kShared] = v;
            sp += kStride;
        }
    }
    __device__ __forceinline__ int pop() {
        if (fast(0)) return pop_fast();
        sp -= kStride;
        return deep[depth() - kShared];
    }
    __device__ __forceinline__ void reset(int end) {
        sp = base;
        push_fast_if(true, end);
    }
};

template <class T, int kCap>
struct Sh4LocalStack {
    T e[kCap];
    int sp;
    __device__ __forceinline__ bool fast(int n) const { return sp + n <= kCap; }
    __device__ __forceinline__ bool room(int n) const { return sp + n <= kCap; }
    __device__ __forceinline__ bool bottom() const { return sp == 1; }
    __device__ __forceinline__ void push(T v) { e[sp++] = v; }
    __device__ __forceinline__ T pop() { return e[--sp]; }
    __device__ __forceinline__ void push_fast_if(bool want, T v) {
        if (want) push(v);
    }
    __device__ __forceinline__ T pop_fast() { return pop(); }
    __device__ __forceinline__ void reset(T end) {
        e[0] = end;
        sp = 1;
    }
};

// Closest-hit walk over the same trees (IntersectScene, scene.cpp:409-535), with
// the reference's answer: boxes are culled only beyond the running closest t
// (conservatively, as above), every triangle test is IntersectTriangle in its
// instance's space, and among hits at equal t the smallest (instance position in
// the reference TLAS's leaf order, triangle index in the reference BLAS order)
// wins, the hit the reference's left-first walks meet first with their strict
// `<`. The nearest hit child is taken into hand, the others are pushed as they stand
// (sorting them too saves 1 % of the node steps).
//
// second_t is the nearest hit seen beyond the closest one's distance. Boxes are culled 2^-18
// of the way beyond the closest t, so every triangle hit up to 15 units in the last place
// (less than 2^-19) beyond it has been tested: bound() is the distance below which the
// reference's walk has no hit when it comes to the closest one's triangle. Hits at the very
// distance do not lower it, for the closest one is the first of them in that walk's order. (With
// no slack left for a hit that another surface coincides with, the check rejected the hits on
// coincident walls: 65 boxes twice over, 1080p: RIS with all rays 3.00 -> 2.05 ms, path tracing
// at depth 4 1.75 -> 1.22, primary rays 0.38 -> 0.15.)
constexpr float kSh4CullPast = 1.0f + 3.814697265625e-06f;
constexpr int kSh4BoundUlps = 15;

template <class Stk, class Src>
struct Closest4Walk : Walk4Base<Stk, Src> {
    using B = Walk4Base<Stk, Src>;
    float best_t, second_t, best_u, best_v;
    int best_rec;   // triangle record of the hit, -1 = none
    int best_inst;  // its instance, -1 = the opened one of its mesh
    int cur_inst;   // the instance the ray is in, -1 = the world

    __device__ __forceinline__ void start(const DeviceScene &s, V3 o, V3 d) {
        best_t = 1e30f;  // IntersectScene's initial closest distance
        second_t = 1e30f;
        best_u = best_v = 0.0f;
        best_rec = best_inst = cur_inst = -1;
        B::begin(s, o, d);
    }
    __device__ __forceinline__ bool found() const { return best_rec >= 0; }
    __device__ __forceinline__ static int rec_inst(const DeviceScene &s, int rec, int inst) {
        return inst >= 0 ? inst : __ldg(&s.sh4_mesh_world[__float_as_int(__ldg(&s.sh4_tris[3 * (size_t)rec + 2].z))]);
    }
    __device__ __forceinline__ static int rec_tri(const DeviceScene &s, int rec) {
        return __float_as_int(__ldg(&s.sh4_tris[3 * (size_t)rec + 2].y));
    }
    __device__ __forceinline__ int hit_inst(const DeviceScene &s) const {
        return found() ? rec_inst(s, best_rec, best_inst) : -1;
    }
    __device__ __forceinline__ int hit_tri(const DeviceScene &s) const { return found() ? rec_tri(s, best_rec) : -1; }
    // units in the last place of best_t up to which no other hit lies
    __device__ __forceinline__ int bound_ulps() const {
        const int u = __float_as_int(second_t) - __float_as_int(best_t);
        return u < kSh4BoundUlps ? u : kSh4BoundUlps;
    }
    __device__ __forceinline__ float bound() const { return __int_as_float(__float_as_int(best_t) + bound_ulps()); }

    template <class St>
    __device__ __forceinline__ void node_step(const DeviceScene &s, unsigned &err, St &st) {
        st.pop();
        float t0[4], t1[4];
        int code[4];
        sh4_children(s.sh4_nodes, B::cur, B::r, best_t * kSh4CullPast, t0, t1, code);
        // entry distances are >= 0: their bits order like the values; the slot breaks ties
        unsigned key[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            key[k] = t0[k] <= t1[k] ? ((__float_as_uint(t0[k]) & ~3u) | (unsigned)k) : 0xffffffffu;
        const unsigned nearest = umin(umin(key[0], key[1]), umin(key[2], key[3]));
        const int first = nearest & 3u;
        // the nearest child moved to the front, the others as they stand
        const int moved[4] = {first == 0 ? code[0] : (first == 1 ? code[1] : (first == 2 ? code[2] : code[3])),
                              first == 1 ? code[0] : code[1], first == 2 ? code[0] : code[2],
                              first == 3 ? code[0] : code[3]};
        const bool hit0 = key[0] != 0xffffffffu;
        const bool hits[4] = {nearest != 0xffffffffu, first == 1 ? hit0 : key[1] != 0xffffffffu,
                              first == 2 ? hit0 : key[2] != 0xffffffffu, first == 3 ? hit0 : key[3] != 0xffffffffu};
        B::take(moved, [&](int k) { return hits[k]; }, err);
    }

    template <class St>
    __device__ __forceinline__ void leaf(const DeviceScene &s, St &st) {
        const int p = ~B::cur, first = p >> 2, cnt = (p & 3) + 1;
        st.leaf();
        for (int q = 0; q < cnt; ++q) {
            st.tri();
            const int rec = first + q;
            float t, u, v;
            if (!tri_test(B::oo, B::od, s.sh4_tris + 3 * (size_t)rec, t, u, v)) continue;
            if (t > best_t) {
                second_t = fminf(second_t, t);
                continue;
            }
            if (t == best_t && found()) {
                const int ra = __ldg(&s.sh4_inst_rank[rec_inst(s, rec, cur_inst)]);
                const int rb = __ldg(&s.sh4_inst_rank[rec_inst(s, best_rec, best_inst)]);
                if (!(ra < rb || (ra == rb && rec_tri(s, rec) < rec_tri(s, best_rec)))) continue;
            } else {
                second_t = best_t;
            }
            best_t = t;
            best_u = u;
            best_v = v;
            best_rec = rec;
            best_inst = cur_inst;
        }
        B::next();
    }

    template <class St>
    __device__ __forceinline__ void switch_ray(const DeviceScene &s, St &st) {
        if (B::cur != kSh4World) st.leaf();
        cur_inst = B::switch_ray(s);
    }
};

// One ray's walk to its end (callers outside the wavefront trace kernels).
template <class W, class St>
__device__ __forceinline__ void walk4_ray(const DeviceScene &s, W &w, unsigned &err, St &st) {
    for (;;) {
        while (sh4_is_node(w.cur)) w.node_step(s, err, st);
        if (sh4_is_leaf(w.cur))
            w.leaf(s, st);
        else if (sh4_is_switch(w.cur))
            w.switch_ray(s, st);
        else
            return;
    }
}

template <class St>
__device__ inline bool shadow4_ray(const DeviceScene &s, V3 o, V3 d, float limit, unsigned &err, St &st) {
    Shadow4Walk<Sh4LocalStack<int, kSh4Stack>, Sh4RayValue> w;
    w.src = Sh4RayValue{o, d};
    w.start(s, o, d, limit);
    walk4_ray(s, w, err, st);
    return w.blocked();
}

// Closest hit of one ray; bound: the distance up to which no other hit lies.
template <class St>
__device__ inline bool closest4_ray(const DeviceScene &s, V3 o, V3 d, HitId &hit, float &bound, unsigned &err,
                                    St &st) {
    Closest4Walk<Sh4LocalStack<int, kSh4Stack>, Sh4RayValue> w;
    w.src = Sh4RayValue{o, d};
    w.start(s, o, d);
    walk4_ray(s, w, err, st);
    hit.t = w.best_t;
    hit.inst = w.hit_inst(s);
    hit.tri = w.hit_tri(s);
    hit.u = w.best_u;
    hit.v = w.best_v;
    bound = w.bound();
    return w.found();
}

}  // namespace hdr
