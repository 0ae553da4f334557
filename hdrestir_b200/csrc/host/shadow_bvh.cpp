// Shadow-ray BVH builder (see shadow_bvh.h).
#include "shadow_bvh.h"

#include "scene_build.h"

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <future>
#include <system_error>

#include "../device/tri_setup.cuh"

namespace hdr {

namespace {

// Triangles per leaf. A leaf is served one triangle at a time by the few lanes of a warp that
// hold one, so smaller leaves in a deeper tree pay: 2 / 3 / 4 triangles take 3.47 / 3.51 /
// 3.67 ms for the 14.5 M shadow rays and 7.50 / 7.55 / 7.75 ms for the 31 M closest hits of
// a 1080p terrain frame.
constexpr int kSh4LeafTris = 2;

struct PrimBox {
    float lo[3], hi[3], c[3];
};

// Coordinates the node encoding serves; beyond them the reference's trees are walked. The walk
// multiplies a node's scale, 128.5 times its extent, by up to 1e20 (sh4_axis's reciprocal of a
// direction along which the ray does not move): 2.7e18 * 1e20 stays below the largest float, so
// that scale and origin do not overflow one without the other.
constexpr float kSh4MaxBound = 1e16f;
inline bool encodable(const float *lo, const float *hi) {
    for (int k = 0; k < 3; ++k)
        if (!(std::fabs(lo[k]) < kSh4MaxBound) || !(std::fabs(hi[k]) < kSh4MaxBound)) return false;
    return true;
}

struct BNode {  // binary SAH node: inner (left >= 0: children left, left + 1) or leaf (prims first..first+count)
    float lo[3], hi[3];
    int left = -1, first = 0, count = 0;
};

inline float half_area(const float *lo, const float *hi) {
    const float x = hi[0] - lo[0], y = hi[1] - lo[1], z = hi[2] - lo[2];
    return (x < 0.0f || y < 0.0f || z < 0.0f) ? 0.0f : x * y + y * z + z * x;
}

inline void grow(float *lo, float *hi, const float *a, const float *b) {
    for (int k = 0; k < 3; ++k) {
        lo[k] = std::min(lo[k], a[k]);
        hi[k] = std::max(hi[k], b[k]);
    }
}

// x, y, z and an unused lane
typedef float F4 __attribute__((vector_size(16)));
typedef int I4 __attribute__((vector_size(16)));
inline F4 load3(const float *v) { return F4{v[0], v[1], v[2], 0.0f}; }
struct Box4 {
    F4 lo{FLT_MAX, FLT_MAX, FLT_MAX, 0.0f}, hi{-FLT_MAX, -FLT_MAX, -FLT_MAX, 0.0f};
    void grow(F4 a, F4 b) {
        lo = a < lo ? a : lo;
        hi = hi < b ? b : hi;
    }
    float half_area() const {
        const F4 d = hi - lo;
        return (d[0] < 0.0f || d[1] < 0.0f || d[2] < 0.0f) ? 0.0f : d[0] * d[1] + d[1] * d[2] + d[2] * d[0];
    }
};

// Binned SAH (16 bins per axis over the centroid bounds), leaves of at most
// max_leaf primitives. The primitives themselves are partitioned, so every node reads a
// consecutive range; order[] is the resulting leaf order. Empty bins cost nothing (most
// nodes hold a few primitives), and the two halves of a large node are built at the same
// time: the tree does not depend on how many threads there are, only the place of a node in
// the array does. A box is one register pair, and only bins that hold something are swept: a
// top level of 3,024 leaves, built again whenever instances move, 3.3 -> 2.2 ms on one core, 1.7
// on several. All trees of 523 thousand triangles on 8 cores: 0.43 s with one thread and leaves
// of four triangles before, 0.24 s now.
class SahBuilder {
  public:
    SahBuilder(const std::vector<PrimBox> &prims, int max_leaf, std::vector<BNode> &nodes)
        : refs_(prims.size()), nodes_(nodes), max_leaf_(max_leaf) {
        for (size_t i = 0; i < prims.size(); ++i)
            refs_[i] = {load3(prims[i].lo), load3(prims[i].hi), load3(prims[i].c), (int)i};
        nodes_.assign(std::max<size_t>(1, 2 * prims.size()), BNode());
    }
    void build(std::vector<int> &order) {
        build_range({0, 0, (int)refs_.size()}, 0);
        nodes_.resize((size_t)used_.load());
        order.resize(refs_.size());
        for (size_t i = 0; i < refs_.size(); ++i) order[i] = refs_[i].index;
    }

  private:
    static constexpr int kBins = 16, kParallelPrims = 512, kParallelDepth = 4;
    struct Ref {
        F4 lo, hi, c;
        int index;
    };
    struct Bin {
        F4 lo, hi;
        int count;
    };
    struct Task {
        int node, start, end;
    };

    void build_range(Task root, int depth) {
        std::vector<Task> todo{root};
        while (!todo.empty()) {
            const Task t = todo.back();
            todo.pop_back();
            const int mid = split(t);
            if (mid < 0) continue;
            const int l = used_.fetch_add(2);
            nodes_[(size_t)t.node].left = l;
            const Task left{l, t.start, mid}, right{l + 1, mid, t.end};
            if (depth < kParallelDepth && t.end - t.start >= kParallelPrims) {
                std::future<void> other;
                try {
                    other = std::async(std::launch::async, [this, right, depth] { build_range(right, depth + 1); });
                } catch (const std::system_error &) {  // no thread to be had
                }
                build_range(left, depth + 1);
                if (other.valid())
                    other.get();
                else
                    build_range(right, depth + 1);
                continue;
            }
            todo.push_back(right);
            todo.push_back(left);
        }
    }

    // The node's bounds, and where its primitives are parted (-1: it is a leaf).
    int split(const Task &t) {
        Box4 box, centres;
        for (int i = t.start; i < t.end; ++i) {
            const Ref &p = refs_[(size_t)i];
            box.grow(p.lo, p.hi);
            centres.grow(p.c, p.c);
        }
        BNode &nd = nodes_[(size_t)t.node];
        for (int k = 0; k < 3; ++k) nd.lo[k] = box.lo[k], nd.hi[k] = box.hi[k];
        if (t.end - t.start <= max_leaf_) {
            nd.first = t.start;
            nd.count = t.end - t.start;
            return -1;
        }
        const F4 clo = centres.lo, extent = centres.hi - clo;
        const F4 scale = extent > 0.0f ? (float)kBins / extent : F4{};
        auto bins_of = [&](const Ref &p) {
            const I4 b = __builtin_convertvector((p.c - clo) * scale, I4);
            const I4 from0 = b > 0 ? b : I4{};
            return from0 < kBins - 1 ? from0 : I4{} + (kBins - 1);
        };
        struct {
            Bin bin[kBins];
            unsigned used = 0;  // bit b: bin b holds a primitive
        } axis[3];
        for (int i = t.start; i < t.end; ++i) {
            const Ref &p = refs_[(size_t)i];
            const I4 at = bins_of(p);
            for (int ax = 0; ax < 3; ++ax) {
                if (!(scale[ax] > 0.0f)) continue;
                Bin &b = axis[ax].bin[at[ax]];
                if (axis[ax].used >> at[ax] & 1u) {
                    b.lo = p.lo < b.lo ? p.lo : b.lo;
                    b.hi = b.hi < p.hi ? p.hi : b.hi;
                    ++b.count;
                } else {
                    axis[ax].used |= 1u << at[ax];
                    b.lo = p.lo, b.hi = p.hi;
                    b.count = 1;
                }
            }
        }
        float best = FLT_MAX;
        int best_axis = -1, best_bin = 0;
        for (int ax = 0; ax < 3; ++ax) {
            // the splits above each bin that holds something, but the highest: from the top what lies
            // above them, then from below
            int held[kBins], n_held = 0;
            for (unsigned left = axis[ax].used; left; left &= left - 1) held[n_held++] = __builtin_ctz(left);
            float area[kBins];
            int count[kBins];
            Box4 above, below;
            int acc = 0;
            for (int k = n_held - 1; k > 0; --k) {
                const Bin &bin = axis[ax].bin[held[k]];
                acc += bin.count;
                above.grow(bin.lo, bin.hi);
                area[k] = above.half_area();
                count[k] = acc;
            }
            acc = 0;
            for (int k = 0; k + 1 < n_held; ++k) {
                const Bin &bin = axis[ax].bin[held[k]];
                acc += bin.count;
                below.grow(bin.lo, bin.hi);
                const float cost = below.half_area() * (float)acc + area[k + 1] * (float)count[k + 1];
                if (cost < best) {
                    best = cost;
                    best_axis = ax;
                    best_bin = held[k] + 1;
                }
            }
        }
        if (best_axis >= 0) {
            const int m = (int)(std::partition(refs_.begin() + t.start, refs_.begin() + t.end,
                                               [&](const Ref &r) { return bins_of(r)[best_axis] < best_bin; }) -
                                refs_.begin());
            if (m > t.start && m < t.end) return m;
        }
        return (t.start + t.end) / 2;
    }

    std::vector<Ref> refs_;
    std::vector<BNode> &nodes_;
    std::atomic<int> used_{1};
    int max_leaf_;
};

void build_binary(const std::vector<PrimBox> &prims, int max_leaf, std::vector<BNode> &nodes, std::vector<int> &order) {
    SahBuilder(prims, max_leaf, nodes).build(order);
}

inline float bits_float(int v) {
    float f;
    std::memcpy(&f, &v, sizeof(f));
    return f;
}

// A node as the builder handles it.
struct Node4 {
    float lo[4][3], hi[4][3];
    int entry[4];
    int children = 0;
    void add(const float *l, const float *h, int e) {
        std::memcpy(lo[children], l, sizeof(lo[0]));
        std::memcpy(hi[children], h, sizeof(hi[0]));
        entry[children++] = e;
    }
};

inline int float_int(float v) {
    int i;
    std::memcpy(&i, &v, sizeof(i));
    return i;
}

// The node's bounds on a grid of 255 steps per axis (sh4_layout.h). Every bound is first
// widened by 2^-13 of the node's extent and 2^-20 of itself: the walk evaluates
// origin / d and scale / d rounded to float, 128 times the extent in magnitude.
void store_node(std::vector<float> &nodes, int index, const Node4 &n) {
    float *a = &nodes[(size_t)index * kSh4NodeFloats + 8 * (size_t)sh4_slot_of(index, 0)];
    float *b = &nodes[(size_t)index * kSh4NodeFloats + 8 * (size_t)sh4_slot_of(index, 1)];
    uint32_t minima[3], maxima[3];
    for (int ax = 0; ax < 3; ++ax) {
        double lo = 0.0, hi = 0.0, wide_lo[4], wide_hi[4];
        for (int k = 0; k < n.children; ++k) {
            lo = k ? std::min(lo, (double)n.lo[k][ax]) : (double)n.lo[k][ax];
            hi = k ? std::max(hi, (double)n.hi[k][ax]) : (double)n.hi[k][ax];
        }
        const double extent = hi - lo;
        for (int k = 0; k < n.children; ++k) {
            wide_lo[k] = (double)n.lo[k][ax] - extent * 0.0001220703125 - std::fabs(n.lo[k][ax]) * 9.5367431640625e-07;
            wide_hi[k] = (double)n.hi[k][ax] + extent * 0.0001220703125 + std::fabs(n.hi[k][ax]) * 9.5367431640625e-07;
            lo = std::min(lo, wide_lo[k]);
            hi = std::max(hi, wide_hi[k]);
        }
        // scale = 32768 steps; base = origin + scale is at or below every bound, base + 255 steps above
        float scale = std::max((float)((hi - lo) / 255.0 * 32768.0), 1e-30f), origin = 0.0f;
        float grown = 1.0001f;  // the origin's rounding can cost a few steps; bounds are finite and below kSh4MaxBound
        for (bool fits = false; !fits; grown = 1.01f) {
            scale *= grown;
            origin = (float)(lo - (double)scale);
            while ((double)origin + (double)scale > lo) origin = std::nextafter(origin, -FLT_MAX);
            fits = (double)origin + (double)scale + 255.0 * ((double)scale / 32768.0) >= hi;
        }
        const double base = (double)origin + (double)scale, step = (double)scale / 32768.0, per_step = 1.0 / step;
        minima[ax] = maxima[ax] = 0;
        for (int k = 0; k < 4; ++k) {
            double q0 = 255.0, q1 = 0.0;  // an empty child
            if (k < n.children) {
                q0 = std::min(255.0, std::max(0.0, (double)(int)((wide_lo[k] - base) * per_step)));
                while (q0 > 0.0 && base + q0 * step > wide_lo[k]) q0 -= 1.0;
                q1 = std::min(255.0, std::max(0.0, (double)(int)((wide_hi[k] - base) * per_step)));
                while (q1 < 255.0 && base + q1 * step < wide_hi[k]) q1 += 1.0;
            }
            minima[ax] |= (uint32_t)q0 << (8 * k);
            maxima[ax] |= (uint32_t)q1 << (8 * k);
        }
        a[ax] = origin;
        a[3 + ax] = scale;
    }
    a[6] = bits_float((int)minima[0]), a[7] = bits_float((int)maxima[0]);
    b[0] = bits_float((int)minima[1]), b[1] = bits_float((int)maxima[1]);
    b[2] = bits_float((int)minima[2]), b[3] = bits_float((int)maxima[2]);
    for (int k = 0; k < 4; ++k) b[4 + k] = bits_float(k < n.children ? n.entry[k] : kSh4Empty);
}
Node4 load_node(const std::vector<float> &nodes, int index) {
    const float *a = &nodes[(size_t)index * kSh4NodeFloats + 8 * (size_t)sh4_slot_of(index, 0)];
    const float *b = &nodes[(size_t)index * kSh4NodeFloats + 8 * (size_t)sh4_slot_of(index, 1)];
    const float *rows[3] = {a + 6, b, b + 2};
    Node4 n;
    for (int k = 0; k < 4; ++k) {
        if (float_int(b[4 + k]) == kSh4Empty) continue;
        float lo[3], hi[3];
        for (int ax = 0; ax < 3; ++ax) {
            const int q0 = (float_int(rows[ax][0]) >> (8 * k)) & 255, q1 = (float_int(rows[ax][1]) >> (8 * k)) & 255;
            lo[ax] = std::nextafter((float)((double)a[ax] + (1.0 + q0 / 32768.0) * (double)a[3 + ax]), -FLT_MAX);
            hi[ax] = std::nextafter((float)((double)a[ax] + (1.0 + q1 / 32768.0) * (double)a[3 + ax]), FLT_MAX);
        }
        n.add(lo, hi, float_int(b[4 + k]));
    }
    return n;
}

// Collapses a binary tree into 4-wide records appended to `out`. leaf_code(node)
// gives a binary leaf's child entry, leaf_code.triangles(node) whether that is a leaf
// of triangles. Returns the depth of the emitted subtree.
struct Collapser {
    const std::vector<BNode> &bn;
    std::vector<float> &out;
    size_t limit;  // maximum nodes in `out` (the TLAS region), 0 = none
    bool overflow = false;
    template <class LeafCode>
    int emit(int b, LeafCode &&leaf_code, int &index) {
        int ch[4], nch = 0;
        if (bn[(size_t)b].left < 0) {
            ch[nch++] = b;  // a tree that is one leaf: a root with a single child
        } else {
            ch[nch++] = bn[(size_t)b].left;
            ch[nch++] = bn[(size_t)b].left + 1;
            while (nch < 4) {  // open the inner child with the largest surface area
                int pick = -1;
                float area = -1.0f;
                for (int k = 0; k < nch; ++k) {
                    const BNode &c = bn[(size_t)ch[k]];
                    if (c.left >= 0 && half_area(c.lo, c.hi) > area) {
                        area = half_area(c.lo, c.hi);
                        pick = k;
                    }
                }
                if (pick < 0) break;
                const int x = ch[pick];
                ch[pick] = bn[(size_t)x].left;
                ch[nch++] = bn[(size_t)x].left + 1;
            }
        }
        index = (int)(out.size() / kSh4NodeFloats);
        if (limit && (size_t)index >= limit) {
            overflow = true;
            return 0;
        }
        out.resize(out.size() + kSh4NodeFloats);
        Node4 node;
        // any-hit order: leaves of triangles first, then the smaller box
        float rank[4];
        for (int k = 0; k < nch; ++k) {
            const BNode &c = bn[(size_t)ch[k]];
            const float r = c.left < 0 && leaf_code.triangles(ch[k]) ? -1.0f : half_area(c.lo, c.hi);
            const int x = ch[k];
            int at = k;  // insertion sort
            for (; at > 0 && rank[at - 1] > r; --at) rank[at] = rank[at - 1], ch[at] = ch[at - 1];
            rank[at] = r, ch[at] = x;
        }
        int depth = 0;
        for (int k = 0; k < nch; ++k) {
            const BNode &c = bn[(size_t)ch[k]];
            int code;
            if (c.left < 0) {
                code = leaf_code(ch[k]);
            } else {
                int idx = 0;
                depth = std::max(depth, emit(ch[k], leaf_code, idx));
                code = idx;
            }
            node.add(c.lo, c.hi, code);
        }
        store_node(out, index, node);
        return depth + 1;
    }
};

}  // namespace

namespace {

bool identity_inverse(const float *m) {
    for (int k = 0; k < 16; ++k)
        if (m[k] != ((k % 5) == 0 ? 1.0f : 0.0f)) return false;
    return true;
}

struct BlasLeafCode {
    const std::vector<BNode> &bn;
    const std::vector<int> &order;
    const std::vector<float> &geo;
    int mesh;
    std::vector<float> &tris;
    bool triangles(int) const { return true; }
    // leaf triangles go to `tris` in leaf order as the collapse meets them
    int operator()(int b) {
        const BNode &lf = bn[(size_t)b];
        const int first = (int)(tris.size() / kTriGeoFloats);
        for (int q = 0; q < lf.count; ++q) {
            const int t = order[(size_t)(lf.first + q)];
            float rec[kTriGeoFloats];
            std::memcpy(rec, &geo[(size_t)t * kTriGeoFloats], sizeof(rec));
            rec[kSh4TriIndex] = bits_float(t);
            rec[kSh4TriMesh] = bits_float(mesh);
            rec[11] = 0.0f;
            tris.insert(tris.end(), rec, rec + kTriGeoFloats);
        }
        return ~((first << 2) | (lf.count - 1));
    }
};

struct TopLeafCode {
    const std::vector<BNode> &bn;
    const std::vector<int> &order;
    const std::vector<ShadowRef> &refs;
    int operator()(int b) const { return refs[(size_t)order[(size_t)bn[(size_t)b].first]].code; }
    bool triangles(int b) const { return (*this)(b) < 0; }
};

// The opened instances' refs replaced by the nodes inside them, the largest box first.
void open_instances(const std::vector<float> &nodes, const std::vector<int> &opened, std::vector<ShadowRef> &refs) {
    auto smaller = [&](int a, int c) {
        return half_area(refs[(size_t)a].lo, refs[(size_t)a].hi) < half_area(refs[(size_t)c].lo, refs[(size_t)c].hi);
    };
    std::vector<int> heap = opened;
    std::make_heap(heap.begin(), heap.end(), smaller);
    const size_t limit = refs.size() + (size_t)kSh4OpenedRefs;
    while (!heap.empty() && refs.size() + 3 <= limit) {
        std::pop_heap(heap.begin(), heap.end(), smaller);
        const int at = heap.back();
        heap.pop_back();
        const Node4 node = load_node(nodes, refs[(size_t)at].code);
        int pos = at;  // the first child takes the opened node's place
        for (int k = 0; k < node.children; ++k) {
            ShadowRef child;
            std::memcpy(child.lo, node.lo[k], sizeof(child.lo));
            std::memcpy(child.hi, node.hi[k], sizeof(child.hi));
            child.code = node.entry[k];
            if (pos < (int)refs.size())
                refs[(size_t)pos] = child;
            else
                refs.push_back(child);
            if (child.code >= 0) {
                heap.push_back(pos);
                std::push_heap(heap.begin(), heap.end(), smaller);
            }
            pos = (int)refs.size();
        }
    }
}

}  // namespace

bool rebuild_shadow_tlas(const float *inst_bounds, const float *inst_records, ShadowBvh &b) {
    const size_t n_inst = b.inst_root.size();
    std::fill(b.mesh_world.begin(), b.mesh_world.end(), -1);
    std::vector<ShadowRef> refs;
    auto make_ref = [](const float *lo, const float *hi, int code) {
        ShadowRef r;
        std::memcpy(r.lo, lo, sizeof(r.lo));
        std::memcpy(r.hi, hi, sizeof(r.hi));
        r.code = code;
        return r;
    };
    std::vector<int> opened;  // positions in refs of the opened instances
    for (size_t i = 0; i < n_inst; ++i) {
        if (b.inst_root[i] < 0) continue;
        if (!encodable(inst_bounds + 6 * i, inst_bounds + 6 * i + 3)) return false;
        int &world = b.mesh_world[(size_t)b.inst_mesh[i]];
        const bool open = world < 0 && identity_inverse(inst_records + 32 * i);
        refs.push_back(make_ref(inst_bounds + 6 * i, inst_bounds + 6 * i + 3,
                                open ? b.inst_root[i] : (kSh4InstBit | (int)i)));
        if (open) {
            world = (int)i;
            opened.push_back((int)refs.size() - 1);
        }
    }
    // An identity instance's nodes stand where they stood: moves that open the same instances again
    // take the leaves of the last time.
    const size_t n_base = refs.size();
    if (!b.opened.empty() && opened == b.opened) {
        for (size_t k = 0; k < opened.size(); ++k) refs[(size_t)opened[k]] = b.opened_refs[k];
        refs.insert(refs.end(), b.opened_refs.begin() + (ptrdiff_t)opened.size(), b.opened_refs.end());
    } else {
        open_instances(b.nodes, opened, refs);
        b.opened = opened;
        b.opened_refs.clear();
        for (int at : opened) b.opened_refs.push_back(refs[(size_t)at]);
        b.opened_refs.insert(b.opened_refs.end(), refs.begin() + (ptrdiff_t)n_base, refs.end());
    }
    std::vector<float> top;
    b.tlas_depth = 0;
    if (!refs.empty()) {
        std::vector<PrimBox> prims;
        prims.reserve(refs.size());
        for (const ShadowRef &r : refs) {
            PrimBox p;
            for (int k = 0; k < 3; ++k) {
                p.lo[k] = r.lo[k];
                p.hi[k] = r.hi[k];
                p.c[k] = 0.5f * (r.lo[k] + r.hi[k]);
            }
            prims.push_back(p);
        }
        std::vector<BNode> bn;
        std::vector<int> order;
        build_binary(prims, 1, bn, order);
        Collapser col{bn, top, (size_t)b.tlas_capacity};
        TopLeafCode code{bn, order, refs};
        int root = 0;
        b.tlas_depth = col.emit(0, code, root);
        if (col.overflow) return false;
    } else {  // nothing to hit: a root whose slots are all empty
        top.resize(kSh4NodeFloats);
        store_node(top, 0, Node4{});
        b.tlas_depth = 1;
    }
    std::memcpy(b.nodes.data(), top.data(), top.size() * sizeof(float));
    b.tlas_nodes = (int)(top.size() / kSh4NodeFloats);
    // a walk holds at most 3 entries per level it has descended, the end marker, one in hand, and one
    // that leads back to the world ray
    return 3 + 3 * (b.tlas_depth + b.blas_depth) <= kSh4Stack;
}

void shadow_ranks(const std::vector<int> &tlas_inst, int num_instances, std::vector<int> &rank) {
    rank.assign((size_t)std::max(0, num_instances), 0x7fffffff);
    for (size_t k = 0; k < tlas_inst.size(); ++k) {
        const int i = tlas_inst[k];
        if (i >= 0 && i < num_instances && rank[(size_t)i] == 0x7fffffff) rank[(size_t)i] = (int)k;
    }
}

bool build_shadow_bvh(const hdr_scene_desc &desc, const FlatScene &flat, ShadowBvh &out, std::string &err) {
    out = ShadowBvh{};
    const int n_inst = desc.num_instances;
    // room for the top-level tree of any transforms: every instance, and the opened nodes (no more
    // than the meshes have triangles)
    size_t triangles = 0;
    for (int mi = 0; mi < desc.num_meshes; ++mi) triangles += (size_t)std::max(0, desc.meshes[mi].num_triangles);
    out.tlas_capacity = std::max(1, n_inst) + (int)std::min<size_t>(triangles, (size_t)kSh4OpenedRefs);
    out.nodes.assign((size_t)out.tlas_capacity * kSh4NodeFloats, 0.0f);
    out.tris.assign(kTriGeoFloats, 0.0f);  // record 0: the triangle without area of kSh4Empty
    std::vector<int> mesh_root((size_t)std::max(0, desc.num_meshes), -1);
    const bool host_geo = !flat.tri_geo.empty() || flat.num_triangles == 0;
    for (int mi = 0; mi < desc.num_meshes; ++mi) {
        // the mesh's triangle records in the reference's BLAS order
        std::vector<float> geo;
        if (host_geo) {
            const size_t b = (size_t)flat.mesh_tri_base[(size_t)mi], n = (size_t)flat.mesh_tri_count[(size_t)mi];
            geo.assign(flat.tri_geo.begin() + (long)(b * kTriGeoFloats),
                       flat.tri_geo.begin() + (long)((b + n) * kTriGeoFloats));
        } else {  // the BLAS was built on the device: the host build gives the same order
            const Blas blas = build_blas(desc.meshes[mi]);
            geo.resize(blas.tris.size() * kTriGeoFloats);
            float a[kTriAttrFloats];
            for (size_t t = 0; t < blas.tris.size(); ++t) pack_triangle(blas.tris[t], &geo[t * kTriGeoFloats], a);
        }
        const size_t nt = geo.size() / kTriGeoFloats;
        if (nt == 0) continue;
        std::vector<PrimBox> prims(nt);
        for (size_t t = 0; t < nt; ++t) {
            const float *g = &geo[t * kTriGeoFloats];
            const float v[3][3] = {{g[0], g[1], g[2]},
                                   {g[0] + g[3], g[1] + g[4], g[2] + g[5]},
                                   {g[0] + g[6], g[1] + g[7], g[2] + g[8]}};
            PrimBox &p = prims[t];
            for (int k = 0; k < 3; ++k) p.lo[k] = FLT_MAX, p.hi[k] = -FLT_MAX;
            // vertices v0 + e1 / v0 + e2 may round: widen the box by a relative ulp margin
            for (const auto &x : v) grow(p.lo, p.hi, x, x);
            for (int k = 0; k < 3; ++k) {
                const float m = (std::fabs(p.lo[k]) + std::fabs(p.hi[k])) * 2.4e-7f + 1e-30f;
                p.lo[k] -= m;
                p.hi[k] += m;
                p.c[k] = 0.5f * (p.lo[k] + p.hi[k]);
            }
            if (!encodable(p.lo, p.hi)) return true;
        }
        std::vector<BNode> bn;
        std::vector<int> order;
        build_binary(prims, kSh4LeafTris, bn, order);
        Collapser col{bn, out.nodes, 0};
        int root = 0;
        const size_t tri_base = out.tris.size() / kTriGeoFloats;
        if (tri_base + nt >= ((size_t)1 << 27)) {  // leaf entries: (first << 2) | ... fits 29 bits
            err = "too many triangles for the shadow BVH encoding";
            return false;
        }
        if (col.out.size() / kSh4NodeFloats + nt >= (size_t)kSh4InstBit) {
            err = "too many triangles for the shadow BVH encoding";
            return false;
        }
        BlasLeafCode code{bn, order, geo, mi, out.tris};
        const int depth = col.emit(0, code, root);
        mesh_root[(size_t)mi] = root;
        out.blas_depth = std::max(out.blas_depth, depth);
    }
    out.inst_root.assign((size_t)std::max(0, n_inst), -1);
    out.inst_mesh.assign((size_t)std::max(0, n_inst), 0);
    out.mesh_world.assign((size_t)std::max(1, desc.num_meshes), -1);
    for (int i = 0; i < n_inst; ++i) {
        const int mesh = desc.instances[i].mesh;
        if (mesh < 0 || mesh >= desc.num_meshes) continue;
        out.inst_mesh[(size_t)i] = mesh;
        out.inst_root[(size_t)i] = mesh_root[(size_t)mesh];
    }
    shadow_ranks(flat.tlas_inst, n_inst, out.inst_rank);
    // not an error when it does not fit: the reference trees serve these queries too
    out.ok = rebuild_shadow_tlas(flat.inst_bounds.data(), flat.instances.data(), out);
    return true;
}

}  // namespace hdr
