// 4-wide SAH trees (no reference counterpart): a second acceleration structure over the same
// triangles and instances, for the query "is there a hit nearer than the light" (the visibility
// test of _evaluateLightSample, ris_direct_light_integrator.cpp:628-658, and of the MIS
// integrator's NEE, mis_direct_light_integrator.cpp:140-151) and for closest hits.
//
// The answer of the first query does not depend on the tree: the reference walks its
// midpoint-split trees and compares the closest hit with the light distance,
// and a hit exists below the limit exactly when some triangle test (the same
// IntersectTriangle arithmetic in the same instance space) returns one. So this
// structure is built for speed: binned-SAH binary trees collapsed to 4 children
// per node, each node holding its children's boxes (tested together, before
// descending), triangles in leaf order.
//
// The same trees answer closest-hit queries with the reference's result: every
// triangle record carries its index in the reference's BLAS triangle order, and
// every instance its position in the reference TLAS's leaf order; among hits at
// equal distance the walk keeps the smallest (instance position, triangle
// index), which is the one the reference's left-first walks find first
// (bvh.cpp:262-304, scene.cpp:414-510, strict `<` on t). Whether the reference's own
// rounded box tests let it reach that hit is checked afterwards (ref_reaches, device/traverse.cuh).
//
// Records and entries: device/sh4_layout.h. Children stand in the order an any-hit walk tries
// them: triangles first, then the smaller box first (a small box is cheap to finish
// and, when the ray hits it, likely to hold a hit; on the 1.03M-triangle terrain scene
// the ray's own near-to-far order takes 22.9 node steps per shadow ray, this order 17.9).
// Nodes: the top-level tree first (its root is node 0; room for a rebuild over the
// same instances), then every mesh's BLAS. Triangles: 12 floats each, the tri_geo
// record (v0, e1 = v1 - v0, e2 = v2 - v0) the reference-order walk tests, with the
// triangle's index in its mesh's reference BLAS order and its mesh.
//
// Opened instances. The object-space ray of an instance whose inverse transform is the
// identity is the world ray, so its BLAS nodes need no ray of their own. For the first
// such instance of every mesh (mesh_world) the top-level tree is built over the nodes
// inside it instead of over its one box: the largest node is replaced by its children
// until kSh4OpenedRefs have been added. A terrain that covers the scene then no longer
// overlaps every other instance's leaf, and a walk enters it without an instance entry
// (17.9 -> 16.8 steps, 1.70 -> 1.11 instance entries per shadow ray of that scene;
// closest hits of bounce rays 20.0 -> 15.5 steps). Other instances of the same mesh,
// and instances that are not the identity, are entered through their leaf.
#pragma once

#include <string>
#include <vector>

#include "../../../include/hdrestir.h"
#include "../device/sh4_layout.h"

namespace hdr {

struct FlatScene;

// A leaf of the top-level tree: an instance, or a node or triangle leaf inside an opened one.
struct ShadowRef {
    float lo[3], hi[3];
    int code;
};

struct ShadowBvh {
    std::vector<float> nodes;
    std::vector<float> tris;
    std::vector<int> inst_root;   // per instance: its mesh's BLAS root node, or -1 (no triangles)
    std::vector<int> inst_mesh;   // per instance: its mesh
    std::vector<int> inst_rank;   // per instance: its position in the reference TLAS's leaf order
    std::vector<int> mesh_world;  // per mesh: the instance whose nodes are opened, -1 = none
    std::vector<int> opened;      // the opened instances, by their place among those with triangles
    std::vector<ShadowRef> opened_refs;  // the leaves in their places, then the other ones inside them
    int tlas_capacity = 0;        // nodes reserved for the top-level tree at the front of `nodes`
    int tlas_nodes = 0;           // and those it takes
    int tlas_depth = 0, blas_depth = 0;
    bool ok = false;              // false: not built (the scene is walked with the reference trees)
};

// Builds the BLAS of every mesh over its triangles in the reference's BLAS order
// (the flat scene's tri_geo records when the host built them, else a host
// build of the reference's tree for the order) and the top-level tree over the
// instances (instances whose mesh has no triangles are left out). Returns
// false only on error; out.ok stays false when the trees would need more than
// kSh4Stack stack entries.
bool build_shadow_bvh(const hdr_scene_desc &desc, const FlatScene &flat, ShadowBvh &out, std::string &err);

// inst_rank from the reference TLAS's instance order (tlas_inst: instance per leaf slot).
void shadow_ranks(const std::vector<int> &tlas_inst, int num_instances, std::vector<int> &rank);

// Rebuilds the top-level tree over instances that moved: `inst_bounds` (6 floats each, the
// world boxes) and `inst_records` (32 floats each, the inverse transform first). Reads the
// BLAS nodes, inst_root and inst_mesh of `b`, and writes its mesh_world, opened, opened_refs, the
// first nodes of b.nodes and b.tlas_depth; returns false when the tree does not fit the reserved room or the
// stack bound.
bool rebuild_shadow_tlas(const float *inst_bounds, const float *inst_records, ShadowBvh &b);

}  // namespace hdr
