// Layout constants of the shadow-ray BVH shared by the host builder
// (host/shadow_bvh.cpp) and the device walk (device/shadow4.cuh).
#pragma once

namespace hdr {

// Node record, 64 bytes: two slots of 32 bytes, each one 256-bit load
//   A: origin x, y, z | scale x, y, z | minima x, maxima x (a byte per child)
//   B: minima y, maxima y, minima z, maxima z | the four child entries (int bits)
// A bound is origin + (1 + byte / 32768) * scale, the form in which the walk reads it: a
// byte put into a float's mantissa. Bounds are rounded outward, an empty child has minima
// 255 and maxima 0. The walk is bound by L1's data stage, which takes a pass for nearly
// every line a divergent load touches: with 112 bytes of float bounds in seven 128-bit
// loads it was 93 % busy.
// Slot A of node i is the first half unless bit 1 of i is set: lanes at different nodes
// read the same slot in one load, and then meet in all of L1's banks instead of in half.
constexpr int kSh4NodeFloats = 16;
constexpr int sh4_slot_of(int node, int slot) { return slot ^ ((node >> 1) & 1); }
// Entry of an empty child: a leaf of triangle record 0, which has no area.
constexpr int kSh4Empty = -1;
// Stack entries of the device walk.
constexpr int kSh4Stack = 96;
// Child entries, which are also the walk's stack entries:
//   0 .. kSh4InstBit - 1 : inner node index
//   < 0                  : triangles of a leaf, ~((first << 2) | (count - 1)), count 1..4
//   kSh4InstBit | i      : instance i, entered with its own ray
constexpr int kSh4InstBit = 0x40000000;
// Triangle record floats beyond the 9 of the test (int bits): the triangle's index in its
// mesh's reference BLAS order, and its mesh.
constexpr int kSh4TriIndex = 9, kSh4TriMesh = 10;
// Instances with the identity transform are opened: up to this many of their nodes become
// leaves of the top-level tree (walked with the world ray), largest first.
constexpr int kSh4OpenedRefs = 1024;

}  // namespace hdr
