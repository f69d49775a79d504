// The four-wide form of the compact SBVH that the device traverses (tt_wide.cuh), made from the
// reference's two-wide arrays at upload (tt_wide_build.cu).
//
// Node: 224 bytes, seven 32-byte sectors. Four slots in two groups, (0, 1) for the left child of a
// two-wide inner node A and (2, 3) for its right child. A group holds either A's child itself in
// its first slot, the second being empty (a "direct" group), or that child's two children. A
// child is replaced by its children only when its box is exactly the union of theirs, so its box
// planes and with them its entry distance follow from the slots'.
//   float xy[4][4][2]   xy[c][s]: an x and a y plane of slot s; bit 0 of c picks hi_x over lo_x,
//                       bit 1 hi_y over lo_y
//   float z[2][2][4]    z[0]: lo_z, hi_z; z[1]: hi_z, lo_z
//   uint32_t ref[4]     what each slot holds
//   uint32_t spare[4]
// The planes are there several times so that a ray finds those it enters and those it leaves by
// address, by the signs of its direction, in three 32-byte loads and without a select: the
// traversal is bound by load sectors and by the arithmetic unit that does minima and selects.
// An empty slot has lo = +inf, hi = -inf (no ray passes it) and the reference kWideEmpty.
//
// Triangle pair: 96 bytes, two triangles of a leaf side by side for the packed two-lane float
// instructions; -v0 and the edges e1 = v1 - v0, e2 = v2 - v0 as the leaf test forms them:
//   float nv0x[2], nv0y[2], nv0z[2], e1x[2], e1y[2], e1z[2], e2x[2], e2y[2], e2z[2]
//   int32_t slot      float4 slot of the first triangle in the compact vertex array (second: + 3)
//   uint32_t flags    kPairLast: the leaf ends here
//   uint32_t spare[4]
// A leaf of an odd number of triangles ends in a pair whose second triangle is all zeros (its
// determinant is 0, so it is never accepted).
#pragma once

#include <cstdint>

namespace tt {

constexpr uint32_t kWideLeaf = 0x80000000u;   // the reference is a leaf's first pair, else a node
constexpr uint32_t kWideMark = 0x40000000u;   // stack entries only (tt_wide.cuh)
constexpr uint32_t kWideIndex = 0x3fffffffu;  // node or pair index
constexpr uint32_t kWideEmpty = 0x7fffffffu;  // an empty slot
constexpr uint32_t kPairLast = 1u;
constexpr int kWideNodeBytes = 224;
constexpr int kWidePairBytes = 96;
constexpr int kWideStack = 72;  // stack entries a traversal may need (deeper trees stay two-wide)
// BvhView::wide_flags
constexpr uint32_t kWideNegZero = 1u;  // some box plane is -0.0

// Bounds under which every float of a box or triangle test stays finite and no slab value of a
// plane other than zero underflows (tt_wide.cuh, wide_regular).
constexpr float kWideCoordMax = 68719476736.0f;   // 2^36: |vertex|, |box plane|, |ray origin|
constexpr float kWideDirMax = 1073741824.0f;      // 2^30: |ray direction component|
constexpr float kWidePlaneMin = 7.703719777548943e-34f;  // 2^-110: |box plane| unless zero

}  // namespace tt
