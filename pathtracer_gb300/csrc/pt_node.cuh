// pt_node.cuh -- the BVH4's nodes: as the builders make them (float boxes) and
// as the traversal reads them (packed to 64 bytes).
#pragma once
#include "pt_common.cuh"

namespace pt {

// A node as the builders make it.
struct alignas(128) Bvh4Node {
  float lo_x[4], hi_x[4];
  float lo_y[4], hi_y[4];
  float lo_z[4], hi_z[4];
  int32_t child[4];  // internal: node index; leaf: first item index
  int32_t count[4];  // internal: 0; leaf: number of items; empty slot: -1
};
static_assert(sizeof(Bvh4Node) == 128, "BVH4 node must be one 128-byte line");

// The node the traversal reads, 64 B: the children's boxes as bytes on a grid
// of 256 planes per axis over the node's box, and the children's traversal
// references.  Plane q of an axis lies at origin + (1 + q * 2^-15) * scale
// (the bracket is a float whose middle byte is q, so it takes one byte
// permute and no conversion).  pack_node rounds the boxes outwards, by 2^-20 of
// the node's coordinates and 1/8 of a grid step at least, which covers the
// roundings of this form and of the ray's: a ray that meets a child's box meets
// its packed box, for origins of up to 3 times the node's coordinates or 1000
// times its extent (each per axis).  From farther away the rounding of origin /
// direction, 2^-24 of the origin, moves the box by more, as it moves a float box.
//
// Two 32-byte loads fetch it.  With float boxes a lane's visit took seven
// 16-byte loads of a 128-byte node, one L1 wavefront per lane and load: in the
// rough-glass scene (0.26 M nodes) the L1 data pipe was 93-96 % busy and the
// issue slots 52-65 %; packed it is 63-69 % and 72-80 %.  Rough glass, 16.8 M
// paths, with the paired fma of visit_node: trace 13.8 -> 10.5 ms, shadow 13.3 ->
// 9.1; material divergence shadow 31.7 -> 24.6 ms.  The float boxes with 32-byte
// loads and the paired fma: 12.9, 12.4 and 29.9 ms, and 6.38 ms against 6.41
// for the Cornell box's shadow rays (boxes of a few steps' thickness are
// entered more often when packed), so the packed form serves every scene.
struct alignas(64) PackedNode {
  float origin[3];
  float scale[3];        // 2^15 grid steps
  uint32_t lo_x, hi_x;   // byte c: child c
  uint32_t lo_y, hi_y, lo_z, hi_z;
  int32_t ref[4];
};
static_assert(sizeof(PackedNode) == 64, "packed node must be half a line");

// Traversal references (a node's children on the device, the stack): a node
// index (>= 0; PT_INST_BIT: entering a moving object), a leaf
// ~(first_item << 3 | count - 1) (count <= 8), PT_FRAME_END (stack only) or
// PT_REF_EMPTY (an empty child slot; as the next reference: nothing pending).
#define PT_REF_EMPTY ((int32_t)0x80000001)
PT_HD int32_t leaf_ref(int32_t first, int32_t count) { return ~((first << 3) | (count - 1)); }
// A child's reference from its (child, count) pair.
PT_HD int32_t trav_ref(int32_t child, int32_t count) {
  return count < 0 ? PT_REF_EMPTY : count == 0 ? child : leaf_ref(child, count);
}

// One axis of a node: `lo`, `hi` of the children (n of them), the grid and the
// children's bytes.  With u = 2^-24, coordinates up to R, a ray origin o and the
// grid's extent 2^15 steps: rounding the origin, o * inv, the fma that joins them
// and the planes' fma moves a plane by at most u (4 R + 4 |o|), which the slack of
// 16 u R covers for |o| <= 3 R, and by 2^-16 of the node's extent, which is far
// below 1/8 of a step (1/2016 of the extent); so is 4 u |o| up to 1000 extents.
// (A slack of the scene's coordinates would cover every origin in it, but a scene
// may have a far light or a wide ground under small objects, whose boxes it
// would swamp.)
PT_HD void pack_axis(const float *lo, const float *hi, int n, float &origin, float &scale, uint32_t &qlo,
                     uint32_t &qhi) {
  double a = lo[0], b = hi[0];
  bool number = true;
  for (int c = 0; c < n; ++c) number = number && lo[c] <= hi[c];
  for (int c = 1; c < n; ++c) {
    if (lo[c] < a) a = lo[c];
    if (hi[c] > b) b = hi[c];
  }
  const double slack = (fabs(a) > fabs(b) ? fabs(a) : fabs(b)) * 0x1p-20;
  a -= slack;
  b += slack;
  double step = (b - a) / 252.0;
  if (step < 1e-30) step = 1e-30;
  scale = (float)(step * 32768.0);
  step = (double)scale / 32768.0;
  const double zero = a - step;  // plane 0
  origin = (float)(zero - (double)scale);
  qlo = 0xffffffffu;  // empty slots: inverted
  qhi = 0;
  for (int c = 0; c < n; ++c) {
    const double l = floor((lo[c] - slack - zero) / step - 0.125), h = ceil((hi[c] + slack - zero) / step + 0.125);
    const uint32_t ql = l >= 0.0 ? (uint32_t)l : 0u, qh = h <= 255.0 ? (uint32_t)h : 255u;
    qlo = (qlo & ~(255u << (8 * c))) | (ql << (8 * c));
    qhi |= qh << (8 * c);
  }
  // a bound that is not a number: planes that are none either, which the slab
  // test's min / max drop, as they drop such a float bound
  if (!number) origin = scale = NAN;
}
PT_HD PackedNode pack_node(const Bvh4Node &N) {
  PackedNode P;
  int n = 0;  // the children are the first slots
  for (int c = 0; c < 4; ++c) {
    P.ref[c] = trav_ref(N.child[c], N.count[c]);
    if (N.count[c] >= 0) n = c + 1;
  }
  if (n == 0) {
    for (int k = 0; k < 3; ++k) P.origin[k] = P.scale[k] = 0.f;
    P.lo_x = P.lo_y = P.lo_z = 0xffffffffu;
    P.hi_x = P.hi_y = P.hi_z = 0;
    return P;
  }
  pack_axis(N.lo_x, N.hi_x, n, P.origin[0], P.scale[0], P.lo_x, P.hi_x);
  pack_axis(N.lo_y, N.hi_y, n, P.origin[1], P.scale[1], P.lo_y, P.hi_y);
  pack_axis(N.lo_z, N.hi_z, n, P.origin[2], P.scale[2], P.lo_z, P.hi_z);
  return P;
}

}  // namespace pt
