// pt_trace.cuh -- closest-hit and any-hit traversal of the BVH4.
//
// The BVH4 is collapsed from the reference's own binary trees (top level
// BVHNode, bvh.hpp:46-102; per mesh MeshBVHNode, meshBVH.cpp:6-55), so the
// leaves hold exactly the reference's leaf primitive sets.  Closest-hit
// traversal is near-to-far; the first PT_STACK_SHARED entries of a thread's stack
// are in shared memory (column per thread, bank-conflict free), the others in
// local memory.  Primitive tests restate the reference arithmetic with rounded,
// never-fused operations so that hit distances match the reference bit for bit:
//   triangle  MeshBVHNode::hitTriangle  meshBVH.cpp:85-143
//   rectangle AARectangle<axis>::intersect  primitive.cpp:31-122
//   sphere    Sphere::intersect  primitive.hpp:124-170
// Acceptance is inclusive (t == tmax accepted), so of two equal-t primitives
// the later one tested wins, as in the reference leaf loop.
#pragma once
#include "pt_scene.cuh"

namespace pt {


struct HitRec {
  float t;
  int32_t prim;
  float u, v;
};

// A hit of t = NaN: 0 / 0 of a ray in a rectangle's plane or along a straight
// curve's axis.  It passes every comparison, so the reference's leaf loop takes
// it where the ray meets the primitive's bounds, and after it any other hit: it
// has no place in an order by t.  A closest-hit ray of trace_rays that meets one
// is marked and walked again, leaf by leaf, in the leaf loop's own order.  Tests
// that take such a hit (EXACT) ask whether the ray meets the primitive's own
// bounds, since the packed boxes, rounded outwards, let more rays through.
enum RayState : uint8_t { RAY_ORDERED = 0, RAY_MARKED = 1, RAY_ALONE = 2 };

// One axis of that test; near and far: what is left of the ray.
__device__ __forceinline__ bool bounds_axis(float o, float d, float lo, float hi, float &near, float &far) {
  if (d == 0.f) return !(o < lo || o > hi);
  const float a = (lo - o) / d, b = (hi - o) / d;
  near = fmaxf(near, fminf(a, b));
  far = fminf(far, fmaxf(a, b));
  return !(near > far);
}
// Its far end: a hit of the same leaf on the bounds may be tmax.
__device__ __forceinline__ float bounds_far(float tmax) { return fmaf(fabsf(tmax), 0x1p-16f, tmax); }

// Moller-Trumbore exactly as hitTriangle orders it.
__device__ __forceinline__ bool hit_triangle(const Item &it, V3 o, V3 d, float tmin, float tmax,
                                             float &t_out, float &u_out, float &v_out) {
  V3 p0 = v3(it.a[0], it.a[1], it.a[2]);
  V3 e1 = v3(it.b[0], it.b[1], it.b[2]);
  V3 e2 = v3(it.c[0], it.c[1], it.c[2]);
  V3 P = xcross(d, e2);
  float det = xdot(e1, P);
  if (fabsf(det) < 1e-8f) return false;
  float inv = xdiv(1.0f, det);
  V3 T = xsubv(o, p0);
  float u = xmul(xdot(T, P), inv);
  if (u < 0.f || u > 1.f) return false;
  V3 Q = xcross(T, e1);
  float v = xmul(xdot(d, Q), inv);
  if (v < 0.f || xadd(u, v) > 1.f) return false;
  float t = xmul(xdot(e2, Q), inv);
  if (t < tmin || t > tmax) return false;
  t_out = t;
  u_out = u;
  v_out = v;
  return true;
}

// AARectangle<axis>::intersect with the normalised direction dn.
template <bool EXACT>
__device__ __forceinline__ bool hit_quad(const Item &it, V3 o, V3 dn, float tmin, float tmax, float &t_out,
                                         uint8_t *state) {
  const int axis = (int)it.b[2];
  const float k = it.a[0], d0min = it.a[1], d0max = it.a[2];
  const float d1min = it.b[0], d1max = it.b[1];
  float oa, da, o0, d0_, o1, d1_;
  if (axis == 0) {
    oa = o.x; da = dn.x; o0 = o.y; d0_ = dn.y; o1 = o.z; d1_ = dn.z;
  } else if (axis == 1) {
    oa = o.y; da = dn.y; o0 = o.x; d0_ = dn.x; o1 = o.z; d1_ = dn.z;
  } else {
    oa = o.z; da = dn.z; o0 = o.x; d0_ = dn.x; o1 = o.y; d1_ = dn.y;
  }
  float t = xdiv(xsub(k, oa), da);
  if (EXACT) {
    if (t < tmin || t > tmax) return false;
    if (t != t && da == 0.f) {
      float near = tmin, far = bounds_far(tmax);
      if (!bounds_axis(o0, d0_, d0min, d0max, near, far) || !bounds_axis(o1, d1_, d1min, d1max, near, far)) return false;
    }
  } else if (!(t >= tmin && t <= tmax)) {
    if (t != t) *state = RAY_MARKED;
    return false;
  }
  float a0 = xadd(o0, xmul(t, d0_));
  float a1 = xadd(o1, xmul(t, d1_));
  if (a0 < d0min || a0 > d0max || a1 < d1min || a1 > d1max) return false;
  t_out = t;
  return true;
}

// Sphere::intersect with the normalised direction dn.
__device__ __forceinline__ bool hit_sphere(const Item &it, V3 o, V3 dn, float tmin, float tmax,
                                           float &t_out) {
  V3 c = v3(it.a[0], it.a[1], it.a[2]);
  const float r = it.b[0];
  V3 oc = xsubv(o, c);
  float a = xdot(dn, dn);
  float b = xmul(2.f, xdot(dn, oc));
  float cc = xsub(xdot(oc, oc), xmul(r, r));
  float disc = xsub(xmul(b, b), xmul(xmul(4.f, a), cc));
  if (disc < 0.f) return false;
  float delta = xsqrt(disc);
  float t = xdiv(xsub(-b, delta), xmul(2.f, a));
  if (t < tmin || t > tmax) {
    t = xdiv(xadd(-b, delta), xmul(2.f, a));
    if (t < tmin || t > tmax) return false;
  }
  t_out = t;
  return true;
}

// 32 bytes with one load.
__device__ __forceinline__ void ld32b(const void *p, uint32_t *v) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "l"(p));
}

// Cubic Bezier point, every operation separately rounded (never fused) in
// bezier.hpp:10-18's order, so that curve hits round like the reference's.
__device__ __forceinline__ V3 bezier_point(const float4 *cp, float u) {
  const float u1 = xsub(1.0f, u);
  const float b0 = xmul(xmul(u1, u1), u1), b1 = xmul(xmul(xmul(3.0f, u), u1), u1);
  const float b2 = xmul(xmul(xmul(3.0f, u), u), u1), b3 = xmul(xmul(u, u), u);
  const float4 c0 = __ldg(cp), c1 = __ldg(cp + 1), c2 = __ldg(cp + 2), c3 = __ldg(cp + 3);
  auto comb = [&](float a0, float a1, float a2, float a3) {
    return xadd(xadd(xadd(xmul(a0, b0), xmul(a1, b1)), xmul(a2, b2)), xmul(a3, b3));
  };
  return v3(comb(c0.x, c1.x, c2.x, c3.x), comb(c0.y, c1.y, c2.y, c3.y), comb(c0.z, c1.z, c2.z, c3.z));
}
// Its derivative (bezier.hpp:20-36).
__device__ __forceinline__ V3 bezier_tangent(const float4 *cp, float u) {
  const float4 c0 = __ldg(cp), c1 = __ldg(cp + 1), c2 = __ldg(cp + 2), c3 = __ldg(cp + 3);
  const V3 d0 = 3.0f * (v3(c1.x, c1.y, c1.z) - v3(c0.x, c0.y, c0.z));
  const V3 d1 = 3.0f * (v3(c2.x, c2.y, c2.z) - v3(c1.x, c1.y, c1.z));
  const V3 d2 = 3.0f * (v3(c3.x, c3.y, c3.z) - v3(c2.x, c2.y, c2.z));
  const float u1 = 1.0f - u;
  return d0 * (u1 * u1) + d1 * (2.0f * u * u1) + d2 * (u * u);
}

// Segment i of a curve, an infinite cylinder cut at its ends
// (primitives/curve.hpp:48-103): start point and radius (the mean of the
// linearly interpolated width at the ends), axis and length.
struct CurveSegment {
  V3 pa;
  float radius;
  V3 axis;
  float len;
};
__device__ __forceinline__ CurveSegment curve_segment(const float4 *cp, int i) {
  const int N = PT_CURVE_SEGMENTS;
  const float u0 = float(i) / N, u1 = float(i + 1) / N;
  const V3 pa = bezier_point(cp, u0), pb = bezier_point(cp, u1);
  const float w0 = __ldg(cp).w, w1 = __ldg(cp + 1).w;
  const float r0 = xadd(w0, xmul(xsub(w1, w0), u0)), r1 = xadd(w0, xmul(xsub(w1, w0), u1));
  const V3 ab = xsubv(pb, pa);
  CurveSegment g;
  g.pa = pa;
  g.radius = xmul(0.5f, xadd(r0, r1));
  g.len = xsqrt(xdot(ab, ab));
  g.axis = v3(xdiv(ab.x, g.len), xdiv(ab.y, g.len), xdiv(ab.z, g.len));
  return g;
}

// Whether a ray meets a curve's bounds (Curve::getAABB, primitives/curve.hpp:
// 33-46).  A function of its own: inlined, it takes registers of the curve
// kernels (hair trace 3.65 -> 3.71 ms).
static __device__ __noinline__ bool meets_curve(const float4 *cp, V3 o, V3 d, float tmin, float tmax) {
  const float4 a = __ldg(cp), b = __ldg(cp + 1), c = __ldg(cp + 2), e = __ldg(cp + 3);
  const float r = fmaxf(a.w, b.w);
  float near = tmin, far = bounds_far(tmax);
  auto axis = [&](float oo, float dd, float p, float q, float s, float t) {
    return bounds_axis(oo, dd, fminf(fminf(p, q), fminf(s, t)) - r, fmaxf(fmaxf(p, q), fmaxf(s, t)) + r, near, far);
  };
  return axis(o.x, d.x, a.x, b.x, c.x, e.x) && axis(o.y, d.y, a.y, b.y, c.y, e.y) && axis(o.z, d.z, a.z, b.z, c.z, e.z);
}

// Curve::intersect (primitives/curve.hpp:48-129) over the curve's segments
// (8 x 32 B); roots from gl::solveQuadratic (utility.hpp:112-124).  Returns
// the segment in u and the position along it in v (fraction of its length).
// The segments are tabulated at upload by curve_segment: computing them in the
// test took two thirds of it (two Bezier points, a root and three divisions
// per segment and ray); hair on curves, 0.96 M paths: trace 5.9 -> 4.4 ms.
__device__ __forceinline__ bool hit_curve(const float4 *seg, V3 o, V3 d, float tmin, float tmax, float &t_out,
                                          float &u_out, float &v_out) {
  float best = tmax;
  bool found = false;
  // Exact (never fused) arithmetic throughout: the cylinder quadratic is
  // ill-conditioned for grazing rays (C is a difference of near-equal
  // squares), so contracted multiply-adds would move t by ~1e-5 relative.
  auto axpy = [](V3 a, float k, V3 b) {  // a - k b
    return v3(xsub(a.x, xmul(k, b.x)), xsub(a.y, xmul(k, b.y)), xsub(a.z, xmul(k, b.z)));
  };
#pragma unroll 1
  for (int i = 0; i < PT_CURVE_SEGMENTS; ++i) {
    uint32_t w[8];
    ld32b(seg + 2 * i, w);
    const V3 pa = v3(u2f(w[0]), u2f(w[1]), u2f(w[2])), axis = v3(u2f(w[4]), u2f(w[5]), u2f(w[6]));
    const float radius = u2f(w[3]), seg_len = u2f(w[7]);
    const V3 d_perp = axpy(d, xdot(d, axis), axis);
    const V3 delta = xsubv(o, pa);
    const V3 o_perp = axpy(delta, xdot(delta, axis), axis);
    const float A = xdot(d_perp, d_perp), B = xmul(2.0f, xdot(d_perp, o_perp));
    const float C = xsub(xdot(o_perp, o_perp), xmul(radius, radius));
    const float disc = xsub(xmul(B, B), xmul(xmul(4.0f, A), C));
    if (disc >= 0.f) {
      const float sq = xsqrt(disc);
      const float q = B < 0 ? xmul(-0.5f, xsub(B, sq)) : xmul(-0.5f, xadd(B, sq));
      float ra = xdiv(q, A), rb = xdiv(C, q);
      if (ra > rb) {
        const float tt = ra;
        ra = rb;
        rb = tt;
      }
      const int nr = ra == rb ? 1 : 2;
      for (int r = 0; r < nr; ++r) {
        const float t = r == 0 ? ra : rb;
        if (t < tmin || t > best) continue;
        const V3 hp = v3(xadd(o.x, xmul(t, d.x)), xadd(o.y, xmul(t, d.y)), xadd(o.z, xmul(t, d.z)));
        const float proj = xdot(xsubv(hp, pa), axis);
        if (proj < 0.0f || proj > seg_len) continue;
        best = t;
        u_out = (float)i;
        v_out = xdiv(proj, seg_len);
        found = true;
      }
    }
  }
  if (found) t_out = best;
  return found;
}

__device__ __forceinline__ Item load_item(const Item *items, int i) {
  const float4 *p = reinterpret_cast<const float4 *>(items + i);
  float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  Item it;
  it.a[0] = a.x; it.a[1] = a.y; it.a[2] = a.z; it.a[3] = a.w;
  it.b[0] = b.x; it.b[1] = b.y; it.b[2] = b.z; it.b[3] = b.w;
  it.c[0] = c.x; it.c[1] = c.y; it.c[2] = c.z; it.c[3] = c.w;
  return it;
}

// Origin of a ray of time `time` in the frame of a primitive moving with
// velocity v: o - v * time (rounded, never fused).
__device__ __forceinline__ V3 moved_origin(const SceneView &S, uint32_t motion, V3 o, float time) {
  const float4 v = __ldg(S.motion + (motion - 1u));
  return v3(xsub(o.x, xmul(v.x, time)), xsub(o.y, xmul(v.y, time)), xsub(o.z, xmul(v.z, time)));
}

// Tests leaf item `idx` against a ray (origin o in its current frame); a
// hit in [tmin, tmax] fills `hit`.  dn points at the ray's normalised
// direction (rectangles and spheres read it).  CURVES = false compiles the
// curve test out (curve items then never hit), MOTION = false the moving
// primitives.  A hit without an order is tested against the primitive's bounds
// (EXACT, as are all tests of CURVES), or left out and the ray marked.
template <bool CURVES, bool MOTION, bool EXACT>
__device__ __forceinline__ bool test_item(const SceneView &S, int idx, V3 o_w, V3 d, const float4 *dn4, float tmin,
                                          float tmax, HitRec &hit, float time, uint8_t *state) {
  Item it = load_item(S.items, idx);
  const int type = (int)f2u(it.b[3]);
  const uint32_t motion = MOTION ? f2u(it.c[3]) : 0u;
  const V3 o = motion ? moved_origin(S, motion, o_w, time) : o_w;
  float t, u = 0.f, v = 0.f;
  bool h;
  if (type == ITEM_TRI) {
    h = hit_triangle(it, o, d, tmin, tmax, t, u, v);
  } else if (CURVES && type == ITEM_CURVE) {
    const size_t curve = f2u(it.a[0]);
    h = hit_curve(S.curve_segments + 2 * PT_CURVE_SEGMENTS * curve, o, d, tmin, tmax, t, u, v);
    if (h && !(t <= tmax)) h = meets_curve(S.curves + 4 * curve, o, d, tmin, tmax);
  } else if (type == ITEM_CURVE) {
    h = false;
  } else {
    const V3 dn = v3(dn4->x, dn4->y, dn4->z);
    h = type == ITEM_QUAD ? hit_quad<EXACT>(it, o, dn, tmin, tmax, t, state) : hit_sphere(it, o, dn, tmin, tmax, t);
  }
  if (h) {
    hit.t = t;
    hit.prim = (int32_t)f2u(it.a[3]);
    hit.u = u;
    hit.v = v;
  }
  return h;
}

__device__ __forceinline__ bool ref_is_node(int32_t r) { return r >= 0 || r == PT_FRAME_END; }
__device__ __forceinline__ bool ref_is_leaf(int32_t r) { return r < 0 && r != PT_FRAME_END && r != PT_REF_EMPTY; }
// References that change the ray's frame (moving objects).
__device__ __forceinline__ bool ref_is_frame(int32_t r) { return r == PT_FRAME_END || (r >= 0 && (r & PT_INST_BIT)); }

// 1/d of one axis for the slab test.  An axis the ray does not move along
// (d = +-0, or |d| so small that 1/d overflows) gets +-1e20 with d's sign in
// place of +-inf: the slab test computes fmaf(plane, inv, -o * inv), and with
// an infinite inv a ray inside the slab gives inf - inf = NaN, which the
// min / max then drop -- that slab is not tested at all, and an axis-aligned
// ray walks every box its other slabs cross (the whole tree, ~10^5 steps for
// one ray).  With a finite inv the slab gives (-huge, +huge) inside it and an
// entry beyond any tmax outside.
__device__ __forceinline__ float slab_inv(float d) { return fabsf(d) > 1e-20f ? 1.f / d : copysignf(1e20f, d); }

// ------------------------------------------------- warp traversal of a queue
// What a traversal warp keeps in shared memory.  A lane's ray is tested
// against leaf items by whichever lane takes the leaf from the warp's list,
// so everything the item tests read is here and not in the owner's registers.
struct WarpRays {
  float4 o[32];   // origin in the ray's current frame; w: time (motion blur)
  float4 d[32];   // direction; w: tmin
  float4 dn[32];  // normalised direction; w: tmax at the start
  int32_t leaf[64];   // leaves reached and not yet tested, oldest first ...
  uint8_t owner[64];  // ... and the lane whose ray reached each
  uint8_t state[32];  // RayState of the lane's ray
};
// Closest-hit rays only: the nearest hit so far.
struct WarpHits {
  float4 hit[32];      // t, prim (int bits, -1: none), u, v
  uint32_t tmax[32];   // float_key of the ray's tmax (RAY_ALONE: the largest key; its tmax is hit.x)
  int32_t who[32];     // tester whose hit the owner takes
};
// A direction's squared length may be off 1 by this before the ray is walked leaf
// by leaf in a scene with rectangles or spheres (whose t is a distance, while
// triangles and boxes count in the direction's length).  A render's sampled
// directions are within 1e-5.
#define PT_UNIT_TOL 0x1p-12f
// Nodes are culled from this much (relative) behind a hit on: the unit's part of
// PT_UNIT_TOL, and the roundings of a node's entry and of the primitives' t, so
// that whether a primitive that lies within them of the nearest hit is tested
// does not depend on when that hit is found.
#define PT_CULL_SLACK 0x1p-12f
// Lanes (of 32) below which a walk pauses to see whether others have ended.
#define PT_WALK_MIN 8
// One kernel per kind of scene: PT_BY_SCENE(S, RUN) expands RUN(CURVES, MOTION).
#define PT_BY_SCENE(S, RUN)          \
  do {                               \
    if ((S).curves) RUN(true, true); \
    else if ((S).has_motion) RUN(false, true); \
    else RUN(false, false);          \
  } while (0)
enum TraceMode { TRACE_CLOSEST = 0, TRACE_ANY = 1, TRACE_MIXED = 2 };

// Dynamic shared memory of a traversal block: the first PT_STACK_SHARED
// entries of every thread's stack, the warps' records and the rays' world
// origins (kernels for moving objects).
inline size_t trace_smem(int threads, bool any_only = false, bool motion = true) {
  const size_t per = PT_STACK_SHARED * sizeof(int32_t) + (motion ? 3 * sizeof(float) : 0);
  return per * threads + (threads / 32) * (sizeof(WarpRays) + (any_only ? 0 : sizeof(WarpHits)));
}

// Unsigned key with the order of the floats (-0 as +0).
__device__ __forceinline__ uint32_t float_key(float x) {
  const uint32_t b = f2u(x + 0.f);
  return b ^ ((uint32_t)((int32_t)b >> 31) | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
  return u2f(k ^ ((k & 0x80000000u) ? 0x80000000u : 0xffffffffu));
}

__device__ __forceinline__ unsigned lanemask_lt() { return (1u << (threadIdx.x & 31)) - 1u; }

// A lane's walk of the BVH4.
struct TravRay {
  V3 inv, oi;  // 1 / direction, -origin / direction in the current frame
  float tmin, tmax;
  int32_t ref;  // next reference: node (>= 0, PT_INST_BIT: entering a moving
                // object), leaf (< 0), PT_FRAME_END or PT_REF_EMPTY
  int sp;       // stack depth
};

// The per-thread stack: PT_STACK_SHARED entries in shared memory (column per
// thread, conflict free) and the rest in local memory, which few rays reach
// (leaves leave the stack as soon as they are met).
struct TravStack {
  int32_t *sh;  // this thread's column
  int32_t deep[PT_STACK - PT_STACK_SHARED];
  __device__ __forceinline__ void push(int &sp, int32_t r) {
    if (sp < PT_STACK_SHARED) sh[sp * blockDim.x] = r;
    else deep[sp - PT_STACK_SHARED] = r;
    ++sp;
  }
  __device__ __forceinline__ int32_t pop(int &sp) {
    if (sp == 0) return PT_REF_EMPTY;
    --sp;
    return sp < PT_STACK_SHARED ? sh[sp * blockDim.x] : deep[sp - PT_STACK_SHARED];
  }
};

// Two floats in a register pair.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
// (u0, u1) * a + c, one instruction for the pair (both rounded as fmaf): a
// node visit's 24 plane distances take 12 issue slots.  The traversal issues
// in 72-84 % of its cycles; rough glass trace 11.9 -> 11.4 ms, shadow 10.6 ->
// 10.2, Cornell 7.19 -> 6.90.
__device__ __forceinline__ void fma2(uint32_t u0, uint32_t u1, uint64_t a, uint64_t c, float &t0, float &t1) {
  asm("{ .reg .b64 u, t;\n mov.b64 u, {%2, %3};\n fma.rn.f32x2 t, u, %4, %5;\n mov.b64 {%0, %1}, t; }"
      : "=f"(t0), "=f"(t1)
      : "r"(u0), "r"(u1), "l"(a), "l"(c));
}
// Visits node R.ref: afterwards R.ref is the next reference (SORTED: the
// nearest hit child, the others pushed far first; else the first hit child in
// node order), or the top of the stack when no child is hit.  Returns false
// on a stack overflow.
template <bool SORTED>
__device__ __forceinline__ bool visit_node(const SceneView &S, TravRay &R, TravStack &K) {
  uint32_t w[16];
  ld32b(S.nodes + R.ref, w);
  ld32b(reinterpret_cast<const char *>(S.nodes + R.ref) + 32, w + 8);
  // Per axis, plane q at the ray parameter fma(1 + q 2^-15, a, c); the slab a
  // child's entry and exit come from is fixed by the ray's octant (with 1/d >= 0
  // the low plane is the near one; fma is monotonic, so these are the values
  // a min / max of both planes would pick).
  const V3 a = v3(u2f(w[3]) * R.inv.x, u2f(w[4]) * R.inv.y, u2f(w[5]) * R.inv.z);
  const V3 c = v3(fmaf(u2f(w[0]), R.inv.x, R.oi.x), fmaf(u2f(w[1]), R.inv.y, R.oi.y),
                  fmaf(u2f(w[2]), R.inv.z, R.oi.z));
  const bool sx = signbit(R.inv.x), sy = signbit(R.inv.y), sz = signbit(R.inv.z);
  const uint32_t nx = sx ? w[7] : w[6], fx = sx ? w[6] : w[7];
  const uint32_t ny = sy ? w[9] : w[8], fy = sy ? w[8] : w[9];
  const uint32_t nz = sz ? w[11] : w[10], fz = sz ? w[10] : w[11];
  const float tmin = R.tmin, tmax = R.tmax;
  // entry distance per child (+inf when missed or empty), kept in registers;
  // closest-hit visits near to far (sorting network), any-hit in node order.
  float d0, d1, d2, d3;
  int32_t r0 = (int32_t)w[12], r1 = (int32_t)w[13], r2 = (int32_t)w[14], r3 = (int32_t)w[15];
#define PT_PLANE(q, k) __byte_perm(q, 0x3f800000u, 0x7604 | (k << 4))
  const uint64_t ax2 = pack2(a.x, a.x), ay2 = pack2(a.y, a.y), az2 = pack2(a.z, a.z);
  const uint64_t cx2 = pack2(c.x, c.x), cy2 = pack2(c.y, c.y), cz2 = pack2(c.z, c.z);
#define PT_PAIR(q, k, a2, c2, t0, t1) fma2(PT_PLANE(q, k), PT_PLANE(q, k + 1), a2, c2, t0, t1)
#define PT_CHILDREN(k, da, db)                                                                       \
  {                                                                                                  \
    float ex, ey, ez, gx, gy, gz, px, py, pz, qx, qy, qz;                                            \
    PT_PAIR(nx, k, ax2, cx2, ex, gx);                                                                \
    PT_PAIR(ny, k, ay2, cy2, ey, gy);                                                                \
    PT_PAIR(nz, k, az2, cz2, ez, gz);                                                                \
    PT_PAIR(fx, k, ax2, cx2, px, qx);                                                                \
    PT_PAIR(fy, k, ay2, cy2, py, qy);                                                                \
    PT_PAIR(fz, k, az2, cz2, pz, qz);                                                                \
    const float na = fmaxf(fmaxf(ex, ey), fmaxf(ez, tmin)), fa = fminf(fminf(px, py), fminf(pz, tmax)); \
    const float nb = fmaxf(fmaxf(gx, gy), fmaxf(gz, tmin)), fb = fminf(fminf(qx, qy), fminf(qz, tmax)); \
    da = na <= fa ? na : INFINITY;                                                                   \
    db = nb <= fb ? nb : INFINITY;                                                                   \
  }
  PT_CHILDREN(0, d0, d1)
  PT_CHILDREN(2, d2, d3)
#undef PT_CHILDREN
#undef PT_PAIR
#undef PT_PLANE
  if (SORTED) {
#define PT_CSWAP(da, ra, db, rb)   \
  if (db < da) {                   \
    float tt = da;                 \
    da = db;                       \
    db = tt;                       \
    int32_t tr = ra;               \
    ra = rb;                       \
    rb = tr;                       \
  }
    PT_CSWAP(d0, r0, d1, r1)
    PT_CSWAP(d2, r2, d3, r3)
    PT_CSWAP(d0, r0, d2, r2)
    PT_CSWAP(d1, r1, d3, r3)
    PT_CSWAP(d1, r1, d2, r2)
#undef PT_CSWAP
  }
  const bool h0 = d0 < INFINITY, h1 = d1 < INFINITY, h2 = d2 < INFINITY, h3 = d3 < INFINITY;
  if (R.sp > PT_STACK_SHARED - 3) {
    // near the end of the shared part: pushes that may go to local memory
    if (R.sp > PT_STACK - 3) return false;
    int32_t first = PT_REF_EMPTY;
    bool have = false;
    if (h3) { first = r3; have = true; }
    if (h2) { if (have) K.push(R.sp, first); first = r2; have = true; }
    if (h1) { if (have) K.push(R.sp, first); first = r1; have = true; }
    if (h0) { if (have) K.push(R.sp, first); first = r0; have = true; }
    R.ref = have ? first : K.pop(R.sp);
    return true;
  }
  // push the other hits (far first, or in node order), descend into the first
  int sp = R.sp;
  int32_t *top = K.sh + sp * blockDim.x;
  int32_t first = PT_REF_EMPTY;
  if (SORTED) {
    if (h3) { *top = r3; top += blockDim.x; ++sp; }
    if (h2) { *top = r2; top += blockDim.x; ++sp; }
    if (h1) { *top = r1; ++sp; }
    first = r0;  // d0 is the smallest
    R.sp = sp;
    R.ref = h0 ? first : K.pop(R.sp);
  } else {
    bool have = false;
    if (h3) { first = r3; have = true; }
    if (h2) { if (have) { *top = first; top += blockDim.x; ++sp; } first = r2; have = true; }
    if (h1) { if (have) { *top = first; top += blockDim.x; ++sp; } first = r1; have = true; }
    if (h0) { if (have) { *top = first; ++sp; } first = r0; have = true; }
    R.sp = sp;
    R.ref = have ? first : K.pop(R.sp);
  }
  return true;
}

// The items of one leaf in order, EXACT: the result is (t, prim or -1, u, v).  A
// function of its own, so that it lengthens no item test: with the bounds tested
// in trace_rays' loop the 16 k-path Cornell frame's trace took 0.471 ms instead of
// 0.452 and rough glass's 10.58 instead of 10.47 (10.44 without either).  The
// curve kernels, which the call itself would spill (hair 3.93 ms), test the
// bounds in the loop (3.67, from 3.57); so do any-hit rays, to which the order
// does not matter.
template <bool MOTION>
static __device__ __noinline__ float4 leaf_alone(const Item *items, const float4 *motion, int32_t code, float4 o,
                                                 float4 d, float4 dn, float tmax, bool any) {
  SceneView S;  // what test_item reads of it
  S.items = items;
  S.motion = motion;
  HitRec hit;
  hit.t = hit.u = hit.v = 0.f;
  hit.prim = -1;
  const int last = (code >> 3) + (code & 7);
  for (int i = code >> 3; i <= last; ++i) {
    if (!test_item<false, MOTION, true>(S, i, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), &dn, d.w, tmax, hit, o.w, nullptr))
      continue;
    if (any) break;
    tmax = hit.t;
  }
  return make_float4(hit.t, __int_as_float(hit.prim), hit.u, hit.v);
}

// Lanes of a traversal warp that hold rays: all 32 while the queue has 32
// rays or more for every warp of the grid, else an even share of the queue.
__device__ __forceinline__ int warp_lanes(int n) {
  const int warps = gridDim.x * (blockDim.x >> 5);
  return min(32, max(1, (n + warps - 1) / warps));
}

// Traces a queue of n rays with persistent warps and dynamic ray fetch (Aila
// and Laine, "Understanding the efficiency of ray traversal on GPUs", HPG
// 2009, and the 2012 addendum): as soon as `refill` of 32 lanes are free, the
// warp claims that many new rays with one atomic on *fetch.
//
// Node visits and item tests are separate phases of the warp.  A lane that
// reaches a leaf appends it to the warp's list and goes on walking its other
// nodes; once the list holds a leaf for every ray in flight (32 in a full
// warp), or no lane has a node left to visit, the oldest 32 leaves are tested,
// one per lane, whichever lane's ray they belong to.  So the item tests run
// with a full warp and no lane waits at a leaf for the others.  A ray walks
// its nodes with the tmax it had when the list was last tested, i.e. it
// may visit nodes a tighter tmax would cull, whose items then fail; its leaves
// are tested in the order it reached them, and of two equal-t hits the later
// one wins, as in the reference's leaf loop.  (RAY_ALONE rays take a leaf off
// the stack only when the one before is tested, with its tmax.)
//
// Measured against turns in which a warp either visits nodes or tests one item
// per lane standing at a leaf (Cornell box, 256 x 256 x 64 spp): 15.3 -> 20.1
// active threads per instruction in the shadow kernel, 8.29 -> 6.66 ms for
// its 51 M rays (with the compact ray list, PT_FETCH_IDLE_SHADOW 16).  Rough
// glass, 16.8 M paths: trace 16.5 -> 13.8 ms (39 M rays), shadow 16.8 ->
// 13.3 ms (45 M).  Testing from 24 leaves on instead of 32 takes any-hit rays
// 23.9 -> 23.2 ms on the material divergence and 5.68 -> 5.62 on Cornell (they
// end sooner); from 20 on 23.9 and 5.69; closest hits +0.4 % at 24, so 32 there.  With 32 lanes always (no
// even share) bounces of few rays wait for each other's leaves: the
// 0.48 M-path glass frame 3.57 -> 3.9 ms.
//
// A turn of the walk does one node visit; done rays and the refill are looked at
// only when PT_WALK_MIN lanes or fewer still walk (rough glass trace 12.9 ->
// 12.2 ms, shadow 11.5 -> 10.6 against a look every turn; 8 / 12 / 16 lanes are
// within 1 %, closest hits at 20 +3 %).  MOTION = false (scenes without
// moving objects) compiles the changes of frame out: trace 11.4 -> 10.9 ms, the
// 0.48 M-path glass frame's 1.60 -> 1.49.
//
// fetch_ray(r, o, d, tmin, tmax, time, any): loads ray r, false: no ray there.
// done(found, hit): the lane's ray is finished.
template <int MODE, bool CURVES, bool MOTION, class Fetch, class Done>
__device__ __forceinline__ void trace_rays(const SceneView &S, int n, int *fetch, int refill32, int *err, char *smem,
                                           Fetch fetch_ray, Done done) {
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  TravStack K;
  K.sh = reinterpret_cast<int32_t *>(smem) + threadIdx.x;
  smem += PT_STACK_SHARED * sizeof(int32_t) * blockDim.x;
  WarpRays &W = reinterpret_cast<WarpRays *>(smem)[threadIdx.x >> 5];
  smem += warps * sizeof(WarpRays);
  WarpHits &H = reinterpret_cast<WarpHits *>(smem)[threadIdx.x >> 5];
  if (MODE != TRACE_ANY) smem += warps * sizeof(WarpHits);
  float *ow = reinterpret_cast<float *>(smem) + 3 * threadIdx.x;  // world origin (MOTION)
  const int lanes = warp_lanes(n), refill = max(1, lanes * refill32 / 32);
  const int walk_min = lanes * PT_WALK_MIN / 32;
  TravRay R;
  R.ref = PT_REF_EMPTY;
  R.sp = 0;
  int iters = 0;
  bool active = false;     // the lane has a ray in flight
  bool pend = false;       // the list holds leaves of this lane's (last) ray
  bool alone = false;      // its ray is RAY_ALONE
  bool any = MODE == TRACE_ANY;
  bool exhausted = false;  // the queue has no unclaimed rays
  int qn = 0;              // leaves in the list
  for (;;) {
    // ---- rays that ended: nothing left to visit or to test
    while (active && !pend && R.ref == PT_REF_EMPTY && R.sp > 0) R.ref = K.pop(R.sp);
    if (active && !pend && R.ref == PT_REF_EMPTY) {
      if (MODE != TRACE_ANY && W.state[lane] == RAY_MARKED) {
        // again, leaf by leaf
        W.state[lane] = RAY_ALONE;
        if (MOTION) {  // in the world's frame
          const V3 o = v3(ow[0], ow[1], ow[2]);
          W.o[lane] = make_float4(o.x, o.y, o.z, W.o[lane].w);
          R.oi = v3(-o.x * R.inv.x, -o.y * R.inv.y, -o.z * R.inv.z);
        }
        R.tmax = W.dn[lane].w;
        H.hit[lane] = make_float4(R.tmax, __int_as_float(-1), 0.f, 0.f);
        H.tmax[lane] = 0xffffffffu;
        R.ref = any ? S.any_root : 0;
        iters = 0;
        alone = true;
      } else {
        HitRec h;
        h.prim = -1;
        if (MODE != TRACE_ANY) {
          const float4 b = H.hit[lane];
          h.t = b.x;
          h.prim = __float_as_int(b.y);
          h.u = b.z;
          h.v = b.w;
        }
        done(h.prim >= 0, h);
        active = false;
      }
    }
    // ---- refill
    const unsigned idle = __ballot_sync(0xffffffffu, !active && !pend);
    const int in_flight = 32 - __popc(idle);
    const int k = lanes - in_flight;  // rays to claim
    if (!exhausted && k >= refill) {
      int base = 0;
      if (lane == 0) base = atomicAdd(fetch, k);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + k >= n) exhausted = true;
      const int rank = __popc(idle & lanemask_lt());
      if (!active && !pend && rank < k) {
        const int r = base + rank;
        V3 o, d;
        float time = 0.f;
        if (r < n && fetch_ray(r, o, d, R.tmin, R.tmax, time, any)) {
          const V3 dn = xnormalize(d);
          W.o[lane] = make_float4(o.x, o.y, o.z, time);
          W.d[lane] = make_float4(d.x, d.y, d.z, R.tmin);
          W.dn[lane] = make_float4(dn.x, dn.y, dn.z, R.tmax);
          W.state[lane] = RAY_ORDERED;
          alone = false;
          if (MODE != TRACE_ANY) {
            H.hit[lane] = make_float4(FLT_MAX, __int_as_float(-1), 0.f, 0.f);
            H.tmax[lane] = float_key(R.tmax);
            H.who[lane] = any ? -2 : -1;  // -2: an any-hit ray
          }
          if (MOTION) {
            ow[0] = o.x;
            ow[1] = o.y;
            ow[2] = o.z;
          }
          R.inv = v3(slab_inv(d.x), slab_inv(d.y), slab_inv(d.z));
          R.oi = v3(-o.x * R.inv.x, -o.y * R.inv.y, -o.z * R.inv.z);
          // the host always emits at least one node
          R.ref = any ? S.any_root : 0;
          R.sp = 0;
          iters = 0;
          active = true;
          // rays of which every hit is without an order: not finite, or so far
          // that products of their coordinates are not; tmax NaN; or of hits in
          // another unit than the boxes', so that what a hit culls depends on
          // when it is found
          const float dd = xdot(d, d), size = fabsf(o.x) + fabsf(o.y) + fabsf(o.z) + dd;
          if (MODE != TRACE_ANY && (!(size < 1e18f) || R.tmax != R.tmax ||
                                    (S.unit_t && !any && fabsf(dd - 1.f) > PT_UNIT_TOL))) {
            W.state[lane] = RAY_MARKED;
            R.ref = PT_REF_EMPTY;
          }
        }
      }
      __syncwarp();
      continue;
    }
    // ---- walk: leaves reached go to the list, a node visit for every lane
    // that stands at one; until the list is full, or so few lanes walk on that
    // others may have ended
    const int full = min(MODE == TRACE_ANY ? 24 : 32, in_flight);
    unsigned rm;
    for (;;) {
      const bool leaf = active && ref_is_leaf(R.ref);
      const unsigned lm = __ballot_sync(0xffffffffu, leaf);
      if (leaf) {
        const int at = qn + __popc(lm & lanemask_lt());
        W.leaf[at] = R.ref;
        W.owner[at] = (uint8_t)lane;
        pend = true;
        ++iters;
        R.ref = MODE != TRACE_ANY && alone ? PT_REF_EMPTY : K.pop(R.sp);  // popped when the leaf is tested
      }
      qn += __popc(lm);
      const bool ready = active && ref_is_node(R.ref) && !(MOTION && pend && ref_is_frame(R.ref));
      rm = __ballot_sync(0xffffffffu, ready);
      if (!rm || qn >= full) break;
      if (ready) {
        bool ok = ++iters <= S.trav_cap;
        if (!ok) *err = 2;
        if (ok && MOTION && ref_is_frame(R.ref)) {
          // the ray in the next frame: a moving object's at its time (until
          // PT_FRAME_END comes off the stack), or back in the world's
          V3 o = v3(ow[0], ow[1], ow[2]);
          if (R.ref == PT_FRAME_END) {
            R.ref = K.pop(R.sp);
          } else {
            R.ref &= ~PT_INST_BIT;
            ok = R.sp < PT_STACK;
            if (ok) K.push(R.sp, PT_FRAME_END);
            o = moved_origin(S, (uint32_t)__ldg(S.node_motion + R.ref), o, W.o[lane].w);
          }
          R.oi = v3(-o.x * R.inv.x, -o.y * R.inv.y, -o.z * R.inv.z);
          W.o[lane] = make_float4(o.x, o.y, o.z, W.o[lane].w);
          if (!ok) *err = 1;
        }
        if (ok && ref_is_node(R.ref) && !(MOTION && ref_is_frame(R.ref))) {
          ok = visit_node<MODE != TRACE_ANY>(S, R, K);
          if (!ok) *err = 1;
        }
        if (!ok) {  // ended with what it has
          R.ref = PT_REF_EMPTY;
          R.sp = 0;
        }
      }
      if (__popc(rm) <= walk_min) break;
    }
    if (rm && qn < full) continue;
    if (!qn) {
      if (exhausted && idle == 0xffffffffu) break;
      continue;
    }
    // ---- item tests: the oldest leaves, one per lane
    __syncwarp();
    const int m = min(qn, 32);
    const int own = lane < m ? W.owner[lane] : 0;
    const int32_t lref = lane < m ? W.leaf[lane] : 0;
    const bool rest = 32 + lane < qn;
    const int rown = rest ? W.owner[32 + lane] : 0;
    const int32_t rleaf = rest ? W.leaf[32 + lane] : 0;
    bool hit = false, eany = MODE == TRACE_ANY;
    HitRec h;
    if (lane < m) {
      const float4 o4 = W.o[own], d4 = W.d[own];
      float tm;
      if (MODE == TRACE_MIXED) eany = H.who[own] == -2;
      if (MODE == TRACE_ANY) tm = W.dn[own].w;
      else tm = key_float(H.tmax[own]);
      const V3 o = v3(o4.x, o4.y, o4.z), d = v3(d4.x, d4.y, d4.z);
      const int32_t code = ~lref;  // first_item << 3 | count - 1
      int last = (code >> 3) + (code & 7);
      const bool again = MODE != TRACE_ANY && W.state[own] == RAY_ALONE;
      if (again && !eany) tm = H.hit[own].x;
      if (!CURVES && again) {
        const float4 b = leaf_alone<MOTION>(S.items, S.motion, code, o4, d4, W.dn[own], tm, eany);
        h.t = b.x;
        h.prim = __float_as_int(b.y);
        h.u = b.z;
        h.v = b.w;
        hit = h.prim >= 0;
        last = -1;  // tested
      }
      for (int i = code >> 3; i <= last; ++i) {
        if (test_item<CURVES, MOTION, CURVES || MODE == TRACE_ANY>(S, i, o, d, &W.dn[own], d4.w, tm, h, o4.w,
                                                                   &W.state[own])) {
          hit = true;
          if (eany) break;
          if (CURVES && !again && !(h.t <= tm)) W.state[own] = RAY_MARKED;
          tm = h.t;
        }
      }
    }
    __syncwarp();
    if (rest) {
      W.owner[lane] = (uint8_t)rown;
      W.leaf[lane] = rleaf;
    }
    qn -= m;
    const unsigned left = __reduce_or_sync(0xffffffffu, rest ? 1u << rown : 0u);
    if (MODE != TRACE_CLOSEST) {
      const unsigned occ = __reduce_or_sync(0xffffffffu, hit && eany ? 1u << own : 0u);
      if (active && any && (occ >> lane & 1u)) {
        HitRec none;
        none.prim = 0;
        done(true, none);
        active = false;
        R.ref = PT_REF_EMPTY;
        R.sp = 0;
      }
    }
    if (MODE != TRACE_ANY) {
      // the nearest of the leaves' hits per owner; of equal ones the latest
      const bool cand = hit && !eany;
      if (__any_sync(0xffffffffu, cand)) {
        const uint32_t key = float_key(h.t);
        if (cand) atomicMin(&H.tmax[own], key);
        __syncwarp();
        const bool best = cand && H.tmax[own] == key;
        if (best) atomicMax(&H.who[own], lane);
        __syncwarp();
        if (best && H.who[own] == lane) H.hit[own] = make_float4(h.t, __int_as_float(h.prim), h.u, h.v);
        __syncwarp();
        if (active && !any) {
          const float t = key_float(H.tmax[lane]);
          R.tmax = alone ? H.hit[lane].x : fmaf(fabsf(t), PT_CULL_SLACK, t);
          if (alone) H.tmax[lane] = 0xffffffffu;
          H.who[lane] = -1;
        }
      }
    }
    pend = (left >> lane) & 1u;
    __syncwarp();
  }
}

}  // namespace pt
