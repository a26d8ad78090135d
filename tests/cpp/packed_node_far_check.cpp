// Host check of the packed BVH nodes (pt_node.cuh) far from the world's origin: up
// to 10^7 node extents away, with ray origins of up to 3 times the node's
// coordinates on each axis, in all directions.  Every ray that meets a child's box
// in 64 bits, or in the plain slab test of the float box, meets its packed box in
// the arithmetic the traversal uses; a box with a bound that is not a number is met
// wherever its other axes are.  Prints one line per check and exits non-zero on a
// mismatch.
#include "../../pathtracer_gb300/csrc/pt_node.cuh"

#include <cstdio>
#include <random>

using namespace pt;

static float slab_inv(float d) { return std::fabs(d) > 1e-20f ? 1.f / d : std::copysign(1e20f, d); }
static float plane(uint32_t bytes, int c) { return u2f(0x3f800000u | (((bytes >> (8 * c)) & 255u) << 8)); }

struct Ray {
  float o[3], d[3], inv[3], oi[3];
};
static bool meets_packed(const PackedNode &P, const Ray &r, int c, float tmin, float tmax) {
  const uint32_t ql[3] = {P.lo_x, P.lo_y, P.lo_z}, qh[3] = {P.hi_x, P.hi_y, P.hi_z};
  float n = tmin, f = tmax;
  for (int a = 0; a < 3; ++a) {
    const bool neg = std::signbit(r.inv[a]);
    const float ax = P.scale[a] * r.inv[a], cx = std::fmaf(P.origin[a], r.inv[a], r.oi[a]);
    n = std::fmax(n, std::fmaf(plane(neg ? qh[a] : ql[a], c), ax, cx));
    f = std::fmin(f, std::fmaf(plane(neg ? ql[a] : qh[a], c), ax, cx));
  }
  return n <= f;
}

int main() {
  std::mt19937_64 gen(11);
  auto uni = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); };
  long long exact = 0, wide_hits = 0, lost_exact = 0, lost_wide = 0, nan_lost = 0;
  for (int it = 0; it < 120000; ++it) {
    const double ext = std::exp(uni(std::log(1e-4), std::log(1e3)));
    const double off = ext * std::exp(uni(0.0, std::log(it % 2 ? 1e7 : 1e3)));
    double ctr[3];
    for (double &x : ctr) x = off * uni(-1, 1);
    Bvh4Node N;
    const int nch = 1 + (int)(gen() % 4);
    float *lo[3] = {N.lo_x, N.lo_y, N.lo_z}, *hi[3] = {N.hi_x, N.hi_y, N.hi_z};
    double reach[3] = {0, 0, 0};
    for (int c = 0; c < 4; ++c) {
      N.child[c] = c;
      N.count[c] = c < nch ? 0 : -1;
      const int flat = (int)(gen() % 5);  // an axis of no extent
      for (int a = 0; a < 3; ++a) {
        lo[a][c] = INFINITY;
        hi[a][c] = -INFINITY;
        if (c >= nch) continue;
        const double m = ctr[a] + uni(-0.5, 0.5) * ext, h = a == flat ? 0.0 : uni(0.0, 0.3) * ext;
        lo[a][c] = (float)(m - h);
        hi[a][c] = (float)(m + h);
        reach[a] = std::fmax(reach[a], std::fmax(std::fabs((double)lo[a][c]), std::fabs((double)hi[a][c])));
      }
    }
    const PackedNode P = pack_node(N);
    Bvh4Node M = N;  // one bound of child 0 is not a number
    const int bad = (int)(gen() % 3);
    (gen() % 2 ? (bad == 0 ? M.lo_x : bad == 1 ? M.lo_y : M.lo_z) : (bad == 0 ? M.hi_x : bad == 1 ? M.hi_y : M.hi_z))[nch - 1] = NAN;
    const PackedNode PM = pack_node(M);
    for (int k = 0; k < 60; ++k) {
      Ray r;
      const int c = (int)(gen() % nch);
      double to[3], tl = 0.0;
      const double near = k % 3 == 0 ? 1.0 : std::exp(uni(std::log(1e-6), 0.0));
      for (int a = 0; a < 3; ++a) {
        // origins of up to 3 times the coordinates, some of them close by
        r.o[a] = (float)(near == 1.0 ? 3.0 * reach[a] * uni(-1, 1) : ctr[a] + near * 2.0 * reach[a] * uni(-1, 1));
        if (std::fabs((double)r.o[a]) > 3.0 * reach[a]) r.o[a] = (float)(2.9 * reach[a]);
        // aim at the box, three quarters of the rays at one of its edges
        const double s = uni(-1, 1), m = 0.5 * ((double)lo[a][c] + hi[a][c]), h = 0.5 * ((double)hi[a][c] - lo[a][c]);
        to[a] = m + (k % 4 == 0 || a == (k / 4) % 3 ? s : std::copysign(1.0, s)) * h - r.o[a];
        if (k % 7 == 0 && a == k % 3) to[a] = 0.0;
        tl += to[a] * to[a];
      }
      tl = std::sqrt(tl);
      for (int a = 0; a < 3; ++a) {
        r.d[a] = (float)(to[a] / (tl > 0 ? tl : 1.0));
        r.inv[a] = slab_inv(r.d[a]);
        r.oi[a] = -r.o[a] * r.inv[a];
      }
      const float tmin = 1e-4f, tmax = 1e30f;
      double en = tmin, ef = tmax;
      float wn = tmin, wf = tmax;
      for (int a = 0; a < 3; ++a) {
        const bool neg = std::signbit(r.inv[a]);
        const float pn = neg ? hi[a][c] : lo[a][c], pf = neg ? lo[a][c] : hi[a][c];
        wn = std::fmax(wn, std::fmaf(pn, r.inv[a], r.oi[a]));
        wf = std::fmin(wf, std::fmaf(pf, r.inv[a], r.oi[a]));
        if (r.d[a] == 0.f) {
          if (r.o[a] < lo[a][c] || r.o[a] > hi[a][c]) ef = -INFINITY;
        } else {
          en = std::fmax(en, ((double)pn - r.o[a]) / r.d[a]);
          ef = std::fmin(ef, ((double)pf - r.o[a]) / r.d[a]);
        }
      }
      const bool packed = meets_packed(P, r, c, tmin, tmax);
      exact += en <= ef;
      wide_hits += wn <= wf;
      lost_exact += en <= ef && !packed;
      lost_wide += wn <= wf && !packed;
      if (en <= ef && c == nch - 1) nan_lost += !meets_packed(PM, r, c, tmin, tmax);
    }
  }
  std::printf("boxes met in 64 bits: %lld, %lld lost by packing\n", exact, lost_exact);
  std::printf("float boxes met: %lld, %lld lost by packing\n", wide_hits, lost_wide);
  std::printf("boxes with a bound that is not a number: %lld lost\n", nan_lost);
  return lost_exact == 0 && lost_wide == 0 && nan_lost == 0 && exact > 100000 ? 0 : 1;
}
