// Host check of the packed BVH nodes (pt_node.cuh): every ray that passes a
// child's float box in the plain slab test passes its packed box in the
// arithmetic the traversal uses, for random nodes of all scales and offsets,
// one to four children, flat and degenerate boxes, rays from inside, near by
// and up to 1000 node extents away, axis-parallel ones among them; empty
// slots are never passed.  Prints one line per check and exits non-zero on a
// mismatch.
#include "../../pathtracer_gb300/csrc/pt_node.cuh"

#include <cstdio>
#include <random>

using namespace pt;

static float slab_inv(float d) { return std::fabs(d) > 1e-20f ? 1.f / d : std::copysign(1e20f, d); }

static float plane(uint32_t bytes, int c) { return u2f(0x3f800000u | (((bytes >> (8 * c)) & 255u) << 8)); }

int main() {
  std::mt19937_64 gen(5);
  auto uni = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); };
  long long wide_hits = 0, lost = 0, extra = 0, tests = 0, ghosts = 0, refs = 0;
  for (int it = 0; it < 40000; ++it) {
    const double ext = std::exp(uni(std::log(1e-4), std::log(1e4)));
    const double off = (it % 3 == 0) ? 0.0 : ext * std::exp(uni(0.0, std::log(1e3)));
    const double ctr[3] = {off * uni(-1, 1), off * uni(-1, 1), off * uni(-1, 1)};
    Bvh4Node N;
    const int nch = 1 + (int)(gen() % 4);
    float *lo[3] = {N.lo_x, N.lo_y, N.lo_z}, *hi[3] = {N.hi_x, N.hi_y, N.hi_z};
    for (int c = 0; c < 4; ++c) {
      N.child[c] = it + c;
      N.count[c] = c < nch ? (int)(gen() % 9) : -1;
      const int flat = (int)(gen() % 5);  // an axis of (nearly) no extent
      for (int a = 0; a < 3; ++a) {
        lo[a][c] = INFINITY;
        hi[a][c] = -INFINITY;
        if (c >= nch) continue;
        const double m = ctr[a] + uni(-0.5, 0.5) * ext, h = a == flat ? 0.0 : uni(0.0, 0.3) * ext;
        lo[a][c] = (float)(m - h);
        hi[a][c] = (float)(m + h);
      }
    }
    const PackedNode P = pack_node(N);
    const uint32_t ql[3] = {P.lo_x, P.lo_y, P.lo_z}, qh[3] = {P.hi_x, P.hi_y, P.hi_z};
    for (int c = 0; c < 4; ++c) refs += P.ref[c] != trav_ref(N.child[c], N.count[c]);
    for (int r = 0; r < 60; ++r) {
      const double dist = (r % 4 == 0) ? 0.4 * ext : ext * std::exp(uni(0.0, std::log(1000.0)));
      float o[3], d[3];
      double dir[3], len = 0.0;
      for (int a = 0; a < 3; ++a) len += (dir[a] = uni(-1, 1)) * dir[a];
      len = std::sqrt(len);
      double to[3], tl = 0.0;
      for (int a = 0; a < 3; ++a) {
        o[a] = (float)(ctr[a] - dist * dir[a] / len);
        to[a] = ctr[a] + uni(-0.6, 0.6) * ext - o[a];
        if (r % 7 == 0 && a == (int)(gen() % 3)) to[a] = 0.0;
        tl += to[a] * to[a];
      }
      tl = std::sqrt(tl);
      for (int a = 0; a < 3; ++a) d[a] = (float)(to[a] / (tl > 0 ? tl : 1.0));
      float inv[3], oi[3], ax[3], cx[3];
      for (int a = 0; a < 3; ++a) {
        inv[a] = slab_inv(d[a]);
        oi[a] = -o[a] * inv[a];
        ax[a] = P.scale[a] * inv[a];
        cx[a] = std::fmaf(P.origin[a], inv[a], oi[a]);
      }
      const float tmin = 1e-4f, tmax = r % 5 == 0 ? (float)(dist) : 1e5f;
      for (int c = 0; c < 4; ++c) {
        float wn = tmin, wf = tmax, pn = tmin, pf = tmax;
        for (int a = 0; a < 3; ++a) {
          const bool neg = std::signbit(inv[a]);
          wn = std::fmax(wn, std::fmaf(neg ? hi[a][c] : lo[a][c], inv[a], oi[a]));
          wf = std::fmin(wf, std::fmaf(neg ? lo[a][c] : hi[a][c], inv[a], oi[a]));
          pn = std::fmax(pn, std::fmaf(plane(neg ? qh[a] : ql[a], c), ax[a], cx[a]));
          pf = std::fmin(pf, std::fmaf(plane(neg ? ql[a] : qh[a], c), ax[a], cx[a]));
        }
        const bool wide = c < nch && wn <= wf, packed = pn <= pf;
        ++tests;
        wide_hits += wide;
        if (wide && !packed) ++lost;
        if (c < nch && packed && !wide) ++extra;
        if (c >= nch && packed) ++ghosts;
      }
    }
  }
  std::printf("children hit: %lld of %lld, %lld lost by packing\n", wide_hits, tests, lost);
  std::printf("extra hits of packed boxes: %lld (%s)\n", extra, extra * 4 < wide_hits ? "0 excess" : "too many");
  std::printf("empty slots hit: %lld, references changed: %lld\n", ghosts, refs);
  return lost == 0 && extra * 4 < wide_hits && ghosts == 0 && refs == 0 && wide_hits > 100000 ? 0 : 1;
}
