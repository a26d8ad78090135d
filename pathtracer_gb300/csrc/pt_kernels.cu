// pt_kernels.cu -- the wavefront stages of the NEE(+MIS) path integrator for
// single-job waves, the job-independent stages shared with merged waves, and
// the batch test kernels behind the C-ABI.
//
// One wave = a contiguous range of (sample, pixel) paths.  Per bounce:
//   k_trace_closest  RayQueue -> HitQueue            (packed BVH4, warp-wide leaf list)
//   k_sort_*         HitQueue -> order by material family (counting sort)
//   k_sample         order -> sampler dimensions and keys of the sorted vertices
//   k_shade<FAM>     logic + BSDF sample + NEE: writes next RayQueue
//                    (warp-aggregated compaction) and ShadowQueue
//   k_trace_shadow   ShadowQueue any-hit visibility
//   k_shadow_resolve visible NEE terms added to L in a fixed order
// and once per wave k_camera (RayQueue 0) and k_film (ordered per-pixel
// accumulation).  Small waves trace a bounce's shadow rays together with the
// next bounce's closest-hit rays (k_trace_pair, pt_wave.cuh).
#include "pt_wave.cuh"

namespace pt {

// ------------------------------------------------------------ test kernels
__global__ void k_sampler_eval(int strategy, const uint16_t *perm, uint32_t first, int n, int dims,
                               float *out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)n * dims;
       i += (long long)gridDim.x * blockDim.x) {
    int s = (int)(i / dims), d = (int)(i % dims);
    uint32_t idx = first + (uint32_t)s;
    float v;
    if (strategy == PT_SAMPLER_HALTON_NONE)
      v = radical_inverse(c_halton, d, idx);
    else if (strategy == PT_SAMPLER_HALTON_PERMUTE)
      v = permuted_radical_inverse(c_halton, perm, d, idx);
    else
      v = owen_radical_inverse(c_halton, d, idx);
    out[i] = v;
  }
}

// Sample values of the paths [first, first + n) of a single-job wave, from
// the device functions the camera and shade stages call: the pixel-grid
// offset of the path's sample (k_camera), the sampler dimensions
// 0..dims-1 (sampler_dim) and, per bounce b < bounces, the LN light-point
// offsets (light_offset at the vertex's slot base 64 + 32 b).
__global__ void k_path_samples(DeviceJob J, long long first, int n, int dims, int bounces, int LN, float *pix,
                               float *dv, float *lo) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    const PathId P = path_id(J, first + s);
    if (pix) {
      const float2 o = J.job.offsets[P.k];
      pix[2 * (size_t)s] = o.x;
      pix[2 * (size_t)s + 1] = o.y;
    }
    if (dv)
      for (int d = 0; d < dims; ++d)
        dv[(size_t)s * dims + d] = sampler_dim(J, d, P.halton_index, P.key, P.pix, P.k);
    if (lo)
      for (int b = 0; b < bounces; ++b)
        for (int ls = 0; ls < LN; ++ls) {
          const float2 o = light_offset(J, P.key, 64u + 32u * (uint32_t)b, ls);
          const size_t i = (((size_t)s * bounces + b) * LN + ls) * 2;
          lo[i] = o.x;
          lo[i + 1] = o.y;
        }
  }
}

void launch_path_samples(const DeviceJob &J, long long first, int n, int dims, int bounces, float *pix, float *dv,
                         float *lo, cudaStream_t st) {
  const int LN = J.job.light_nx * J.job.light_ny;
  k_path_samples<<<grid_for(n, 128, 152 * 8), 128, 0, st>>>(J, first, n, dims, bounces, LN, pix, dv, lo);
}

// Blocks of a query: the warps of the whole chip, down to 4 rays per warp (a
// warp of few rays ends sooner: its rays do not wait for each other's turns).
static int query_grid(int n) { return grid_for(n, 16, 152 * 7); }

// The batch ray queries: closest hits or occlusion of n given rays.  fetch.now
// is 0 at the start; the kernel clears fetch.next for the next query (queries of
// a context take turns, which saves clearing it by a memset: 2 of ~110 us for
// 2500 rays).  The bounds hold 7 blocks per SM (6 with motion); left free, the
// closest-hit form takes 80 registers and 6: 262 k rays in a closed scene 342
// instead of 333 us.
template <bool ANY, bool CURVES, bool MOTION>
__global__ void __launch_bounds__(128, ANY ? (CURVES ? 7 : 8) : (MOTION ? 6 : 7))
    k_trace_test(SceneView S, const float *rays, const float *tmaxs, int n, float tmin, float tmax, float *t_out,
                 int *prim_out, float *uv_out, uint8_t *occ, FetchPair fetch, int *err) {
  extern __shared__ __align__(16) char smem[];  // trace_smem
  if (blockIdx.x == 0 && threadIdx.x == 0) *fetch.next = 0;
  int i = 0;
  trace_rays<ANY ? TRACE_ANY : TRACE_CLOSEST, CURVES, MOTION>(
      S, n, fetch.now, ANY ? PT_FETCH_IDLE_SHADOW : PT_FETCH_IDLE, err, smem,
      [&](int r, V3 &o, V3 &d, float &t0, float &t1, float &, bool &) {
        i = r;
        const float *p = rays + 6 * (size_t)r;
        o = v3(p[0], p[1], p[2]);
        d = v3(p[3], p[4], p[5]);
        t0 = tmin;
        t1 = ANY ? tmaxs[r] : tmax;
        return true;
      },
      [&](bool found, const HitRec &h) {
        if (ANY) {
          occ[i] = found ? 1 : 0;
        } else {
          t_out[i] = found ? h.t : FLT_MAX;
          prim_out[i] = found ? h.prim : -1;
          uv_out[2 * (size_t)i] = found ? h.u : 0.f;
          uv_out[2 * (size_t)i + 1] = found ? h.v : 0.f;
        }
      });
}

// Hittable::intersect's HitRecord (base/primitive.hpp:30-79) at the closest
// hit: t, primitive, position, the normal turned towards the ray
// (HitRecord::set_normal) and is_inside (the front-face flag, FlipFace
// toggled) -- what surface_at gives the shade stage.
__global__ void __launch_bounds__(128, 6) k_intersect(SceneView S, const float *rays, int n, float tmin, float tmax,
                                                   float *t_out, int *prim_out, float *pos, float *nrm,
                                                   uint8_t *front, FetchPair fetch, int *err) {
  extern __shared__ __align__(16) char smem[];  // trace_smem
  if (blockIdx.x == 0 && threadIdx.x == 0) *fetch.next = 0;
  int i = 0;
  trace_rays<TRACE_CLOSEST, true, true>(
      S, n, fetch.now, PT_FETCH_IDLE, err, smem,
      [&](int r, V3 &o, V3 &d, float &t0, float &t1, float &, bool &) {
        i = r;
        const float *p = rays + 6 * (size_t)r;
        o = v3(p[0], p[1], p[2]);
        d = v3(p[3], p[4], p[5]);
        t0 = tmin;
        t1 = tmax;
        return true;
      },
      [&](bool found, const HitRec &h) {
        const float *p = rays + 6 * (size_t)i;
        Surf sf;
        sf.p = sf.n = v3(0.f);
        sf.front = false;
        if (found) sf = surface_at(S, v3(p[0], p[1], p[2]), v3(p[3], p[4], p[5]), h, 0.f);
        t_out[i] = found ? h.t : FLT_MAX;
        prim_out[i] = found ? h.prim : -1;
        pos[3 * (size_t)i] = sf.p.x;
        pos[3 * (size_t)i + 1] = sf.p.y;
        pos[3 * (size_t)i + 2] = sf.p.z;
        nrm[3 * (size_t)i] = sf.n.x;
        nrm[3 * (size_t)i + 1] = sf.n.y;
        nrm[3 * (size_t)i + 2] = sf.n.z;
        front[i] = (found && sf.front) ? 1 : 0;
      });
}

void launch_intersect(const SceneView &S, const float *rays, int n, float tmin, float tmax, float *t, int *prim,
                      float *pos, float *nrm, uint8_t *front, FetchPair fetch, int *err, cudaStream_t st) {
  k_intersect<<<query_grid(n), 128, trace_smem(128), st>>>(S, rays, n, tmin, tmax, t, prim, pos, nrm,
                                                                         front, fetch, err);
}

// The Light methods of one light of a resident scene at n (u, v, x) items:
// get_sample, get_normal_at, the direction from x, L_emit towards x and
// pdf_value(x, dir) -- light_point / light_pdf_value, the code NEE runs.
__global__ void k_light_eval(SceneView S, int light, int n, const float *uv, const float *x, const float *pdf_dir,
                             float *point, float *normal, float *dir, float *le, float *pdf) {
  const LightRec &Lr = S.lights[light];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const V3 xi = v3(x[3 * i], x[3 * i + 1], x[3 * i + 2]);
    const LightPoint P = light_point(S, Lr, uv[2 * i], uv[2 * i + 1], xi, 0.f);
    const V3 pd = pdf_dir ? v3(pdf_dir[3 * i], pdf_dir[3 * i + 1], pdf_dir[3 * i + 2]) : P.w;
    const float pv = light_pdf_value(Lr, xi, pd);
    const V3 out[4] = {P.p, P.n, P.w, P.Le};
    float *dst[4] = {point, normal, dir, le};
    for (int k = 0; k < 4; ++k) {
      dst[k][3 * i] = out[k].x;
      dst[k][3 * i + 1] = out[k].y;
      dst[k][3 * i + 2] = out[k].z;
    }
    pdf[i] = pv;
  }
}

void launch_light_eval(const SceneView &S, int light, int n, const float *uv, const float *x, const float *pdf_dir,
                       float *point, float *normal, float *dir, float *le, float *pdf, cudaStream_t st) {
  k_light_eval<<<grid_for(n, 128, 152 * 8), 128, 0, st>>>(S, light, n, uv, x, pdf_dir, point, normal, dir, le, pdf);
}

__global__ void k_bsdf_eval(const MatRec *m, int n, const float *wo, const float *wi,
                            const float *nrm, const uint8_t *front, float *f, float *pdf) {
  MatRec mat = *m;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    V3 o = v3(wo[3 * i], wo[3 * i + 1], wo[3 * i + 2]);
    V3 w = v3(wi[3 * i], wi[3 * i + 1], wi[3 * i + 2]);
    V3 nn = v3(nrm[3 * i], nrm[3 * i + 1], nrm[3 * i + 2]);
    V3 fv = bsdf_f(mat, o, w, nn, front[i] != 0);
    f[3 * i] = fv.x;
    f[3 * i + 1] = fv.y;
    f[3 * i + 2] = fv.z;
    pdf[i] = bsdf_pdf(mat, o, w, nn, front[i] != 0);
  }
}

__global__ void k_bsdf_sample(const MatRec *m, int n, const float *wo, const float *nrm,
                              const uint8_t *front, const float *uc, const float *u, uint8_t *ok,
                              float *wi, float *att, float *pdf, uint32_t *type) {
  MatRec mat = *m;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    V3 o = v3(wo[3 * i], wo[3 * i + 1], wo[3 * i + 2]);
    V3 nn = v3(nrm[3 * i], nrm[3 * i + 1], nrm[3 * i + 2]);
    BsdfSample s = bsdf_sample(mat, o, nn, front[i] != 0, uc[i], u[2 * i], u[2 * i + 1]);
    ok[i] = s.ok ? 1 : 0;
    wi[3 * i] = s.ok ? s.wi.x : 0.f;
    wi[3 * i + 1] = s.ok ? s.wi.y : 0.f;
    wi[3 * i + 2] = s.ok ? s.wi.z : 0.f;
    att[3 * i] = s.ok ? s.att.x : 0.f;
    att[3 * i + 1] = s.ok ? s.att.y : 0.f;
    att[3 * i + 2] = s.ok ? s.att.z : 0.f;
    pdf[i] = s.ok ? s.pdf : 0.f;
    type[i] = s.ok ? s.type : 0u;
  }
}

// Sort bins: material type 0..7 of the surface hit, PT_KEY_MISS,
// PT_KEY_MEDIUM, with one more bin after the Disney type: its inside hits.
// DisneyPrincipledBSDF evaluates the glass lobe alone on a front-face hit and
// the mixture of five lobes behind it, so warps that mix the two run both
// (11 of 32 threads active).  The side is a grouping hint, taken from the
// geometric normal: a vertex's values don't depend on the order.  Material
// divergence, 8.3 M paths: shade 22.8 -> 20.4 ms, sort 0.94 -> 0.99.
// Counting sort in two passes (histogram, scatter); the second pass also
// publishes the segment bounds Q.seg[0..PT_SORT_BINS], by key.
#define PT_BIN_INSIDE 6
__device__ __forceinline__ int sort_bin(int key) { return key + (key >= PT_BIN_INSIDE); }
__device__ __forceinline__ bool hit_front(const PrimShade &ps, float4 hit, float4 ro, float4 rd) {
  const int flags = ps.flags, kind = PT_PRIM_KIND(flags);
  if (flags & PT_PRIM_FACE_FIXED) return (flags & PT_PRIM_FACE_FRONT) != 0;
  const V3 d = v3(rd.x, rd.y, rd.z);
  float c;
  if (kind == ITEM_TRI) {
    c = dot(d, v3(ldf(ps.ng), ldf(ps.ng + 1), ldf(ps.ng + 2)));
  } else if (kind == ITEM_QUAD) {
    const int axis = PT_PRIM_AXIS(flags);
    c = axis == 0 ? d.x : axis == 1 ? d.y : d.z;
  } else if (kind == ITEM_SPHERE) {
    c = dot(d, v3(ro.x - ldf(ps.n0), ro.y - ldf(ps.n0 + 1), ro.z - ldf(ps.n0 + 2)) + normalize(d) * hit.x);
  } else {
    return true;
  }
  return (c < 0.f) != ((flags & PT_PRIM_FLIP) != 0);
}
__device__ __forceinline__ int sort_key(const SceneView &S, const Queues &Q, int qsel, int i) {
  const float4 hit = ld4(Q.hit + i);
  const int prim = __float_as_int(hit.y);
  if (prim == PT_HIT_MEDIUM) return sort_bin(PT_KEY_MEDIUM);
  if (prim < 0) return sort_bin(PT_KEY_MISS);
  const PrimShade &ps = S.shade[prim];
  const int type = S.materials[__ldg(&ps.material)].type;
  if (type == 5) return hit_front(ps, hit, ld4(Q.ray_o[qsel] + i), ld4(Q.ray_d[qsel] + i)) ? 5 : PT_BIN_INSIDE;
  return sort_bin(type);
}
__global__ void k_sort_hist(SceneView S, Queues Q, int qsel) {
  __shared__ int h[PT_SORT_BINS];
  for (int b = threadIdx.x; b < PT_SORT_BINS; b += blockDim.x) h[b] = 0;
  __syncthreads();
  const int n = Q.counts[qsel];
  // the bounce's traversal and the last one's shadow terms are done: counters
  // of the next ray queue, the shadow queue and both fetches
  if (blockIdx.x == 0 && threadIdx.x < 6 && (int)threadIdx.x != qsel) Q.counts[threadIdx.x] = 0;
  const int lane = threadIdx.x & 31;
  const int stride = gridDim.x * blockDim.x;
  const int nround = (n + stride - 1) / stride * stride;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nround; i += stride) {
    const bool act = i < n;
    int key = -1;
    if (act) {
      key = sort_key(S, Q, qsel, i);
      Q.sort_key[i] = key;
    }
    // one shared atomic per (warp, key)
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (act && lane == __ffs(peers) - 1) atomicAdd(&h[key], __popc(peers));
  }
  __syncthreads();
  for (int b = threadIdx.x; b < PT_SORT_BINS; b += blockDim.x)
    if (h[b]) atomicAdd(&Q.bins[b], h[b]);
}
__global__ void k_sort_scatter(Queues Q, int qsel) {
  __shared__ int base[PT_SORT_BINS + 1];
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int b = 0; b < PT_SORT_BINS; ++b) {
      base[b] = acc;
      acc += Q.bins[b];
    }
    base[PT_SORT_BINS] = acc;
    if (blockIdx.x == 0)
      for (int b = 0; b <= PT_SORT_BINS; ++b) Q.seg[b] = base[b < PT_SORT_BINS ? sort_bin(b) : b];
  }
  __syncthreads();
  // per tile of blockDim entries: warp-aggregated ranks in shared memory, one
  // global atomic per (tile, key) to reserve the tile's range of each key
  __shared__ int cnt[PT_SORT_BINS], gbase[PT_SORT_BINS];
  const int n = Q.counts[qsel];
  const int lane = threadIdx.x & 31;
  const int stride = gridDim.x * blockDim.x;
  const int nround = (n + stride - 1) / stride * stride;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nround; i += stride) {
    if (threadIdx.x < PT_SORT_BINS) cnt[threadIdx.x] = 0;
    __syncthreads();
    const bool act = i < n;
    const int key = act ? Q.sort_key[i] : PT_SORT_BINS - 1;
    const unsigned peers = __match_any_sync(0xffffffffu, act ? key : -1);
    const int leader = __ffs(peers) - 1;
    const int rank = __popc(peers & ((1u << lane) - 1u));
    int wbase = 0;
    if (act && lane == leader) wbase = atomicAdd(&cnt[key], __popc(peers));
    wbase = __shfl_sync(0xffffffffu, wbase, leader);
    __syncthreads();
    if (threadIdx.x < PT_SORT_BINS) {
      const int c = cnt[threadIdx.x];
      gbase[threadIdx.x] = c ? atomicAdd(&Q.bins[PT_SORT_BINS + threadIdx.x], c) : 0;
    }
    __syncthreads();
    if (act) Q.order[base[key] + gbase[key] + wbase + rank] = i;
    __syncthreads();
  }
}

// k_trace_shadow, k_shadow_resolve, k_film: their bodies are in pt_wave.cuh
// (trace_shadow_body, shadow_resolve_body, film_body).
template <bool CURVES, bool MOTION>
__global__ void __launch_bounds__(128, CURVES ? 7 : 8) k_trace_shadow(SceneView S, Queues Q) {
  extern __shared__ __align__(16) char smem[];  // trace_smem
  trace_shadow_body<CURVES, MOTION>(S, Q, smem);
}
__global__ void k_shadow_resolve(Queues Q, int LN) { shadow_resolve_body(Q, LN); }
__global__ void k_film(DeviceJob J, Queues Q, long long g0, int n, long long slot0, float *film) {
  film_body(J, Q, g0, n, slot0, film);
}

// Serving: RMSE of a request's mean image estimated from its two
// independent half films A (even passes) and B (odd passes),
// 0.5 * sqrt(mean((A/na - B/nb)^2)), for many requests in one launch.  Fixed
// grid and fixed-order reductions: the estimate, and hence when a request
// stops, does not depend on what else is being served.
__global__ void __launch_bounds__(256) k_film_rmse(const FilmPair *pairs, double *partials) {
  const FilmPair P = pairs[blockIdx.y];
  double acc = 0.0;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < P.n; i += (long long)gridDim.x * 256) {
    double d = (double)P.a[i] * P.ia - (double)P.b[i] * P.ib;
    if (isfinite(d)) acc += d * d;
  }
  __shared__ double sh[256];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partials[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = sh[0];
}
__global__ void k_film_rmse_finish(const FilmPair *pairs, int npairs, int per, const double *partials,
                                   double *out) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npairs; p += gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int k = 0; k < per; ++k) acc += partials[(size_t)p * per + k];
    out[p] = 0.5 * sqrt(acc / (double)pairs[p].n);
  }
}
// a = (a + b) * inv: the mean image of a request from its two half films.
__global__ void k_film_combine(float *a, const float *b, float inv, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    a[i] = (a[i] + b[i]) * inv;
}

// FrameBuffer::gaussianBlur (framebuffer.cpp:60-129): the full k x k kernel
// (weights computed on the host exactly as the reference does) over the film
// with clamp-to-edge, taps summed row-major in the reference's order with
// rounded, never-fused operations, one thread per pixel.
__global__ void k_gaussian_blur(const float *in, float *out, int W, int H, int K, const float *w) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < W * H; p += gridDim.x * blockDim.x) {
    const int i = p / W, j = p % W;  // row, column (row 0 = bottom, as the film)
    float cx = 0.f, cy = 0.f, cz = 0.f;
    for (int s = 0; s < K; ++s) {
      const int ix = min(max(i - K / 2 + s, 0), H - 1);
      for (int t = 0; t < K; ++t) {
        const int iy = min(max(j - K / 2 + t, 0), W - 1);
        const float wt = __ldg(w + s * K + t);
        const float *q = in + 3 * ((size_t)ix * W + iy);
        cx = __fadd_rn(cx, __fmul_rn(__ldg(q), wt));
        cy = __fadd_rn(cy, __fmul_rn(__ldg(q + 1), wt));
        cz = __fadd_rn(cz, __fmul_rn(__ldg(q + 2), wt));
      }
    }
    out[3 * (size_t)p] = cx;
    out[3 * (size_t)p + 1] = cy;
    out[3 * (size_t)p + 2] = cz;
  }
}

// film *= inv: the mean from the sum of a render's samples (the last step of
// pt_render's pixel loop, renderManager.hpp:115).
__global__ void k_film_scale(float *film, float inv, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    film[i] = __fmul_rn(film[i], inv);
}
void launch_film_scale(float *film, float inv, long long n, cudaStream_t st) {
  k_film_scale<<<grid_for(n, 256, 152 * 8), 256, 0, st>>>(film, inv, n);
}

// FrameBuffer::writeToFile pixel path (framebuffer.cpp:27-58).
__global__ void k_tonemap(const float *film, int W, int H, float inv_gamma, uint8_t *out) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < W * H * 3; t += gridDim.x * blockDim.x) {
    int c = t % 3, p = t / 3, i = p % W, j = p / W;
    float v = film[t];
    if (v != v)
      v = 0.f;
    else
      v = powf(v, inv_gamma);
    v = fminf(fmaxf(v, 0.f), 1.f);
    out[((H - 1 - j) * W + i) * 3 + c] = (uint8_t)(v * 255.f);
  }
}

// The tables of first Owen-scrambled digits, one entry per thread (a context's
// creation).
__global__ void k_owen_tables(uint32_t *tables, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int dim = 0;
    while (c_halton.owen_at[dim + 1] <= i) ++dim;
    tables[i] = owen_first_digits(c_halton, dim, i - c_halton.owen_at[dim]);
  }
}
void launch_owen_tables(uint32_t *tables, uint32_t n, cudaStream_t st) {
  k_owen_tables<<<grid_for(n, 256, 152 * 16), 256, 0, st>>>(tables, n);
}

// The curves' segments, one per thread (a scene upload).
__global__ void k_curve_segments(const float4 *curves, int n, float4 *out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n * PT_CURVE_SEGMENTS; i += gridDim.x * blockDim.x) {
    const CurveSegment g = curve_segment(curves + 4 * (size_t)(i / PT_CURVE_SEGMENTS), i % PT_CURVE_SEGMENTS);
    out[2 * (size_t)i] = make_float4(g.pa.x, g.pa.y, g.pa.z, g.radius);
    out[2 * (size_t)i + 1] = make_float4(g.axis.x, g.axis.y, g.axis.z, g.len);
  }
}
void launch_curve_segments(const float4 *curves, int n, float4 *out, cudaStream_t st) {
  k_curve_segments<<<grid_for((long long)n * PT_CURVE_SEGMENTS, 128, 152 * 16), 128, 0, st>>>(curves, n, out);
}

// The traversal's nodes from the built ones, one per thread (a scene upload).
__global__ void k_pack_nodes(const Bvh4Node *nodes, int n, PackedNode *out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = pack_node(nodes[i]);
}

// ---------------------------------------------------------------- launchers
void launch_pack_nodes(const Bvh4Node *nodes, int n, PackedNode *out, cudaStream_t st) {
  k_pack_nodes<<<grid_for(n, 128, 152 * 16), 128, 0, st>>>(nodes, n, out);
}

void upload_halton_tables(const HaltonTables &T, cudaStream_t st) {
  cudaMemcpyToSymbolAsync(c_halton, &T, sizeof(T), 0, cudaMemcpyHostToDevice, st);
}


void launch_sampler_eval(int strategy, const uint16_t *perm, uint32_t first, int n, int dims,
                         float *out, cudaStream_t st) {
  long long tot = (long long)n * dims;
  k_sampler_eval<<<grid_for((int)std::min<long long>(tot, 1 << 30), 256, 152 * 16), 256, 0, st>>>(
      strategy, perm, first, n, dims, out);
}

void launch_trace_test(const SceneView &S, bool any, const float *rays, const float *tmaxs, int n,
                       float tmin, float tmax, float *t, int *prim, float *uv, uint8_t *occ, FetchPair fetch, int *err,
                       cudaStream_t st) {
  const int g = query_grid(n);
#define PT_RUN(C, M)                                                                                             \
  if (any)                                                                                                       \
    k_trace_test<true, C, M><<<g, 128, trace_smem(128, true, M), st>>>(S, rays, tmaxs, n, tmin, tmax, t, prim, uv, \
                                                                       occ, fetch, err);                         \
  else                                                                                                           \
    k_trace_test<false, C, M><<<g, 128, trace_smem(128, false, M), st>>>(S, rays, tmaxs, n, tmin, tmax, t, prim, uv, occ, \
                                                                  fetch, err)
  if (S.curves) {
    PT_RUN(true, true);
  } else if (S.has_motion) {
    PT_RUN(false, true);
  } else {
    PT_RUN(false, false);
  }
#undef PT_RUN
}

void launch_bsdf_eval(const MatRec *m, int n, const float *wo, const float *wi, const float *nrm,
                      const uint8_t *front, float *f, float *pdf, cudaStream_t st) {
  k_bsdf_eval<<<grid_for(n, 128, 152 * 8), 128, 0, st>>>(m, n, wo, wi, nrm, front, f, pdf);
}
void launch_bsdf_sample(const MatRec *m, int n, const float *wo, const float *nrm,
                        const uint8_t *front, const float *uc, const float *u, uint8_t *ok,
                        float *wi, float *att, float *pdf, uint32_t *type, cudaStream_t st) {
  k_bsdf_sample<<<grid_for(n, 128, 152 * 8), 128, 0, st>>>(m, n, wo, nrm, front, uc, u, ok, wi, att,
                                                          pdf, type);
}

// One wave of a single job: camera, max_depth (+1 for MIS) bounces, film.
void launch_wave(const SceneView &S, const DeviceJob &J, const Queues &Q, long long g0, int n,
                 float *film, const LaunchCfg &cfg, cudaStream_t st, Profiler *prof, cudaEvent_t film_after,
                 cudaEvent_t film_done, const ShadeStreams *ss) {
  const int LN = J.job.light_nx * J.job.light_ny;
  const int bounces = J.job.max_depth + (J.job.estimator == PT_EST_NEE_MIS ? 1 : 0);
  Profiler dummy;
  Profiler &P = prof ? *prof : dummy;
  const JobTable none{nullptr, nullptr, 0};
  launch_wave_stages<false>(S, J, none, Q, g0, n, LN, bounces, cfg, st, P, ss);
  if (film_after) cudaStreamWaitEvent(st, film_after, 0);
  P.begin(STAGE_FILM, st);
  launch_film(J, Q, g0, n, 0, film, cfg, st);
  P.end(st);
  P.count(STAGE_FILM, 1);
  if (film_done) cudaEventRecord(film_done, st);
}

void launch_sort(const SceneView &S, const Queues &Q, int qsel, const LaunchCfg &cfg, cudaStream_t st) {
  k_sort_hist<<<cfg.max_blocks_simple, 256, 0, st>>>(S, Q, qsel);
  k_sort_scatter<<<cfg.max_blocks_simple, 256, 0, st>>>(Q, qsel);
}

void launch_shadow(const SceneView &S, const Queues &Q, int LN, const LaunchCfg &cfg, cudaStream_t st) {
#define PT_RUN(C, M) k_trace_shadow<C, M><<<cfg.trace_blocks, 128, trace_smem(128, true, M), st>>>(S, Q)
  PT_BY_SCENE(S, PT_RUN);
#undef PT_RUN
  k_shadow_resolve<<<cfg.max_blocks_simple, 256, 0, st>>>(Q, LN);
}
void launch_shadow_resolve(const Queues &Q, int LN, const LaunchCfg &cfg, cudaStream_t st) {
  k_shadow_resolve<<<cfg.max_blocks_simple, 256, 0, st>>>(Q, LN);
}

void launch_film(const DeviceJob &J, const Queues &Q, long long lo, int cnt, long long slot0, float *film,
                 const LaunchCfg &cfg, cudaStream_t st) {
  k_film<<<grid_for(std::min<long long>((long long)J.job.width * J.job.height, 1 << 30), 256,
                    cfg.max_blocks_simple),
           256, 0, st>>>(J, Q, lo, cnt, slot0, film);
}

void launch_film_rmse(const FilmPair *pairs, int npairs, double *partials, double *out, cudaStream_t st) {
  if (npairs <= 0) return;
  k_film_rmse<<<dim3(PT_RMSE_BLOCKS, npairs), 256, 0, st>>>(pairs, partials);
  k_film_rmse_finish<<<grid_for(npairs, 128, 152), 128, 0, st>>>(pairs, npairs, PT_RMSE_BLOCKS, partials, out);
}
void launch_film_combine(float *a, const float *b, float inv, long long n, cudaStream_t st) {
  k_film_combine<<<grid_for((int)std::min<long long>(n, 1 << 30), 256, 152 * 8), 256, 0, st>>>(a, b, inv, n);
}

void launch_gaussian_blur(const float *in, float *out, int W, int H, int K, const float *w, cudaStream_t st) {
  k_gaussian_blur<<<grid_for((long long)W * H, 128, 152 * 16), 128, 0, st>>>(in, out, W, H, K, w);
}

void launch_tonemap(const float *film, int W, int H, float gamma, uint8_t *out, cudaStream_t st) {
  k_tonemap<<<grid_for(W * H * 3, 256, 152 * 8), 256, 0, st>>>(film, W, H, 1.f / gamma, out);
}

void kernel_attributes(KernelInfo *info) {
  cudaFuncAttributes a;
  cudaFuncGetAttributes(&a, k_trace_closest<false, false, false>);
  info->trace_regs = a.numRegs;
  cudaFuncGetAttributes(&a, k_shade<-1, false>);
  info->shade_regs = a.numRegs;
  int nb = 0;
  const size_t smax = trace_smem(128);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trace_closest<false, false, false>, 128, smax);
  info->trace_blocks_per_sm = nb;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_shade<-1, false>, 128, 0);
  info->shade_blocks_per_sm = nb;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trace_shadow<false, false>, 128, smax);
  info->shadow_blocks_per_sm = nb;
  int *fb = info->shade_fam_blocks_per_sm;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fb[0], k_shade<0, false>, shade_threads(0), 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fb[1], k_shade<1, false>, shade_threads(1), 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fb[2], k_shade<2, false>, shade_threads(2), 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fb[3], k_shade<3, false>, shade_threads(3), 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fb[4], k_shade<4, false>, shade_threads(4), 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fb[5], k_shade<5, false>, shade_threads(5), 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fb[6], k_shade<6, false>, shade_threads(6), 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fb[PT_FAM_MISC], k_shade<PT_FAM_MISC, false>, shade_threads(PT_FAM_MISC), 0);
  fb[PT_FAM_MISC + 1] = info->shade_blocks_per_sm;
}

}  // namespace pt
