// gt_trace_common.cuh — pieces shared by the trace kernels: per-ray
// statistics, the box-test ray, the exact ray/proxy test and work helpers.
#pragma once

#include <math_constants.h>

#include "gt_device.cuh"
#include "gt_internal.cuh"

namespace gt {

constexpr int kTileW = 8, kTileH = 4;
constexpr uint32_t kTileBlock = 16;  // tiles per side of a tile block

// Pixel of position s (0..31) in tile lt of a view.  Tiles go in blocks of
// 16 x 16 (128 x 64 pixels), blocks row-major, tiles in Morton order inside a
// block, so that the tiles in flight at any time cover a compact patch of
// the image (1 % faster than row-major tiles on the 1M-Gaussian view).  The
// view's tile grid is padded to whole blocks; pixels past the image edge are
// skipped.
__device__ __forceinline__ void tile_pixel(uint32_t tiles_x, uint32_t lt, uint32_t s, uint32_t& px, uint32_t& py) {
  const uint32_t blk = lt >> 8, in = lt & 255u;
  const uint32_t bpr = tiles_x / kTileBlock;  // blocks per row
  const uint32_t bx = blk % bpr, by = blk / bpr;
  uint32_t mx = in & 0x55u, my = (in >> 1) & 0x55u;  // de-interleave the 8-bit Morton code
  mx = (mx | (mx >> 1)) & 0x33u;
  mx = (mx | (mx >> 2)) & 0x0Fu;
  my = (my | (my >> 1)) & 0x33u;
  my = (my | (my >> 2)) & 0x0Fu;
  px = (bx * kTileBlock + mx) * kTileW + (s % kTileW);
  py = (by * kTileBlock + my) * kTileH + (s / kTileW);
}

// Work counters of one warp, kept in its shared scratch (not in registers)
// and updated by lane 0 with warp totals.
struct RayStats {
  unsigned long long rounds, entries, contributing, proxy_tests, node_visits, anyhits;
};

// Box-test state of a ray: inverse direction, origin times inverse direction
// and, per axis, a padding of the slab planes that covers the rounding of
// the object-space triangle test (hit points lie within ~1e-6 relative of
// |origin| + scene size of the true surface).
struct BoxRay {
  float ix, iy, iz, ox, oy, oz, px, py, pz;
};

__device__ __forceinline__ float safe_inv(float d) {
  float a = fabsf(d) < 1e-30f ? copysignf(1e-30f, d) : d;
  return __frcp_rn(a);
}

__device__ __forceinline__ BoxRay make_boxray(V3 o, V3 d, float scene_mag) {
  BoxRay b;
  b.ix = safe_inv(d.x);
  b.iy = safe_inv(d.y);
  b.iz = safe_inv(d.z);
  b.ox = o.x * b.ix;
  b.oy = o.y * b.iy;
  b.oz = o.z * b.iz;
  float m = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fabsf(o.z));
  float pad = 4e-6f * (m + scene_mag) + 1e-7f;
  b.px = pad * fabsf(b.ix);
  b.py = pad * fabsf(b.iy);
  b.pz = pad * fabsf(b.iz);
  return b;
}

// The icosahedron's faces in shared memory, for lanes that test different faces
// (a kernel parameter serves one address at a time): (n, p0.x), (p0.yz, e1.xy),
// (e1.z, e0).  Row q is face pa[q] of pair q, row 10 + q its antipode pb[q].
struct FaceRows {
  float4 row[20][3];
};
// Fills the rows (lane of a warp; the caller synchronises).
__device__ __forceinline__ void load_face_rows(const FaceTable& F, FaceRows& S, uint32_t lane) {
  if (lane >= 20) return;
  const int f = lane < 10 ? F.pa[lane] : F.pb[lane - 10];
  const float *n = F.n[f], *p = F.p0[f], *e1 = F.e1[f], *e0 = F.e0[f];
  S.row[lane][0] = make_float4(n[0], n[1], n[2], p[0]);
  S.row[lane][1] = make_float4(p[1], p[2], e1[0], e1[1]);
  S.row[lane][2] = make_float4(e1[2], e0[0], e0[1], e0[2]);
}

// The bounding-sphere filter of a proxy: false only when the ray certainly
// misses proxy j.  Every triangle lies inside the circumsphere, and the
// triangle test cannot report a point farther than its rounding error (covered
// by the 1e-3 + 1e-5 |o_obj| margin) from its triangle.
__device__ __forceinline__ bool proxy_sphere(const FaceTable& F, const float4* w2o, uint32_t j, V3 o, V3 d) {
  Affine W = load_affine(w2o + 3 * (size_t)j);
  V3 oo = xpoint(W, o), od = xdir(W, d);
  float l1o = fabsf(oo.x) + fabsf(oo.y) + fabsf(oo.z);
  float dd = __fmaf_rn(od.x, od.x, __fmaf_rn(od.y, od.y, od.z * od.z));
  float ox = __fmaf_rn(oo.x, od.x, __fmaf_rn(oo.y, od.y, oo.z * od.z));
  float tc = -__fdividef(ox, dd);
  float cx = __fmaf_rn(tc, od.x, oo.x), cy = __fmaf_rn(tc, od.y, oo.y), cz = __fmaf_rn(tc, od.z, oo.z);
  float r2 = __fmaf_rn(cx, cx, __fmaf_rn(cy, cy, cz * cz));
  float rp = __fmaf_rn(1e-5f, l1o, F.r_circ + 1e-3f);
  return (r2 <= rp * rp) || !(dd == dd && r2 == r2);
}

// The faces of proxy j that the reference triangle test hits with t in (tlo,
// thi), whatever their facing (debugMode 1), as calls on_hit(t, face).
template <class OnHit>
__device__ __forceinline__ void proxy_any_face(const FaceTable& F, const float4* w2o, uint32_t j, V3 o, V3 d, float tlo,
                                               float thi, OnHit&& on_hit) {
  const Affine W = load_affine(w2o + 3 * (size_t)j);
  const V3 oo = xpoint(W, o), od = xdir(W, d);
#pragma unroll 1
  for (int f = 0; f < 20; ++f) {
    float dn = vdot(mk(F.n[f][0], F.n[f][1], F.n[f][2]), od);
    float t;
    if (tri_test(F, f, oo, tlo, od, thi, dn, t)) on_hit(t, f);
  }
}

// n_q . v of the ten pairs' normals, up to rounding.
__device__ __forceinline__ void pair_dots(const FaceTable& F, V3 v, float out[10]) {
  const float a = F.na, b = F.nb, c = F.nc;
  const float ax = a * v.x, ay = a * v.y, az = a * v.z;
  const float s = ay + ax, t = ay - ax;
  out[0] = t + az;
  out[3] = t - az;
  out[5] = s + az;
  out[9] = s - az;
  const float by = b * v.y, bx = b * v.x, bz = b * v.z;
  out[1] = __fmaf_rn(c, v.z, by);
  out[2] = __fmaf_rn(-c, v.z, by);
  out[4] = __fmaf_rn(c, v.y, -bx);
  out[7] = __fmaf_rn(-c, v.y, -bx);
  out[6] = __fmaf_rn(-c, v.x, bz);
  out[8] = __fmaf_rn(-c, v.x, -bz);
}

// The front-face hits of proxy j: calls on_hit(t, row) for every face that the
// reference triangle test hits with t in (tlo, thi) and that faces the ray.
// Two exact filters run before that test; each skips only work whose outcome
// is already known:
//   * facing: dot(n, d_obj) and the reference's world-space facing product
//     both approximate n^T W2O d within tau = 1e-5 * nmax * sum(|W2O||d|), so
//     a face whose dot(n, d_obj) exceeds tau is back-facing, and one below
//     -tau is front-facing (the product is within 12 u nmax s of it, u =
//     2^-24); only faces in between need the product computed;
//   * candidate faces.  For front faces e, f (dn < -tau) with plane crossings
//     t_e >= t_f, the ray at t_f lies outside plane e by (t_e - t_f)|dn_e|/|n|
//     while triangle f lies inside it (the proxy is convex), so the crossing
//     X_f is at least that far from triangle f.  The reference's triangle test
//     accepts points only within its rounding of the triangle, about
//     10 u |od| |p0 - oo| / |dn_f| in barycentric units.  Hence a face can pass
//     only if (t_e - t_f) |dn_e| |dn_f| stays below a few tens of u |od|_1
//     (|oo|_1 + 2); faces above 128 u times that are skipped (a CPU check of
//     4e7 adversarial rays, edges, vertices and grazing faces, found the first
//     misses below 8, which leaves room for the approximate reciprocals here).
// The faces are planes n . x = c in antipodal pairs (n_b == -n_a bit for bit),
// so the ray enters pair q's slab at t_q = -(c + s n_q . o) / |n_q . d|, s =
// sign(n_q . d): one pass finds the latest entry, a second the faces within
// the bound of it.  All planes have the same c, and the normals are (+-a, +-a,
// +-a) and the cyclic (0, +-b, +-c') (make_face_table; checked when a context is
// created), so the ten products with a vector share their terms: 18 operations
// instead of 30.  1080p, 1M Gaussians, list tracer: 17.1 -> 14.2 ms against a
// single pass with products instead of reciprocals, t-range prefilters and the
// faces in kernel parameters, and 9.50 -> 9.26 ms (960x540: 3.41 -> 3.35) with
// the shared terms and the faces chosen by pair.
template <class OnHit>
__device__ __forceinline__ void proxy_faces(const FaceTable& F, const FaceRows& S, const float4* w2o, uint32_t j, V3 o,
                                            V3 d, float tlo, float thi, OnHit&& on_hit) {
  const Affine W = load_affine(w2o + 3 * (size_t)j);
  const V3 oo = xpoint(W, o), od = xdir(W, d);
  const float l1o = fabsf(oo.x) + fabsf(oo.y) + fabsf(oo.z);
  const float* m = W.m;
  const float s = fabsf(d.x) * (fabsf(m[0]) + fabsf(m[1]) + fabsf(m[2])) +
                  fabsf(d.y) * (fabsf(m[3]) + fabsf(m[4]) + fabsf(m[5])) +
                  fabsf(d.z) * (fabsf(m[6]) + fabsf(m[7]) + fabsf(m[8]));
  const float tau = 1e-5f * F.nmax * s;
  const float gbound = 7.62939453125e-6f * (fabsf(od.x) + fabsf(od.y) + fabsf(od.z)) * (l1o + 2.0f);
  float dn[10], num[10];
  pair_dots(F, od, dn);
  pair_dots(F, oo, num);
  float te = -CUDART_INF_F, re = 0.0f, least = CUDART_INF_F;
#pragma unroll
  for (int q = 0; q < 10; ++q) {
    // distance of the origin in front of the pair's front face: -(c + s n.o)
    num[q] = -__uint_as_float(__float_as_uint(num[q]) ^ (__float_as_uint(dn[q]) & 0x80000000u)) - F.plane;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fabsf(dn[q])));
    const float t = num[q] * r;
    if (t > te) {
      te = t;
      re = r;
    }
    least = fminf(least, fabsf(dn[q]));
  }
  // the pairs to test: the front face of each, or both faces of every pair
  // when some pair grazes the ray
  uint32_t cand = 0x3FFu;
  const bool both = !(least > 1.01f * tau && te < 1e30f);
  if (!both) {
    const float slack = gbound * re;
    cand = 0;
#pragma unroll
    for (int q = 0; q < 10; ++q)
      if (!(__fmaf_rn(te, fabsf(dn[q]), -num[q]) > slack)) cand |= 1u << q;
  }
  int row = -1;  // the antipode still to test (both)
#pragma unroll 1
  while (cand || row >= 0) {
    float4 a;
    float dnf;
    if (row >= 0) {
      a = S.row[row][0];
      dnf = vdot(mk(a.x, a.y, a.z), od);
    } else {
      row = __ffs(cand) - 1;
      cand &= cand - 1;
      a = S.row[row][0];
      dnf = vdot(mk(a.x, a.y, a.z), od);
      if (!both && dnf >= 0.0f) {  // the antipode is the front face: n and dn change sign exactly
        row += 10;
        dnf = -dnf;
        a = S.row[row][0];
      }
    }
    const float4 b = S.row[row][1], c = S.row[row][2];
    const int f = row;
    row = both && row < 10 ? row + 10 : -1;
    // tri_test
    const V3 n = mk(a.x, a.y, a.z);
    const float r = __frcp_rn(dnf);
    const V3 e2 = vscale(r, vsub(mk(a.w, b.x, b.y), oo));
    const float t = vdot(n, e2);
    if (t <= tlo || thi <= t || t != t) continue;
    const V3 i = vcross(od, e2);
    const float beta = vdot(i, mk(b.z, b.w, c.x)), gamma = vdot(i, mk(c.y, c.z, c.w));
    if (!(beta >= 0.0f && gamma >= 0.0f && beta + gamma <= 1.0f)) continue;
    if (fabsf(dnf) > tau ? dnf < 0.0f : front_facing(n, load_affine(w2o + 3 * (size_t)j), d)) on_hit(t, f);
  }
}

// next float above x: the far bound of the triangle test that still admits
// a tie with the k-th hit
__device__ __forceinline__ float next_up(float x) { return nextafterf(x, CUDART_INF_F); }

// Adds a warp's counters to the launch totals.  `rays` is counted by lane 0;
// `st` is the warp's shared counter block.
__device__ __forceinline__ void flush_stats(DevCounters* ctr, const RayStats& st, uint32_t rays, uint32_t status) {
  uint32_t s = __reduce_or_sync(0xFFFFFFFFu, status);
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&ctr->rays, (unsigned long long)rays);
    atomicAdd(&ctr->rounds, st.rounds);
    atomicAdd(&ctr->entries, st.entries);
    atomicAdd(&ctr->contributing, st.contributing);
    atomicAdd(&ctr->proxy_tests, st.proxy_tests);
    atomicAdd(&ctr->node_visits, st.node_visits);
    atomicAdd(&ctr->anyhits, st.anyhits);
    if (s) atomicOr(&ctr->status, s);
  }
}

__device__ __forceinline__ uint32_t find_view(const ViewDev* views, uint32_t n_views, uint32_t tile) {
  uint32_t lo = 0, hi = n_views - 1;
  while (lo < hi) {
    uint32_t mid = (lo + hi + 1) >> 1;
    if (views[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
  }
  return lo;
}

}  // namespace gt
