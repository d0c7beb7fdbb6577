// gt_stream.cu — forward tracer over per-view proxy lists (the default for
// plain and checkpointing renders).
//
// All primary rays of a view start at the camera, so a view needs no
// hierarchy: each proxy is projected once, entered into the list of every
// image bin its outline may touch, ordered by a lower bound of the distance
// at which a ray can enter it, and a bin's tiles then stream through that
// list front to back.  Same output as k_trace8 and k_trace_packet bit for
// bit: the exact proxy test, the rounds and the compositing arithmetic are
// the same; the lists only decide which (proxy, ray) pairs are tested, and
// they leave out none that could hit.
//
// Lists (k_list_project, k_list_pass, k_list_rows, k_list_bins):
//   * a proxy lies inside its circumscribed ellipsoid, whose outline seen
//     from the camera is an ellipse in the image plane (u, v) of the camera
//     frame.  The projection is done in double from the world-to-object map
//     and origin the exact test uses, and the ellipse is grown by the test's
//     rounding reach (the bounding-sphere margin) and by 2e-6 (1 + |u| + |v|)
//     in the image plane for the rounding of a ray's (u, v).  One that reaches
//     the camera plane has no ellipse but bounds of u and v (side_range), open on
//     one side or, where it surrounds the camera, on both; every ray within them
//     tests it (a sphere test first saved nothing and cost other views 2 %).
//     Entered in every bin and tested by every ray, such proxies (17k of 1M
//     Gaussians in clusters seen from their middle) took 840 ms of a 1080p view
//     that takes 6.8 ms so;
//   * every point of it is at least |c| - h from the camera (c its centre, h
//     its extent along c): the bound by which lists are ordered, taken 1e-4
//     lower for the rounding of t.  Order within a list is by bucket of that
//     bound's float bits: a counting sort of (bin, bucket) cells, whose
//     order inside a cell is arbitrary and does not show in the results.
//
// Trace (k_trace_stream): a warp takes the rays of an 8x4 tile, one a lane
// (small views: a quarter of it).  32 list entries at a time are tested
// against the tile's (u, v) range; for those that overlap it, every ray
// tests the outline ellipse; the rays inside become (proxy, ray) pairs that
// go through the exact face tests 32 at a time.  A ray's hits wait in a
// 4-ary min-heap in shared memory; a hit is final once its t is below the
// bound of everything not tested yet, and final hits are composited in order
// (t, particle), in rounds of k exactly as the other kernels do.  Each pair
// is tested once, where the hierarchy kernels start over for every kbuf hits
// of a ray (1M Gaussians at 1080p: 305 sphere tests and about 180 face tests
// a ray there).
//   * A ray whose heap overflows, or that receives a hit below the bound it
//     has already composited to (possible only through rounding past the
//     margins above), goes back to the start of its round and is handed to
//     the warp-per-ray kernel; so are a tile's rays once every tile of the
//     launch is taken and the tile has composited some hits (the launch's
//     end would wait on them), and all rays of a bin whose list did not fit.
#include <math_constants.h>

#include <math.h>

#include <algorithm>

#include "gt_device.cuh"
#include "gt_internal.cuh"
#include "gt_trace_common.cuh"
#include "gt_warp.cuh"

namespace gt {

// ------------------------------------------------------------------ lists
// Bin of bin coordinates (bx, by) in a view: bins are 2^s x 2^s tiles (s =
// shift / 2) and numbered like the tiles (tile_pixel: blocks of 16 x 16 tiles
// row by row, Morton order inside), so that bin = tile >> shift.
__device__ __forceinline__ uint32_t bin_index(uint32_t bx, uint32_t by, uint32_t shift, uint32_t bpr) {
  const uint32_t s = shift >> 1;
  const uint32_t tx = bx << s, ty = by << s;
  uint32_t mx = tx & 15u, my = ty & 15u;
  mx = (mx | (mx << 2)) & 0x33u;
  mx = (mx | (mx << 1)) & 0x55u;
  my = (my | (my << 2)) & 0x33u;
  my = (my | (my << 1)) & 0x55u;
  const uint32_t lt = (((ty >> 4) * bpr + (tx >> 4)) << 8) | mx | (my << 1);
  return lt >> shift;
}

// Distance buckets of a view: bound bits (floats >= 0 order like their bits)
// between the view's smallest and largest, in equal steps.
struct Buckets {
  uint32_t lo;
  double per_bit, width;
};
__device__ __forceinline__ Buckets make_buckets(uint32_t bmin, uint32_t bmax) {
  Buckets b;
  b.lo = bmin;
  b.width = (double)(bmax - bmin + 1u) * (1.0 / (1 << kListBucketBits));
  b.per_bit = 1.0 / b.width;
  return b;
}
__device__ __forceinline__ uint32_t bucket_of(const Buckets& b, uint32_t bits) {
  return min((uint32_t)((double)(bits - b.lo) * b.per_bit), (1u << kListBucketBits) - 1u);
}
// A value no larger than any bound of the bucket.
__device__ __forceinline__ uint32_t bucket_edge(const Buckets& b, uint32_t bucket) {
  const uint32_t e = (uint32_t)((double)bucket * b.width);
  return b.lo + (e > 0u ? e - 1u : 0u);
}

// The camera frame and bin grid of every view, and an empty bound range.
__global__ void k_list_views(const ViewDev* __restrict__ views, uint32_t n_views, ListView* __restrict__ lviews,
                             const Lists L) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_views) return;
  const ViewDev& V = views[i];
  ListView P;
  double nx = 0.0, ny = 0.0, nz = 0.0;
  for (int a = 0; a < 3; ++a) {
    P.X[a] = -(double)V.u.tw[a];
    P.Y[a] = (double)V.u.tw[4 + a];
    P.Z[a] = -(double)V.u.tw[8 + a];
    nx += P.X[a] * P.X[a];
    ny += P.Y[a] * P.Y[a];
    nz += P.Z[a] * P.Z[a];
  }
  nx = sqrt(nx);
  ny = sqrt(ny);
  nz = sqrt(nz);
  for (int a = 0; a < 3; ++a) {
    P.X[a] /= nx;
    P.Y[a] /= ny;
    P.Z[a] /= nz;
    P.Xf[a] = (float)P.X[a];
    P.Yf[a] = (float)P.Y[a];
    P.Zf[a] = (float)P.Z[a];
  }
  // ray_gen: u = (2 (px + 1/2) / w - 1) asp_x |cx| / |cz|, and so on
  P.sx = 0.5 * V.w * nz / ((double)V.u.asp[0] * nx);
  P.sy = 0.5 * V.h * nz / ((double)V.u.asp[1] * ny);
  P.ox = 0.5 * V.w;
  P.oy = 0.5 * V.h;
  P.reach = 1.0 + P.ox / P.sx + P.oy / P.sy;
  const uint32_t s = L.shift >> 1;
  P.inv_bw = 1.0 / (double)((uint32_t)kTileW << s);
  P.inv_bh = 1.0 / (double)((uint32_t)kTileH << s);
  P.bins_x = (V.w + ((uint32_t)kTileW << s) - 1) / ((uint32_t)kTileW << s);
  P.bins_y = (V.h + ((uint32_t)kTileH << s) - 1) / ((uint32_t)kTileH << s);
  P.bin_begin = V.tile_begin >> L.shift;
  P.rec_begin = V.rec_begin;
  lviews[i] = P;
  L.range[2 * i] = 0xFFFFFFFFu;
  L.range[2 * i + 1] = 0u;
}

// Bounds of u = x / z over the rays that meet an ellipsoid which reaches the
// camera plane z = 0 (v from the y terms): centre (cx, ., cz), shape E, D = cz^2 -
// Ezz.  It lies on one side of the plane x = u z where f(u) = cx - u cz is larger
// in size than the root of Exx - 2 u Exz + u^2 Ezz, so the ends are roots of
// D u^2 - 2 (cx cz - Exz) u + cx^2 - Exx.  With D > 0 (it stays in front) the range
// lies between them.  With D < 0 it lies on one side of all planes between them:
// f < 0 there keeps only the u below both, f > 0 those above; without roots it
// surrounds the camera in this section, and any u is possible.  (Widened for the
// rounding of a ray's u by about reach, 1 and the largest |u| and |v| of the view.)
__device__ __forceinline__ void side_range(double cx, double cz, double Exx, double Exz, double D, double reach,
                                           double& lo, double& hi) {
  const double b = cx * cz - Exz, c = cx * cx - Exx, disc = b * b - D * c;
  if (!(disc > 0.0)) return;
  const double q = b + copysign(sqrt(disc), b);
  const double ra = q / D, rb = c / q;  // (D near 0: ra far out, rb exact)
  const double r0 = fmin(ra, rb), r1 = fmax(ra, rb);
  if (D > 0.0) {
    lo = r0;
    hi = r1;
  } else if (D < 0.0) {
    const double f = cx - b / D * cz;
    if (f < 0.0) hi = r0;
    if (f > 0.0) lo = r1;
  }
  lo -= 2e-6 * reach * (1.0 + fabs(lo));
  hi += 2e-6 * reach * (1.0 + fabs(hi));
}

// Projection of every proxy of every view (grid.y): outline ellipse, its
// bounding rectangle, distance bound and bins; a view's smallest and largest
// bound.  Bound by its double arithmetic and 96 bytes of traffic a proxy.
__global__ void __launch_bounds__(128) k_list_project(const ViewDev* __restrict__ views,
                                                      const ListView* __restrict__ lviews, float r_circ,
                                                      const Lists L) {
  const ViewDev& V = views[blockIdx.y];
  const ListView& P = lviews[blockIdx.y];
  uint32_t key_lo = 0xFFFFFFFFu, key_hi = 0u;
  // (a grid-stride loop: a launch captured in a batch graph serves later
  // batches of the same shape whose scenes hold more proxies)
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < V.s.n_kept; j += gridDim.x * blockDim.x) {
    const Affine W = load_affine(V.s.w2o + 3 * (size_t)j);
    const V3 oo = xpoint(W, mk(V.u.tw[12], V.u.tw[13], V.u.tw[14]));
    const float l1o = fabsf(oo.x) + fabsf(oo.y) + fabsf(oo.z);
    const double rp = (double)r_circ + 1e-3 + 1e-5 * (double)l1o;
    // object to world (rows), then to the camera frame
    const double a0 = W.m[0], a1 = W.m[1], a2 = W.m[2], b0 = W.m[3], b1 = W.m[4], b2 = W.m[5], c0 = W.m[6],
                 c1 = W.m[7], c2 = W.m[8];
    double r[3][3] = {{b1 * c2 - b2 * c1, b2 * c0 - b0 * c2, b0 * c1 - b1 * c0},
                      {c1 * a2 - c2 * a1, c2 * a0 - c0 * a2, c0 * a1 - c1 * a0},
                      {a1 * b2 - a2 * b1, a2 * b0 - a0 * b2, a0 * b1 - a1 * b0}};
    const double inv_det = 1.0 / (a0 * r[0][0] + a1 * r[0][1] + a2 * r[0][2]);
    double M[3][3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double c = inv_det * rp;
      M[0][q] = c * (P.X[0] * r[0][q] + P.X[1] * r[1][q] + P.X[2] * r[2][q]);
      M[1][q] = c * (P.Y[0] * r[0][q] + P.Y[1] * r[1][q] + P.Y[2] * r[2][q]);
      M[2][q] = c * (P.Z[0] * r[0][q] + P.Z[1] * r[1][q] + P.Z[2] * r[2][q]);
    }
    const double ox = oo.x / rp, oy = oo.y / rp, oz = oo.z / rp;
    const double cx = -(M[0][0] * ox + M[0][1] * oy + M[0][2] * oz);
    const double cy = -(M[1][0] * ox + M[1][1] * oy + M[1][2] * oz);
    const double cz = -(M[2][0] * ox + M[2][1] * oy + M[2][2] * oz);
    const double Exx = M[0][0] * M[0][0] + M[0][1] * M[0][1] + M[0][2] * M[0][2];
    const double Exy = M[0][0] * M[1][0] + M[0][1] * M[1][1] + M[0][2] * M[1][2];
    const double Exz = M[0][0] * M[2][0] + M[0][1] * M[2][1] + M[0][2] * M[2][2];
    const double Eyy = M[1][0] * M[1][0] + M[1][1] * M[1][1] + M[1][2] * M[1][2];
    const double Eyz = M[1][0] * M[2][0] + M[1][1] * M[2][1] + M[1][2] * M[2][2];
    const double Ezz = M[2][0] * M[2][0] + M[2][1] * M[2][1] + M[2][2] * M[2][2];
    // distance bound
    const double dist2 = cx * cx + cy * cy + cz * cz;
    const double hc2 = (Exx * cx * cx + Eyy * cy * cy + Ezz * cz * cz +
                        2.0 * (Exy * cx * cy + Exz * cx * cz + Eyz * cy * cz)) / dist2;
    const double tb = sqrt(dist2) - sqrt(hc2);
    const float tbf = tb > 0.0 ? __double2float_rd(tb * (1.0 - 1e-4)) : 0.0f;  // (NaN: 0)
    // outline: dual conic E - c c^T, as centre (u0, v0) and covariance S
    float4 rec0 = make_float4(0.f, 0.f, 0.f, 0.f), rec1 = make_float4(0.f, tbf, 0.f, 0.f);
    float4 bb = make_float4(-CUDART_INF_F, CUDART_INF_F, -CUDART_INF_F, CUDART_INF_F);
    bool visible = true;
    uint32_t bx0 = 0, bx1 = P.bins_x - 1, by0 = 0, by1 = P.bins_y - 1;
    const double D = cz * cz - Ezz;
    double ulo = -CUDART_INF, uhi = CUDART_INF, vlo = -CUDART_INF, vhi = CUDART_INF;
    if (cz > 0.0 && D > 1e-4 * cz * cz) {
      const double iD = 1.0 / D;
      const double u0 = (cx * cz - Exz) * iD, v0 = (cy * cz - Eyz) * iD;
      double Sxx = (Exx - cx * cx) * iD + u0 * u0, Sxy = (Exy - cx * cy) * iD + u0 * v0,
             Syy = (Eyy - cy * cy) * iD + v0 * v0;
      const double eps = 2e-6 * (1.0 + fabs(u0) + fabs(v0) + sqrt(fmax(Sxx, 0.0)) + sqrt(fmax(Syy, 0.0)));
      // (1 + a) S + (1 + 1/a) eps^2 I contains the eps neighbourhood of S's ellipse
      Sxx = 1.02 * Sxx + 51.0 * eps * eps;
      Syy = 1.02 * Syy + 51.0 * eps * eps;
      Sxy = 1.02 * Sxy;
      const double det = Sxx * Syy - Sxy * Sxy;
      if (Sxx > 0.0 && Syy > 0.0 && det > 0.0 && Sxx < 1e30 && Syy < 1e30) {
        const double hw = sqrt(Sxx), hh = sqrt(Syy);
        rec0 = make_float4((float)u0, (float)v0, (float)(-Sxy / Syy), (float)sqrt(Syy / det));
        rec1.x = (float)(1.0 / hh);
        ulo = u0 - hw - eps;
        uhi = u0 + hw + eps;
        vlo = v0 - hh - eps;
        vhi = v0 + hh + eps;
      }
    } else if (cz + sqrt(Ezz) <= 0.0) {
      visible = false;  // behind the camera plane
    } else {
      // The ellipsoid reaches the camera plane, or nearly: no ellipse (rec0 = 0
      // passes every ray), but bounds of u and v.
      side_range(cx, cz, Exx, Exz, D, P.reach, ulo, uhi);
      side_range(cy, cz, Eyy, Eyz, D, P.reach, vlo, vhi);
    }
    // (values that are not finite leave the bounds open: every ray of every bin)
    if (visible) {
      bb = make_float4(__double2float_rd(ulo), __double2float_ru(uhi), __double2float_rd(vlo),
                       __double2float_ru(vhi));
      // pixel range, a twentieth of a pixel wider for the rounding here
      const double x0 = ulo * P.sx + P.ox - 0.05, x1 = uhi * P.sx + P.ox + 0.05;
      const double y0 = vlo * P.sy + P.oy - 0.05, y1 = vhi * P.sy + P.oy + 0.05;
      visible = x1 >= 0.0 && y1 >= 0.0 && x0 <= (double)V.w && y0 <= (double)V.h;
      if (visible) {
        bx0 = (uint32_t)(fmax(x0, 0.0) * P.inv_bw);
        by0 = (uint32_t)(fmax(y0, 0.0) * P.inv_bh);
        bx1 = min((uint32_t)(fmin(x1, (double)V.w) * P.inv_bw), P.bins_x - 1);
        by1 = min((uint32_t)(fmin(y1, (double)V.h) * P.inv_bh), P.bins_y - 1);
        bx0 = min(bx0, bx1);
        by0 = min(by0, by1);
      }
    }
    const size_t at = (size_t)P.rec_begin + j;
    if (visible) {
      // (bounds over single bins lie between the proxy's and about its centre's distance)
      key_lo = min(key_lo, __float_as_uint(tbf));
      key_hi = max(key_hi, max(__float_as_uint(tbf), __float_as_uint(fminf((float)sqrt(dist2), 1e30f))));
      rec1.z = __uint_as_float(bx0 | (bx1 << 16));
      rec1.w = __uint_as_float(by0 | (by1 << 16));
      L.rec[2 * at] = rec0;
      L.rec[2 * at + 1] = rec1;
      L.box[at] = bb;
    } else {
      rec1.z = rec1.w = __uint_as_float(0xFFFFFFFFu);
      L.rec[2 * at + 1] = rec1;
    }
  }
  key_lo = __reduce_min_sync(kFull, key_lo);
  key_hi = __reduce_max_sync(kFull, key_hi);
  if ((threadIdx.x & 31) == 0 && key_lo <= key_hi) {
    atomicMin(&L.range[2 * blockIdx.y], key_lo);
    atomicMax(&L.range[2 * blockIdx.y + 1], key_hi);
  }
}

// A proxy's circumscribed sphere in its object space, for bounds over bins.
struct ProxySlab {
  float u, v;     // outline centre
  float tb;       // distance bound over all rays
  float rp;       // sphere radius (0: no bounds but tb)
  float least;    // plane distances below this are too inexact to use
  V3 oo;          // camera
  V3 wx, wy, wz;  // the camera frame's axes
};

// Lower bound of the distance at which a ray through the image-plane
// rectangle can enter the proxy.  Every point x of the sphere satisfies
// x . p <= rp^2 for any p on it, so a ray oo + s (u wx + v wy + wz) enters it
// at s >= (oo . p - rp^2) / -((u wx + v wy + wz) . p); the denominator is
// linear in (u, v), largest at a corner.  p is where the ray through the
// rectangle's point nearest to the outline's centre enters the sphere: the
// front surface recedes from there, so the bound is nearly the true
// smallest entry distance.  (2e-4 lower for the rounding here and of t.)
__device__ __forceinline__ float bin_bound(const ProxySlab& S, float u0, float u1, float v0, float v1) {
  if (!(S.rp > 0.0f)) return S.tb;
  const float u = fminf(fmaxf(S.u, u0), u1), v = fminf(fmaxf(S.v, v0), v1);
  const V3 w = mk(__fmaf_rn(u, S.wx.x, __fmaf_rn(v, S.wy.x, S.wz.x)), __fmaf_rn(u, S.wx.y, __fmaf_rn(v, S.wy.y, S.wz.y)),
                  __fmaf_rn(u, S.wx.z, __fmaf_rn(v, S.wy.z, S.wz.z)));
  const float a = vdot(w, w), b = vdot(S.oo, w);
  const float sm = -b / a;  // closest approach
  V3 c = mk(__fmaf_rn(sm, w.x, S.oo.x), __fmaf_rn(sm, w.y, S.oo.y), __fmaf_rn(sm, w.z, S.oo.z));
  const float h2 = S.rp * S.rp - vdot(c, c);
  if (h2 > 0.0f) {
    const float back = sqrtf(h2 / a);
    c = mk(c.x - back * w.x, c.y - back * w.y, c.z - back * w.z);
  }
  const float cl = vdot(c, c);
  if (!(cl > 0.0f)) return S.tb;
  const float sc = S.rp * rsqrtf(cl) * 0.999999f;  // (inside the sphere: a looser half-space)
  const V3 p = mk(c.x * sc, c.y * sc, c.z * sc);
  const float num = vdot(S.oo, p) - S.rp * S.rp;
  if (!(num > S.least)) return S.tb;
  const float px = -vdot(S.wx, p), py = -vdot(S.wy, p), pz = -vdot(S.wz, p);
  const float den = fmaxf(u0 * px, u1 * px) + fmaxf(v0 * py, v1 * py) + pz;
  if (!(den > 0.0f)) return S.tb;
  const float un = fminf(fmaxf(0.0f, u0), u1), vn = fminf(fmaxf(0.0f, v0), v1);
  const float q = sqrtf(__fmaf_rn(un, un, __fmaf_rn(vn, vn, 1.0f)));
  const float t = num / den * q * (1.0f - 2e-4f);
  return t > S.tb && t < 1e30f ? t : S.tb;
}

// The two passes of the counting sort over (bin, bucket) cells: SCATTER
// false counts each cell's entries, true writes them (a cell then holds the
// next free place of its bin's list).
// A warp takes 32 proxies (8 of a small scene) and shares their pairs with bins out evenly (a proxy
// meets one bin or hundreds: with a lane a proxy 158 + 260 us for 1080p and 1M
// proxies, 74 + 137 so).
constexpr uint32_t kPassBlock = 128;
struct PassRow {
  ProxySlab slab;
  uint32_t bx, by, nx;  // bins: the first, and how many across
};
template <bool SCATTER>
__global__ void __launch_bounds__(kPassBlock) k_list_pass(const ViewDev* __restrict__ views,
                                                   const ListView* __restrict__ lviews, float r_circ,
                                                   uint32_t per_warp, const Lists L) {
  const ViewDev& V = views[blockIdx.y];
  const ListView& P = lviews[blockIdx.y];
  const uint32_t lane = threadIdx.x & 31;
  const Buckets B = make_buckets(L.range[2 * blockIdx.y], L.range[2 * blockIdx.y + 1]);
  const uint32_t bpr = V.tiles_x / kTileBlock;
  const float bw = 1.0f / (float)P.inv_bw, bh = 1.0f / (float)P.inv_bh;
  const float isx = (float)(1.0 / P.sx), isy = (float)(1.0 / P.sy), ox = (float)P.ox, oy = (float)P.oy;
  const V3 o = mk(V.u.tw[12], V.u.tw[13], V.u.tw[14]);
  auto put = [&](uint32_t bx, uint32_t by, const ProxySlab& S, uint32_t j) {
    const uint32_t bin = P.bin_begin + bin_index(bx, by, L.shift, bpr);
    // the bin's image-plane rectangle, a little larger
    const float u0 = ((float)bx * bw - 0.1f - ox) * isx, u1 = ((float)(bx + 1) * bw + 0.1f - ox) * isx;
    const float v0 = ((float)by * bh - 0.1f - oy) * isy, v1 = ((float)(by + 1) * bh + 0.1f - oy) * isy;
    const uint32_t bucket = bucket_of(B, __float_as_uint(bin_bound(S, u0, u1, v0, v1)));
    uint32_t* cell = L.cells + ((size_t)bin << kListBucketBits) + bucket;
    if (SCATTER) {
      const uint32_t pos = L.bin_base[bin] + atomicAdd(cell, 1u);
      if (pos < L.cap) {
        L.ent_box[pos] = __ldg(L.box + (size_t)P.rec_begin + j);
        L.ent[pos] = make_uint2(j, bucket_edge(B, bucket));
      }
    } else {
      atomicAdd(cell, 1u);
    }
  };
  __shared__ PassRow rows_s[kPassBlock];
  __shared__ uint32_t first_s[kPassBlock + kPassBlock / 32];
  PassRow* rows = rows_s + (threadIdx.x & ~31u);
  uint32_t* first = first_s + 33u * (threadIdx.x >> 5);
  const uint32_t warps = gridDim.x * (kPassBlock / 32);
  for (uint32_t w = blockIdx.x * (kPassBlock / 32) + (threadIdx.x >> 5); (uint64_t)w * per_warp < V.s.n_kept; w += warps) {
    const uint32_t base = w * per_warp, j = base + lane;
    uint32_t total = 0;
    if (lane < per_warp && j < V.s.n_kept) {
      const size_t at = (size_t)P.rec_begin + j;
      const float4 r1 = __ldg(L.rec + 2 * at + 1);
      const uint32_t rx = __float_as_uint(r1.z), ry = __float_as_uint(r1.w);
      if (rx != 0xFFFFFFFFu) {
        PassRow& Q = rows[lane];
        const float4 r0 = __ldg(L.rec + 2 * at);
        ProxySlab S;
        S.u = r0.x;
        S.v = r0.y;
        S.tb = r1.y;
        const Affine W = load_affine(V.s.w2o + 3 * (size_t)j);
        S.oo = xpoint(W, o);
        const float l1o = fabsf(S.oo.x) + fabsf(S.oo.y) + fabsf(S.oo.z);
        // rec0 = 0: no outline, the proxy's own bound for every bin
        S.rp = r0.w > 0.0f ? (r_circ + 1e-3f + 1e-5f * l1o) * 1.000001f : 0.0f;
        S.least = 0.01f * l1o * S.rp + 0.05f * S.rp * S.rp;
        S.wx = xdir(W, mk(P.Xf[0], P.Xf[1], P.Xf[2]));
        S.wy = xdir(W, mk(P.Yf[0], P.Yf[1], P.Yf[2]));
        S.wz = xdir(W, mk(P.Zf[0], P.Zf[1], P.Zf[2]));
        Q.slab = S;
        Q.bx = rx & 0xFFFFu;
        Q.by = ry & 0xFFFFu;
        Q.nx = (rx >> 16) - (rx & 0xFFFFu) + 1;
        total = Q.nx * ((ry >> 16) - (ry & 0xFFFFu) + 1);
      }
    }
    // the warp's (proxy, bin) pairs, shared out evenly
    uint32_t end = total;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, end, off);
      if ((int)lane >= off) end += y;
    }
    first[lane] = end - total;
    const uint32_t pairs = __shfl_sync(kFull, end, 31);
    __syncwarp();
    for (uint32_t t = lane; t < pairs; t += 32) {
      uint32_t src = 0;  // the last row whose first pair is not past t
#pragma unroll
      for (uint32_t step = 16; step > 0; step >>= 1)
        if (first[src + step] <= t) src += step;
      const PassRow& Q = rows[src];
      const uint32_t q = t - first[src], dy = q / Q.nx;
      put(Q.bx + (q - dy * Q.nx), Q.by + dy, Q.slab, base + src);
    }
    __syncwarp();
  }
}

// One bin a block: its cells' counts become offsets within the bin's list.
__global__ void __launch_bounds__(128) k_list_rows(const Lists L) {
  constexpr uint32_t kPer = (1u << kListBucketBits) / 128;
  uint32_t* row = L.cells + ((size_t)blockIdx.x << kListBucketBits) + threadIdx.x * kPer;
  uint32_t v[kPer], sum = 0;
#pragma unroll
  for (uint32_t i = 0; i < kPer; ++i) {
    v[i] = row[i];
    sum += v[i];
  }
  __shared__ uint32_t ws[4];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, x, off);
    if ((int)lane >= off) x += y;
  }
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  uint32_t pre = x - sum;
  for (uint32_t w = 0; w < warp; ++w) pre += ws[w];
  if (threadIdx.x == 127) L.bin_base[blockIdx.x] = pre + sum;
#pragma unroll
  for (uint32_t i = 0; i < kPer; ++i) {
    row[i] = pre;
    pre += v[i];
  }
}

// One block: the bins' lengths become the starts of their lists, and the bins
// are ordered by length (in powers of two, longest first).  Tiles of long lists
// take longest, and the launch's end waits on those taken last (256x256 of 16k
// Gaussians 483 -> 435 us, 960x540 of 1M 3.86 -> 3.67 ms, 1080p unchanged).
// The sums stop at kListFull, above every capacity (proxies times bins has no
// bound below 2^32): lists from there on count as not fitting, and a list is
// shorter than 2^31, so that no position past them wraps either.
constexpr uint32_t kListFull = 0x7FFFFFFFu;
__device__ __forceinline__ uint32_t list_add(uint32_t a, uint32_t b) { return min(a + b, kListFull); }

__global__ void __launch_bounds__(1024) k_list_bins(const Lists L, uint32_t n_bins) {
  __shared__ uint32_t ws[32];
  __shared__ uint32_t carry;
  __shared__ uint32_t place[33];  // bins per class, then their first places
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  if (threadIdx.x < 33) place[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t base = 0; base < n_bins; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < n_bins ? L.bin_base[i] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, x, off);
      if ((int)lane >= off) x = list_add(x, y);
    }
    uint32_t pre = __shfl_up_sync(kFull, x, 1);
    if (lane == 0) pre = 0;
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t s = ws[lane];
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, s, off);
        if ((int)lane >= off) s = list_add(s, y);
      }
      ws[lane] = s;
    }
    __syncthreads();
    const uint32_t before = list_add(carry, warp ? ws[warp - 1] : 0u);
    if (i < n_bins) {
      const uint32_t at = list_add(before, pre);
      L.bin_base[i] = at;
      atomicAdd(&place[__clz(list_add(at, v) - at)], 1u);  // (the length that the starts give)
    }
    __syncthreads();
    if (threadIdx.x == 1023) carry = list_add(carry, ws[31]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    L.bin_base[n_bins] = carry;
    if (carry > L.cap) *reinterpret_cast<volatile uint32_t*>(L.need) = carry;
    uint32_t at = 0;
    for (int c = 0; c < 33; ++c) {
      const uint32_t k = place[c];
      place[c] = at;
      at += k;
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n_bins; i += 1024) {
    const uint32_t v = L.bin_base[i + 1] - L.bin_base[i];
    L.order[atomicAdd(&place[__clz(v)], 1u)] = i;
  }
}

// ------------------------------------------------------------------ trace
// Waiting hits per ray in shared memory; the count of some ray that starts
// compositing, and how many more than were left the last time (rays whose hits
// cannot be final yet would start it after every batch).  32 rows and 128
// registers allow 16 warps an SM (1M Gaussians at 1080p: 24 rows 22.0 ms, 32
// 17.1, 48 17.8, 64 19.5 before the spill rows; starting at 16 to 28: within
// 0.4 %; 20 warps an SM of 96 registers: 21.2).
constexpr int kStreamKb = 32;
constexpr int kStreamHot = 24;
constexpr uint32_t kStreamStep = 10;
// Chunks of a list after which a tile looks whether every tile is taken (481x271 of
// 1M Gaussians from radius 300 with a few proxies far out, so that their box fills
// the image: 13.5 ms without, 1.57 / 1.62 / 1.71 at 32 / 64 / 128; 1080p of the
// scene alone 9.31 -> 9.33).
constexpr uint32_t kStreamLook = 32;

template <int R>
struct StreamScratch {
  FaceRows faces;
  unsigned long long hk[kStreamKb][R];  // 4-ary min-heap of ray r in column r
  float4 ca[32];                        // outlines of the current survivors: u0, v0, slope, g11
  float cg[32];                         // g22
  uint32_t cj[32];                      // their proxies
  float ce[32];                         // and distance bounds
  uint32_t sqj[64];                     // entries that overlap the tile, not yet loaded
  float sqe[64];
  uint32_t pj[64];  // (proxy, ray) pairs
  uint8_t pr[64];
  float dx[R], dy[R], dz[R];       // ray directions
  float lim[R];                    // hits from here on were dropped (a full heap); -inf: start over
  uint32_t hn[R];                  // waiting hits (past kStreamKb: dropped ones)
  float sT[R], s0[R], s1[R], s2[R];  // a ray's state at the start of its round
  uint32_t sh[R], sf[R];             // (checkpointing: its record and that record's entries)
  RayStats stats;
};

// Key of hit (t, p): ordered like (t, p); -0 is folded into +0.
__device__ __forceinline__ uint32_t s_ord(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ unsigned long long s_key(float t, uint32_t p) {
  return ((unsigned long long)s_ord(t + 0.0f) << 32) | p;
}
__device__ __forceinline__ float s_key_t(unsigned long long k) {
  const uint32_t u = (uint32_t)(k >> 32);
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Rows of a ray's column: the first kStreamKb in shared memory, the next
// kStreamSpill (rays with many hits at nearly one distance, a few in a
// hundred; all rays of a dense scene whose proxies surround the camera, where no
// hit is final before the last of these is tested) in the warp's part of a global
// buffer.  96 / 224 / 480 rows: 1M uniform Gaussians from their centre, 960x540,
// 82.7 / 12.8 / 12.9 ms (hierarchy kernels 57.1), 31k of four times the size
// 100 / 22.8 / 19.0, 1M clusters from (4, 1, 3) 5.36 / 4.09 / 3.38; views from
// outside are the same.  224 rows take 136 MB.
template <int R>
__device__ __forceinline__ unsigned long long* stream_row(StreamScratch<R>& W, unsigned long long* sp, uint32_t i,
                                                          uint32_t r) {
  return i < (uint32_t)kStreamKb ? &W.hk[i][r] : sp + (i - kStreamKb) * R + r;
}

// Puts the keys in rows n .. end - 1 of column r into its heap of n entries.
template <int R, bool SPILL>
__device__ __forceinline__ void stream_push(StreamScratch<R>& W, unsigned long long* sp, uint32_t r, uint32_t n,
                                            uint32_t end) {
  auto row = [&](uint32_t i) { return SPILL ? stream_row(W, sp, i, r) : &W.hk[i][r]; };
  for (; n < end; ++n) {
    const unsigned long long x = *row(n);
    uint32_t i = n;
    while (i > 0) {
      const uint32_t par = (i - 1) >> 2;
      const unsigned long long pk = *row(par);
      if (!(x < pk)) break;
      *row(i) = pk;
      i = par;
    }
    *row(i) = x;
  }
}

// Removes the smallest key of column r (n entries before).
template <int R, bool SPILL>
__device__ __forceinline__ void stream_pop(StreamScratch<R>& W, unsigned long long* sp, uint32_t r, uint32_t n) {
  const uint32_t last = n - 1;
  if (last == 0) return;
  auto row = [&](uint32_t i) { return SPILL ? stream_row(W, sp, i, r) : &W.hk[i][r]; };
  const unsigned long long x = *row(last);
  uint32_t i = 0;
  while (true) {
    const uint32_t c = 4 * i + 1;
    if (c >= last) break;
    const uint32_t c1 = min(c + 1, last - 1), c2 = min(c + 2, last - 1), c3 = min(c + 3, last - 1);
    const unsigned long long k0 = *row(c), k1 = *row(c1), k2 = *row(c2), k3 = *row(c3);
    const bool s01 = k1 < k0, s23 = k3 < k2;
    const unsigned long long m01 = s01 ? k1 : k0, m23 = s23 ? k3 : k2;
    const uint32_t i01 = s01 ? c1 : c, i23 = s23 ? c3 : c2;
    const bool s = m23 < m01;
    const unsigned long long ck = s ? m23 : m01;
    if (!(ck < x)) break;
    *row(i) = ck;
    i = s ? i23 : i01;
  }
  *row(i) = x;
}

__device__ __forceinline__ bool stream_more(const RayUniforms& u, float T, float t_curr, uint32_t step) {
  return u.T_min < T && t_curr < u.t_max && u.early_stop != step;
}

// Work items are the R-ray parts of the tiles [0, total_tiles) of the
// launch's views.
template <int R, bool CKPT>
__global__ void __launch_bounds__(32, 16) k_trace_stream(const ViewDev* __restrict__ views,
                                                     const ListView* __restrict__ lviews, uint32_t n_views,
                                                     uint32_t total_tiles, DevCounters* ctr,
                                                     const __grid_constant__ FaceTable F, const Lists L,
                                                     const Handoff hand, const Ckpt ck) {
  constexpr uint32_t kParts = 32 / R;  // parts of a tile; also survivors tested at once
  extern __shared__ __align__(16) unsigned char smem_raw[];
  StreamScratch<R>& W = *reinterpret_cast<StreamScratch<R>*>(smem_raw);
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t r = lane % R, grp = lane / R;
  const uint32_t lt_mask = (1u << lane) - 1u;
  unsigned long long* sp = L.spill + (size_t)blockIdx.x * (kStreamSpill * R);
  if (lane == 0) W.stats = RayStats{0, 0, 0, 0, 0, 0};
  load_face_rows(F, W.faces, lane);
  __syncwarp();
  uint32_t status = 0, rays = 0;
  uint32_t n_rounds = 0, n_entries = 0, n_contrib = 0;
  const uint32_t total = total_tiles * kParts;
  while (true) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(&ctr->work, 1u);
    item = __shfl_sync(kFull, item, 0);
    if (item >= total) break;
    const uint32_t part = item % kParts;
    uint32_t tile = item / kParts;
    tile = (__ldg(L.order + (tile >> L.shift)) << L.shift) | (tile & ((1u << L.shift) - 1u));
    const uint32_t vi = n_views == 1 ? 0u : find_view(views, n_views, tile);
    const ViewDev& V = views[vi];
    // R = 32: the tile; 8: its 4x2 quarter (part & 1, part >> 1)
    uint32_t s = r;
    if (R == 8) s = ((part >> 1) * 2 + (r >> 2)) * 8 + (part & 1) * 4 + (r & 3);
    uint32_t px, py;
    tile_pixel(V.tiles_x, tile - V.tile_begin, s, px, py);
    const bool valid = px < V.w && py < V.h;
    if (__ballot_sync(kFull, valid) == 0) continue;
    V3 o, d;
    ray_gen(V.u, V.w, V.h, valid ? px : 0u, valid ? py : 0u, o, d);
    float u, v;
    {
      const ListView& P = lviews[vi];
      const float z = d.x * P.Zf[0] + d.y * P.Zf[1] + d.z * P.Zf[2];
      u = __fdiv_rn(d.x * P.Xf[0] + d.y * P.Xf[1] + d.z * P.Xf[2], z);
      v = __fdiv_rn(d.x * P.Yf[0] + d.y * P.Yf[1] + d.z * P.Yf[2], z);
    }
    const uint32_t bin = tile >> L.shift;
    uint32_t pos = L.bin_base[bin];
    const uint32_t end = L.bin_base[bin + 1];
    const float t_min = V.u.t_min, t_max = V.u.t_max;
    const uint32_t k = V.u.k;
    float L0 = 0.f, L1 = 0.f, L2 = 0.f, T = 1.f, t_curr = t_min;
    uint32_t step = 0, e = 0, rc = 0;  // rounds done; entries of the open round, those that contribute
    uint32_t heap = 0;                 // waiting hits that are in heap order
    uint32_t cc = 0;                   // contributing entries of the rounds done
    uint32_t ck_head = kInvalid, ck_fill = ck.kc;
    bool live = valid && grp == 0 && stream_more(V.u, T, t_curr, step);
    bool handed = false;
    if (grp == 0) {
      W.dx[r] = d.x;
      W.dy[r] = d.y;
      W.dz[r] = d.z;
      W.lim[r] = end > L.cap ? -CUDART_INF_F : CUDART_INF_F;  // a list that did not fit is not used
      W.hn[r] = 0;
      W.sT[r] = T;
      W.s0[r] = W.s1[r] = W.s2[r] = 0.f;
      if (CKPT) {
        W.sh[r] = ck_head;
        W.sf[r] = ck_fill;
      }
    }
    // rays of the other groups' lanes mirror group 0's
    uint32_t live_m = __ballot_sync(kFull, live);
    bool mine = (live_m >> r) & 1u;
    int nq = 0, nsq = 0, sv_n = 0, sv_i = 0;
    float pedge = CUDART_INF_F, done = -CUDART_INF_F;
    uint32_t scanned = 0, tested = 0;
    float ulo = 0.f, uhi = 0.f, vlo = 0.f, vhi = 0.f;
    auto bounds = [&]() {
      float a = mine ? u : CUDART_INF_F, b = mine ? u : -CUDART_INF_F, c = mine ? v : CUDART_INF_F,
            f = mine ? v : -CUDART_INF_F;
#pragma unroll
      for (int off = R / 2; off > 0; off >>= 1) {
        a = fminf(a, __shfl_xor_sync(kFull, a, off));
        b = fmaxf(b, __shfl_xor_sync(kFull, b, off));
        c = fminf(c, __shfl_xor_sync(kFull, c, off));
        f = fmaxf(f, __shfl_xor_sync(kFull, f, off));
      }
      ulo = a;
      uhi = b;
      vlo = c;
      vhi = f;
    };
    bounds();
    bool hot = end > L.cap;
    uint32_t hot_n = kStreamHot;
    if (hot) pos = end;
    // the next chunk of 32 list entries, loaded one chunk ahead
    float4 nbx = make_float4(0.f, 0.f, 0.f, 0.f);
    uint2 nen = make_uint2(0u, 0x7F800000u);
    if (pos + lane < end) {
      nbx = __ldg(L.ent_box + pos + lane);
      nen = __ldg(L.ent + pos + lane);
    }
    __syncwarp();
    while (live_m) {
      const bool dry = sv_i == sv_n && nsq == 0 && pos >= end;
      if (nq >= 32 || (dry && nq > 0)) {
        // exact face tests of 32 pairs, oldest first
        const int nb = nq < 32 ? nq : 32;
        const bool have = (int)lane < nb;
        uint32_t j = 0, pr = 0;
        if (have) {
          j = W.pj[lane];
          pr = W.pr[lane];
        }
        uint32_t mj = 0, mr = 0;
        const bool mv = (int)lane < nq - nb;
        if (mv) {
          mj = W.pj[nb + lane];
          mr = W.pr[nb + lane];
        }
        __syncwarp();
        if (mv) {
          W.pj[lane] = mj;
          W.pr[lane] = (uint8_t)mr;
        }
        nq -= nb;
        // (what is left came from the survivor tested last)
        if (sv_n > 0) pedge = W.ce[max(0, min(sv_i, sv_n) - (int)kParts)];
        tested += (uint32_t)nb;
        // hits are appended to their ray's column; its own lane puts them into
        // the heap when it composites
        uint32_t nh = 0;
        if (have) {
          const uint32_t p = __ldg(V.s.leaf_pidx + j);
          auto on_hit = [&](float t, int) {
            const uint32_t at = atomicAdd(&W.hn[pr], 1u);
            if (at < (uint32_t)(kStreamKb + kStreamSpill)) *stream_row(W, sp, at, pr) = s_key(t, p);
            // dropped, or late (-inf: the ray starts over): floats >= 0 and
            // -inf order like their bits as ints
            if (at >= (uint32_t)(kStreamKb + kStreamSpill) || t < done)
              atomicMin(reinterpret_cast<int*>(&W.lim[pr]), __float_as_int(t < done ? -CUDART_INF_F : t));
            ++nh;
          };
          proxy_faces(F, W.faces, V.s.w2o, j, o, mk(W.dx[pr], W.dy[pr], W.dz[pr]), t_min, t_max, on_hit);
        }
        const uint32_t found = __reduce_add_sync(kFull, nh);
        if (lane == 0) W.stats.anyhits += found;
        __syncwarp();
        hot = found && __any_sync(kFull, mine && W.hn[r] >= hot_n);
        if (!hot && !dry) continue;
        if (nq > 0 && dry) continue;
      }
      if (hot || dry) {
        // composite every hit below the bound of what is not tested yet
        float B = CUDART_INF_F;
        if (nq > 0)
          B = pedge;
        else if (sv_i < sv_n)
          B = W.ce[sv_i];
        else if (nsq > 0)
          B = W.sqe[0];
        else if (pos < end)
          B = __uint_as_float(__shfl_sync(kFull, nen.y, 0));
        hot = false;
        const float lim = W.lim[r];
        const float Bl = fminf(B, lim);
        uint32_t n = min(W.hn[r], (uint32_t)(kStreamKb + kStreamSpill));
        if (live) {
          if (n <= (uint32_t)kStreamKb)
            stream_push<R, false>(W, sp, r, heap, n);
          else
            stream_push<R, true>(W, sp, r, heap, n);
        }
        unsigned long long root = 0;
        Shade sd{};
        if (live && n > 0) {
          root = W.hk[0][r];
          sd = load_shade(V.s.shade, (uint32_t)root);
        }
        while (true) {
          const bool act = live && n > 0 && s_key_t(root) < Bl;
          if (!__any_sync(kFull, act)) break;
          bool contrib = false, full = false;
          float alpha = 0.f, x0 = 0.f, x1 = 0.f, x2 = 0.f, t = 0.f;
          uint32_t ep = 0;
          if (act) {
            t = s_key_t(root);
            ep = (uint32_t)root;
            const Shade cur = sd;
            if (n <= (uint32_t)kStreamKb)
              stream_pop<R, false>(W, sp, r, n);
            else
              stream_pop<R, true>(W, sp, r, n);
            --n;
            if (n > 0) {  // the next entry's record loads while this one is shaded
              root = W.hk[0][r];
              sd = load_shade(V.s.shade, (uint32_t)root);
            }
            if (t > t_curr) {  // (else within 1e-4 past the last round's k-th hit)
              alpha = response(cur, o, d) * cur.opacity;
              ++e;
              full = e == k;
              if (V.u.alpha_min < alpha) {
                contrib = true;
                if (V.rgb) {
                  const float4 q = __ldg(V.rgb + ep);
                  x0 = q.x;
                  x1 = q.y;
                  x2 = q.z;
                } else {
                  entry_colour(V.s.sh, ep, cur.mu, o, V.u.deg, x0, x1, x2);
                }
              }
            }
          }
          if (CKPT && ck.kc) {
            // checkpoint mode: the entry goes to the ray's open record
            const bool open = contrib && ck_fill >= ck.kc;
            const uint32_t om = __ballot_sync(kFull, open);
            if (om) {
              const int leader = __ffs(om) - 1;
              uint32_t base = 0;
              if ((int)lane == leader) base = atomicAdd(ck.pool_next, (uint32_t)__popc(om));
              base = __shfl_sync(kFull, base, leader);
              if (open) {
                const uint32_t rec = base + (uint32_t)__popc(om & lt_mask);
                if (rec < ck.pool_cap) {  // past the pool the host sizes it up and runs again
                  uint32_t* rr = ck.pool + (size_t)rec * (kCkptHeader + ck.kc);
                  rr[0] = __float_as_uint(t_curr);
                  rr[1] = __float_as_uint(T);
                  rr[2] = ck_head;
                }
                ck_head = rec;
                ck_fill = 0;
              }
            }
            if (contrib) {
              if (ck_head < ck.pool_cap) {
                uint32_t* rr = ck.pool + (size_t)ck_head * (kCkptHeader + ck.kc);
                rr[kCkptHeader + ck_fill] = ep;
                rr[3] = ck_fill + 1;
              }
              ++ck_fill;
            }
          }
          if (contrib) {
            const float ta = T * alpha;
            L0 = L0 + ta * x0;
            L1 = L1 + ta * x1;
            L2 = L2 + ta * x2;
            T = T * (1.0f - alpha);
            ++rc;
          }
          if (CKPT && ck.kc == 0) {
            // replay mode: one record a round
            const uint32_t fm = __ballot_sync(kFull, full);
            if (fm) {
              uint32_t base = 0;
              if ((int)lane == __ffs(fm) - 1) base = atomicAdd(ck.pool_next, (uint32_t)__popc(fm));
              base = __shfl_sync(kFull, base, __ffs(fm) - 1);
              const uint32_t rec = base + (uint32_t)__popc(fm & lt_mask);
              if (full && rec < ck.pool_cap) {
                uint32_t* rr = ck.pool + (size_t)rec * (kCkptHeader + ck.kc);
                rr[0] = __float_as_uint(t_curr);
                rr[1] = __float_as_uint(W.sT[r]);
                rr[2] = ck_head;
                rr[3] = e;
                ck_head = rec;
              }
            }
          }
          if (full) {  // the round is complete
            t_curr = t + 1e-4f;
            ++step;
            cc += rc;
            e = rc = 0;
            if (step >= F.lim_rounds && stream_more(V.u, T, t_curr, step)) {
              status |= kStatusRoundCap;
              t_curr = t_max;
            }
            live = stream_more(V.u, T, t_curr, step);
            if (!live) {
              n_rounds += step;
              n_entries += step * k;
              n_contrib += cc;
            }
            W.sT[r] = T;
            W.s0[r] = L0;
            W.s1[r] = L1;
            W.s2[r] = L2;
            if (CKPT) {
              W.sh[r] = ck_head;
              W.sf[r] = ck_fill;
            }
          }
        }
        heap = n;
        hot_n = max((uint32_t)kStreamHot, __reduce_max_sync(kFull, live ? n : 0u) + kStreamStep);
        if (grp == 0) W.hn[r] = n;
        done = fmaxf(done, B);
        // rays that cannot go on here: their next hit was dropped or came late
        bool off = live && lim <= B && lim < CUDART_INF_F;
        bool again = off && lim == -CUDART_INF_F;
        if (dry && nq == 0) {
          if (live && !off) {
            // no hit is left: the last round, of the e entries there were
            if (CKPT && ck.kc == 0) {
              const uint32_t rec = atomicAdd(ck.pool_next, 1u);
              if (rec < ck.pool_cap) {
                uint32_t* rr = ck.pool + (size_t)rec * (kCkptHeader + ck.kc);
                rr[0] = __float_as_uint(t_curr);
                rr[1] = __float_as_uint(W.sT[r]);
                rr[2] = ck_head;
                rr[3] = e;
                ck_head = rec;
              }
            }
            n_rounds += step + 1;
            n_entries += step * k + e;
            n_contrib += cc + rc;
            live = false;
          }
        } else if (hand.rays) {
          // once every tile is taken the launch's end waits on the tiles
          // still tracing: their rays go to the warp-per-ray kernel
          uint32_t taken = 0;
          if (lane == 0) taken = *reinterpret_cast<volatile const uint32_t*>(&ctr->work);
          if (__shfl_sync(kFull, taken, 0) >= total + hand.late) off = live;
        }
        const uint32_t om = __ballot_sync(kFull, off);
        if (om) {
          const uint32_t hm = __ballot_sync(kFull, off && !again);
          uint32_t base = 0;
          if (lane == 0 && hm) base = atomicAdd(&ctr->handoff, (uint32_t)__popc(hm));
          base = __shfl_sync(kFull, base, 0);
          if (off && !again) {
            const uint32_t idx = base + (uint32_t)__popc(hm & lt_mask);
            if (idx < hand.cap) {
              // back to the start of the open round
              if (CKPT) {
                ck_head = W.sh[r];
                ck_fill = W.sf[r];
                if (ck.kc && ck_head < ck.pool_cap && ck_fill <= ck.kc)
                  ck.pool[(size_t)ck_head * (kCkptHeader + ck.kc) + 3] = ck_fill;
              }
              hand.rays[idx] =
                  HandoffRay{32u * tile + s, step, t_curr, W.sT[r], W.s0[r], W.s1[r], W.s2[r], ck_head, ck_fill};
              n_rounds += step;
              n_entries += step * k;
              n_contrib += cc;
            } else {
              again = true;
            }
          }
          const uint32_t am = __ballot_sync(kFull, again);
          if (am) {
            uint32_t rb = 0;
            if (lane == 0) rb = atomicAdd(&ctr->redo, (uint32_t)__popc(am));
            rb = __shfl_sync(kFull, rb, 0);
            if (again) hand.redo[rb + (uint32_t)__popc(am & lt_mask)] = 32u * tile + s;
          }
          if (off) {
            live = false;
            handed = true;
          }
        }
        live_m = __ballot_sync(kFull, live);
        const bool was = mine;
        mine = (live_m >> r) & 1u;
        if (__any_sync(kFull, was != mine)) bounds();
        __syncwarp();
        continue;
      }
      if (sv_i < sv_n) {
        // survivors, kParts at a time: the rays inside their outlines become pairs
        do {
          const int si = sv_i + (int)grp;
          bool in = false;
          uint32_t j = 0;
          if (si < sv_n) {
            const float4 a = W.ca[si];
            const float dv = v - a.y;
            const float x = a.w * __fmaf_rn(a.z, dv, u - a.x), y = W.cg[si] * dv;
            in = mine && !(__fmaf_rn(x, x, y * y) > 1.0f);
            j = W.cj[si];
          }
          const uint32_t m = __ballot_sync(kFull, in);
          if (nq == 0) pedge = W.ce[sv_i];
          if (in) {
            const int q = nq + __popc(m & lt_mask);
            W.pj[q] = j;
            W.pr[q] = (uint8_t)r;
          }
          nq += __popc(m);
          sv_i += (int)kParts;
        } while (nq < 32 && sv_i < sv_n);
        if (sv_i > sv_n) sv_i = sv_n;
        __syncwarp();
        continue;
      }
      // scan the list until 32 entries overlap the tile or it ends, then
      // load their outlines
      while (nsq < 32 && pos < end) {
        const bool ov = pos + lane < end && nbx.x <= uhi && nbx.y >= ulo && nbx.z <= vhi && nbx.w >= vlo;
        const uint32_t m = __ballot_sync(kFull, ov);
        if (ov) {
          const int q = nsq + __popc(m & lt_mask);
          W.sqj[q] = nen.x;
          W.sqe[q] = __uint_as_float(nen.y);
        }
        nsq += __popc(m);
        pos += 32;
        if (pos + lane < end) {
          nbx = __ldg(L.ent_box + pos + lane);
          nen = __ldg(L.ent + pos + lane);
        }
        // a tile that goes through a long list without many hits looks up now and
        // then whether the others are done (it then hands its rays over, above)
        if ((++scanned & (kStreamLook - 1)) == 0 && hand.rays) {
          uint32_t taken = 0;
          if (lane == 0) taken = *reinterpret_cast<volatile const uint32_t*>(&ctr->work);
          hot = __shfl_sync(kFull, taken, 0) >= total + hand.late;
          if (hot) break;
        }
      }
      __syncwarp();
      sv_i = 0;
      sv_n = nsq < 32 ? nsq : 32;
      if ((int)lane < sv_n) {
        const uint32_t j = W.sqj[lane];
        const float4* rec = L.rec + 2 * ((size_t)lviews[vi].rec_begin + j);
        W.ca[lane] = __ldg(rec);
        W.cg[lane] = __ldg(reinterpret_cast<const float*>(rec + 1));
        W.cj[lane] = j;
        W.ce[lane] = W.sqe[lane];
      }
      uint32_t mj = 0;
      float me = 0.f;
      const bool mv = (int)lane < nsq - sv_n;
      if (mv) {
        mj = W.sqj[sv_n + lane];
        me = W.sqe[sv_n + lane];
      }
      __syncwarp();
      if (mv) {
        W.sqj[lane] = mj;
        W.sqe[lane] = me;
      }
      nsq -= sv_n;
      __syncwarp();
    }
    if (lane == 0) {
      W.stats.node_visits += scanned;
      W.stats.proxy_tests += tested;
    }
    if (valid && grp == 0 && !handed) {
      if (CKPT) ck.head[32u * tile + s] = ck_head < ck.pool_cap ? ck_head : kInvalid;
      const float4 q = make_float4(L0, L1, L2, 1.0f);
      float4* dst = V.out + (size_t)py * V.w + px;
      *dst = V.u.aa ? aa_blend(*dst, q, V.u.frames) : q;
      ++rays;
    }
    __syncwarp();
  }
  const uint32_t s_rays = __reduce_add_sync(kFull, rays);
  const uint32_t s_rounds = __reduce_add_sync(kFull, n_rounds);
  const uint32_t s_entries = __reduce_add_sync(kFull, n_entries);
  const uint32_t s_contrib = __reduce_add_sync(kFull, n_contrib);
  if (lane == 0) {
    W.stats.rounds += s_rounds;
    W.stats.entries += s_entries;
    W.stats.contributing += s_contrib;
  }
  __syncwarp();
  flush_stats(ctr, W.stats, lane == 0 ? s_rays : 0u, status);
}

template <int R, bool CKPT>
static Err launch_stream_r(const ViewDev* d_views, uint32_t n_views, uint32_t total_tiles, DevCounters* counters,
                           const FaceTable& faces, int num_sms, cudaStream_t stream, uint64_t* launches,
                           const Lists& L, Handoff hand, const Ckpt& ck) {
  const size_t smem = sizeof(StreamScratch<R>);
  GT_CUDA_TRY(
      cudaFuncSetAttribute(k_trace_stream<R, CKPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  GT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_stream<R, CKPT>, 32, smem));
  uint32_t grid = (uint32_t)num_sms * (uint32_t)std::max(1, per_sm);
  const uint32_t items = total_tiles * (32 / R);
  if (grid > items) grid = std::max(1u, items);
  grid = std::min(grid, (uint32_t)(L.spill_bytes / (sizeof(unsigned long long) * kStreamSpill * R)));
  // idle warps at which the tiles still tracing hand over: the rays of a
  // quarter tile lose less to one another, so theirs leave earlier (us with 50 /
  // 62 / 75 / 90 / 95 % idle: 200x150 of 1M Gaussians 1240 / 1248 / 1237 / 1268 /
  // 1331, of 200k 394 / 398 / 406 / 426 / 441, 256x256 of 1M 1556 / 1538 / 1590 /
  // 1599 / 1548, of 16k 353 / 347 / 348 / 348 / 348; with 32 rays a warp 481x271 of
  // 1M 1992 / 1760 / 1589 / 1693 / 1756, 640x360 2236 / 2123 / 2072 / 2010 / 2132,
  // 400x300 of 200k 701 / 626 / 560 / 554 / 590, 1080p within 1 %)
  hand.late = R == 8 ? grid / 8 * 5 : grid / 10 * 9;
  k_trace_stream<R, CKPT><<<grid, 32, smem, stream>>>(d_views, L.views, n_views, total_tiles, counters, faces, L,
                                                      hand, ck);
  ++*launches;
  GT_CUDA_TRY(cudaGetLastError());
  return Err{};
}

uint32_t pixels_of_box(const RayUniforms& u, uint32_t w, uint32_t h, const float* box) {
  double axis[3][3], len[3];  // right, up, view direction
  for (int r = 0; r < 3; ++r) {
    len[r] = 0.0;
    for (int q = 0; q < 3; ++q) {
      axis[r][q] = (r == 1 ? 1.0 : -1.0) * (double)u.tw[4 * r + q];
      len[r] += axis[r][q] * axis[r][q];
    }
    len[r] = sqrt(len[r]);
  }
  // x and y in half images from the centre, as ray_gen places the pixels
  double lo[2] = {1.0, 1.0}, hi[2] = {-1.0, -1.0};
  for (int c = 0; c < 8; ++c) {
    double v[3] = {0.0, 0.0, 0.0};
    for (int q = 0; q < 3; ++q) {
      const double p = (double)box[(c >> q & 1) * 3 + q] - (double)u.tw[12 + q];
      for (int r = 0; r < 3; ++r) v[r] += axis[r][q] * p;
    }
    if (!(v[2] > 1e-3 * len[2] * (fabs(v[0]) / len[0] + fabs(v[1]) / len[1]))) return w * h;
    for (int a = 0; a < 2; ++a) {
      const double x = v[a] / len[a] / (v[2] / len[2]) * len[2] / (len[a] * (double)u.asp[a]);
      if (!(fabs(x) < 1e30)) return w * h;
      lo[a] = std::min(lo[a], std::max(-1.0, x));
      hi[a] = std::max(hi[a], std::min(1.0, x));
    }
  }
  const double part = std::max(0.0, hi[0] - lo[0]) * std::max(0.0, hi[1] - lo[1]) / 4.0;
  return (uint32_t)(part * (double)w * (double)h + 0.5);
}

bool stream_views(const ViewDev* views, uint32_t n_views, uint32_t total_tiles, const FaceTable& faces) {
  if (n_views == 0 || n_views > 65535u || (uint64_t)total_tiles * 32u > kStreamMaxSlots) return false;
  // lowered limits (gt_set_limits) act on the hierarchy's loops
  if (faces.lim_steps != 0xFFFFFFFFu || faces.lim_stack != (uint32_t)kWarpStack || faces.lim_rounds != kMaxRounds)
    return false;
  bool any = false;
  for (uint32_t i = 0; i < n_views; ++i) {
    const RayUniforms& u = views[i].u;
    if (u.debug != 0 || !(u.t_min >= 0.0f) || u.t_min > 1e30f) return false;
    if (views[i].w > 1u << 20 || views[i].h > 1u << 19) return false;  // (16-bit bin coordinates)
    any = any || views[i].s.n_kept > 0;
    // a pinhole camera: finite, orthogonal axes (any lengths)
    double a[3][3], len[3];
    for (int r = 0; r < 3; ++r) {
      const float* c = u.tw + 4 * r;
      len[r] = 0.0;
      for (int q = 0; q < 3; ++q) {
        a[r][q] = c[q];
        len[r] += a[r][q] * a[r][q];
      }
      len[r] = sqrt(len[r]);
      if (!(len[r] > 1e-6 && len[r] < 1e6) || !(fabs((double)u.tw[12 + r]) < 1e15)) return false;
    }
    for (int r = 0; r < 3; ++r) {
      double dot = 0.0;
      for (int q = 0; q < 3; ++q) dot += a[r][q] * a[(r + 1) % 3][q];
      if (!(fabs(dot) <= 1e-6 * len[r] * len[(r + 1) % 3])) return false;
    }
    // the image plane's extent: u, v up to about 30 (a field of view of 176 degrees)
    const double eu = (double)u.asp[0] * len[0] / len[2], ev = (double)u.asp[1] * len[1] / len[2];
    if (!(eu > 1e-6 && eu < 30.0 && ev > 1e-6 && ev < 30.0)) return false;
  }
  return any;
}

// Rays per warp and bin size of a launch (rays = 0: not by lists).  B200, us
// as warp per ray / 8 rays per warp / 32 rays per warp, bins of 16x8 pixels for
// 8 rays and 32x16 for 32:
//   rays          uniform 16k k 6   clusters 200k k 8   clusters 1M k 16
//   64x64         203 /  315 /  368    242 /  517 /  710     750 / 2462 / 2660
//   128x96        314 /  316 /  429    294 /  462 /  561     910 / 1574 / 1942
//   200x150       566 /  331 /  434    479 /  463 /  552    1500 / 1525 / 1711
//   256x256       983 /  390 /  472    841 /  499 /  589    2174 / 2009 / 1954
//   400x300      1946 /  646 /  501   1491 /  559 /  614    3951 / 2138 / 1916
//   800x600      7472 / 1980 / 1155   5542 / 1362 /  970   14931 / 5222 / 3504
// With few tiles the warps with the most hits decide the time, so fewer rays
// share one; below 160 rays an SM even those are too few warps, and the lists of
// many proxies need a few more rays to pay (warp per ray / 8 rays per warp, us:
//   179x150 (181 an SM): 200k k 8 418 / 407, 360k k 7 531 / 618, 1M k 8 809 / 951
//   200x150 (203 an SM): 360k k 7 579 / 570, 700k k 8 535 / 627, 1M k 6 623 / 715
//   220x160 (238 an SM): 700k k 8 604 / 568, 1M k 8 1084 / 971, k 16 1407 / 1159),
// unless rounds are so short that a ray per warp pays for each (1M k 1, 200x150:
// 1852 / 1356).
// The rays that count are those that may meet the scene (`met`, pixels_of_box):
// a far scene fills few tiles, whose warps go through long lists while the others
// are idle (lists of a few thousand proxies are short: 400 that fill a sixth of
// 180x140, 846 / 583; warp per ray / lists, us):
//   481x271, radius 60:  200k k 8 401 / 609, 1M k 16 822 / 2206; radius 300: 1M
//   626 / 12920; 200x150: uniform 65k k 6 radius 12 288 / 349, radius 30 246 / 461.
// A warp for each of many rays that meet nothing costs more (2M rays 1.9 ms) than
// the lists of a few proxies (radius 100, k 6, 960x540: 16k 542 / 288, 65k
// 562 / 567; 1080p: 16k 1872 / 363, 65k 1943 / 538; radius 300, 960x540: 200k
// 636 / 1093, 1M 769 / 5570; 1080p: 200k 1881 / 740, 1M 1984 / 2355).
StreamPlan stream_plan(uint64_t rays, uint64_t met, uint64_t proxies, uint32_t k_min, int num_sms) {
  StreamPlan p;
  const uint64_t sms = (uint64_t)std::max(1, num_sms);
  if (proxies < 4096) met = rays;
  const bool near = met / sms >= 160 + (k_min >= 4 ? proxies / 14000 : 0);
  if (near || rays >= 200000 + 6 * proxies) {
    p.rays = (near ? met : rays) / sms < 640 ? 8 : 32;
    p.shift = p.rays == 8 ? 2u : 4u;
  }
  return p;
}

Err launch_trace_stream(const ViewDev* views, const ViewDev* d_views, uint32_t n_views, uint32_t total_tiles,
                        DevCounters* counters, const FaceTable& faces, int num_sms, cudaStream_t stream,
                        uint64_t* launches, const Lists& L, const Handoff& hand, const Ckpt* ckpt) {
  uint32_t kept = 0;
  for (uint32_t i = 0; i < n_views; ++i) kept = std::max(kept, views[i].s.n_kept);
  const uint32_t n_bins = total_tiles >> L.shift;
  GT_CUDA_TRY(cudaMemsetAsync(L.cells, 0, ((size_t)n_bins << kListBucketBits) * 4, stream));
  k_list_views<<<(n_views + 63) / 64, 64, 0, stream>>>(d_views, n_views, L.views, L);
  k_list_project<<<dim3(std::max(1u, (kept + 127) / 128), n_views), 128, 0, stream>>>(d_views, L.views, faces.r_circ, L);
  // proxies per warp: fewer where they would leave the GPU short of warps
  const uint32_t per_warp = (uint64_t)kept * n_views >= 32u * 16u * (uint64_t)num_sms ? 32u : 8u;
  const dim3 pass_grid(std::max(1u, (kept + per_warp * (kPassBlock / 32) - 1) / (per_warp * (kPassBlock / 32))),
                       n_views);
  k_list_pass<false><<<pass_grid, kPassBlock, 0, stream>>>(d_views, L.views, faces.r_circ, per_warp, L);
  k_list_rows<<<n_bins, 128, 0, stream>>>(L);
  k_list_bins<<<1, 1024, 0, stream>>>(L, n_bins);
  k_list_pass<true><<<pass_grid, kPassBlock, 0, stream>>>(d_views, L.views, faces.r_circ, per_warp, L);
  *launches += 6;
  GT_CUDA_TRY(cudaGetLastError());
  const Ckpt ck = ckpt ? *ckpt : Ckpt{};
  if (L.rays == 32)
    return ckpt ? launch_stream_r<32, true>(d_views, n_views, total_tiles, counters, faces, num_sms, stream, launches,
                                            L, hand, ck)
                : launch_stream_r<32, false>(d_views, n_views, total_tiles, counters, faces, num_sms, stream,
                                             launches, L, hand, ck);
  return ckpt ? launch_stream_r<8, true>(d_views, n_views, total_tiles, counters, faces, num_sms, stream, launches, L,
                                         hand, ck)
              : launch_stream_r<8, false>(d_views, n_views, total_tiles, counters, faces, num_sms, stream, launches,
                                          L, hand, ck);
}

}  // namespace gt
