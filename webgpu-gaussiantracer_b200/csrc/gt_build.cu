// gt_build.cu — GPU scene build: proxies, hierarchy, shading records.
//
// Replaces the reference's host-side acceleration-structure build
// (gaussianSceneToBvh, src/main.ts:30-111; Tlas.build,
// webrtx/src/wasm_bvh_builder.ts:260-377; build_blas/build_tlas,
// webrtx/bvh/src/lib.rs:254-347, 512-603) with a hierarchy built on the GPU:
//
//   1. one pass over the packed records (k_records): keep flags (opacity >
//      alpha_min), shading records in particle order (mean, opacity, precision
//      matrix, SH), proxy matrix M = T R diag(s*scale) and its inverse, world
//      AABB of the 12 transformed icosahedron vertices, bounds of the centres
//   2. an exclusive scan of the flags, 30-bit Morton codes of the box centres
//   3. LSD radix sort of (code, particle), hand-written: 3 passes of 10 bits in
//      one cooperative launch (k_radix_sort)
//   4. leaf records in leaf order (world-to-object map, particle index, box)
//   5. binary hierarchy: H-PLOC (gt_ploc.cu), or with fast_build Karras (2012)
//      over the sorted codes, ties broken by index, and a bottom-up refit
//   6. checks, and the greedy 8-wide collapse
//
// Node layout (4 x float4 per internal node; children's boxes in the parent):
//   f0 = (c0.lo.x, c0.hi.x, c0.lo.y, c0.hi.y)
//   f1 = (c1.lo.x, c1.hi.x, c1.lo.y, c1.hi.y)
//   f2 = (c0.lo.z, c0.hi.z, c1.lo.z, c1.hi.z)
//   f3 = (child0, child1, 0, 0) as uint bits; kLeafBit | j marks leaf j.
#include <cooperative_groups.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "gt_device.cuh"
#include "gt_internal.cuh"

namespace gt {

// ---------------------------------------------------------------- faces
// Icosahedron with inradius 1 (src/main.ts:12-25).
static const int kIcoIdx[60] = {0, 11, 5,  0, 5,  1,  0,  1,  7,  0,  7,  10, 0, 10, 11,
                                1, 5,  9,  5, 11, 4,  11, 10, 2,  10, 7,  6,  7, 1,  8,
                                3, 9,  4,  3, 4,  2,  3,  2,  6,  3,  6,  8,  3, 8,  9,
                                4, 9,  5,  2, 4,  11, 6,  2,  10, 8,  6,  7,  9, 8,  1};

static void ico_vertices(float v[36]) {
  double rr = (3.0 + sqrt(5.0)) / (2.0 * sqrt(3.0));
  double ss = 1.0 / rr;
  double tt = (1.0 + sqrt(5.0)) / (2.0 * rr);
  double t[36] = {-ss, tt, 0, ss,  tt, 0,  -ss, -tt, 0,   ss,  -tt, 0,   0,   -ss, tt,  0, ss,  tt,
                  0,   -ss, -tt, 0, ss, -tt, tt,  0,   -ss, tt,  0,   ss,  -tt, 0,   -ss, -tt, 0, ss};
  for (int i = 0; i < 36; ++i) v[i] = (float)t[i];
}

void make_face_table(FaceTable* F) {
  // Host code is compiled with -ffp-contract=off: each expression below is
  // rounded exactly as the device and the oracle round it.
  float v[36];
  ico_vertices(v);
  float nmax = 0.0f;
  for (int f = 0; f < 20; ++f) {
    const float* p0 = v + 3 * kIcoIdx[3 * f];
    const float* p1 = v + 3 * kIcoIdx[3 * f + 1];
    const float* p2 = v + 3 * kIcoIdx[3 * f + 2];
    float e0[3], e1[3];
    for (int a = 0; a < 3; ++a) {
      e0[a] = p1[a] - p0[a];
      e1[a] = p0[a] - p2[a];
      F->p0[f][a] = p0[a];
      F->e0[f][a] = e0[a];
      F->e1[f][a] = e1[a];
    }
    // n = cross(e1, e0)
    F->n[f][0] = e1[1] * e0[2] - e1[2] * e0[1];
    F->n[f][1] = e1[2] * e0[0] - e1[0] * e0[2];
    F->n[f][2] = e1[0] * e0[1] - e1[1] * e0[0];
    for (int a = 0; a < 3; ++a) nmax = fmaxf(nmax, fabsf(F->n[f][a]));
  }
  F->nmax = nmax;
  float r = 0.0f;
  for (int i = 0; i < 12; ++i)
    r = fmaxf(r, sqrtf(v[3 * i] * v[3 * i] + v[3 * i + 1] * v[3 * i + 1] + v[3 * i + 2] * v[3 * i + 2]));
  F->r_circ = r;
  float c[20];  // plane offsets
  for (int f = 0; f < 20; ++f)
    c[f] = F->n[f][0] * F->p0[f][0] + F->n[f][1] * F->p0[f][1] + F->n[f][2] * F->p0[f][2];
  // antipodal pairs: the face whose vertices are the negated vertices of f
  int q = 0;
  bool used[20] = {false};
  for (int f = 0; f < 20 && q < 10; ++f) {
    if (used[f]) continue;
    for (int g = f + 1; g < 20; ++g) {
      int match = 0;
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
          const float* va = v + 3 * kIcoIdx[3 * f + a];
          const float* vb = v + 3 * kIcoIdx[3 * g + b];
          if (va[0] == -vb[0] && va[1] == -vb[1] && va[2] == -vb[2]) ++match;
        }
      bool neg = F->n[g][0] == -F->n[f][0] && F->n[g][1] == -F->n[f][1] && F->n[g][2] == -F->n[f][2];
      if (match == 3 && neg) {
        F->pa[q] = f;
        F->pb[q] = g;
        used[f] = used[g] = true;
        ++q;
        break;
      }
    }
  }
  // the structure pair_dots builds on: one plane offset, the normals' signs and zeros
  {
    const float a = F->n[5][0], bb = F->n[1][1], cc = F->n[1][2];
    const float want[10][3] = {{-a, a, a}, {0, bb, cc},  {0, bb, -cc},  {-a, a, -a}, {-bb, cc, 0},
                               {a, a, a},  {-cc, 0, bb}, {-bb, -cc, 0}, {-cc, 0, -bb}, {a, a, -a}};
    bool same = q == 10;
    for (int r = 0; r < q && same; ++r) {
      for (int x = 0; x < 3; ++x) same = same && F->n[F->pa[r]][x] == want[r][x];
      same = same && c[F->pa[r]] == c[0] && c[F->pb[r]] == c[0];
    }
    if (!same) q = 0;  // (the context is not created)
    F->na = a;
    F->nb = bb;
    F->nc = cc;
    F->plane = c[0];
  }
  F->npairs = q;
  F->lim_steps = 0xFFFFFFFFu;
  F->lim_stack = kWarpStack;
  F->lim_rounds = kMaxRounds;
}
static_assert(sizeof(kIcoIdx) == 60 * sizeof(int), "table size");

struct IcoVerts {
  float v[36];
};

// ---------------------------------------------------------------- proxies
// src/main.ts:79-94: s = sqrt(2 ln(o / alpha_min)); M = T(mu) R diag(s*scale)
// with R = wgpu-matrix mat3.fromQuat([x, y, z, w]) evaluated in double and
// rounded to binary32 (Float32Array), s*scale rounded to binary32, and each
// column entry the binary32 product of the two.
// The activated values the proxy is built from: opacity, scale xyz and
// rotation wxyz.  The reference builds its proxies from the JS numbers of
// gaussianData (double); when the caller supplies them (act64, 8 doubles per
// particle in that order) they are used, else the packed binary32 values.
struct Act64 {
  double o, s[3], q[4];
};
__device__ __forceinline__ Act64 activation(const float* rec, const double* act64, uint64_t i) {
  Act64 a;
  if (act64) {
    const double* p = act64 + 8 * i;
    a.o = p[0];
#pragma unroll
    for (int c = 0; c < 3; ++c) a.s[c] = p[1 + c];
#pragma unroll
    for (int c = 0; c < 4; ++c) a.q[c] = p[4 + c];
  } else {
    a.o = rec[12];
#pragma unroll
    for (int c = 0; c < 3; ++c) a.s[c] = rec[4 + c];
#pragma unroll
    for (int c = 0; c < 4; ++c) a.q[c] = rec[8 + c];
  }
  return a;
}

__device__ __forceinline__ void proxy_o2w(const float* rec, const Act64& A, double alpha_min, float M[12]) {
  double o = A.o;
  double s = __dsqrt_rn(__dmul_rn(2.0, det_log(__ddiv_rn(o, alpha_min))));
  double w = A.q[0], x = A.q[1], y = A.q[2], z = A.q[3];
  double x2 = x + x, y2 = y + y, z2 = z + z;
  double xx = x * x2, yx = y * x2, yy = y * y2;
  double zx = z * x2, zy = z * y2, zz = z * z2;
  double wx = w * x2, wy = w * y2, wz = w * z2;
  double R[9] = {1.0 - yy - zz, yx + wz, zx - wy, yx - wz, 1.0 - xx - zz, zy + wx, zx + wy, zy - wx, 1.0 - xx - yy};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float Sc = __double2float_rn(__dmul_rn(s, A.s[c]));
#pragma unroll
    for (int r = 0; r < 3; ++r) M[3 * c + r] = __double2float_rn(R[3 * c + r]) * Sc;
  }
  M[9] = rec[0];
  M[10] = rec[1];
  M[11] = rec[2];
}

// Affine inverse (replaces glam Affine3A::inverse, webrtx/bvh/src/lib.rs:501-505):
// adjugate from cross products of the columns a, b, c; det = dot(c, cross(a, b)).
__device__ __forceinline__ void affine_inverse(const float M[12], float W[12]) {
  V3 a = mk(M[0], M[1], M[2]), b = mk(M[3], M[4], M[5]), c = mk(M[6], M[7], M[8]);
  V3 p = mk(M[9], M[10], M[11]);
  V3 t0 = vcross(b, c), t1 = vcross(c, a), t2 = vcross(a, b);
  float det = vdot(c, t2);
  float inv = __fdiv_rn(1.0f, det);
  W[0] = t0.x * inv; W[1] = t1.x * inv; W[2] = t2.x * inv;
  W[3] = t0.y * inv; W[4] = t1.y * inv; W[5] = t2.y * inv;
  W[6] = t0.z * inv; W[7] = t1.z * inv; W[8] = t2.z * inv;
  W[9] = -((W[0] * p.x + W[3] * p.y) + W[6] * p.z);
  W[10] = -((W[1] * p.x + W[4] * p.y) + W[7] * p.z);
  W[11] = -((W[2] * p.x + W[5] * p.y) + W[8] * p.z);
}

// float min/max through order-preserving integer maps (for atomics)
__device__ __forceinline__ uint32_t f2ord(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Everything the build takes from the packed records, in one pass over them:
// the keep flag, and for kept particles the shading records ((mu, opacity),
// the precision matrix A of computeResponse (6 unique entries), the SH floats
// made tight, scale and rotation), the proxy's world-to-object map and padded
// world box, and the bounds of the box centres.
//
// Bound by HBM: 320 bytes a record read, 344 written (0.66 GB for 1M).  The
// usual 320-byte records are read as coalesced quads, whose SH part leaves
// again as coalesced quads (the particles that are not kept included); only
// the head goes through shared memory (rows of an odd number of words: a
// thread a record reads without bank conflicts).  Other strides stage whole
// records.  Three kernels with a thread a record reading it from global memory
// took 191 + 191 + 22 us for 1M records on a B200, and the leaves' gather of
// the records 68; this takes 115 (231 with an atomic of every warp on the
// shared bounds).
constexpr uint32_t kRecBlock = 64;

// FULL: 320-byte records of 16 coefficients on 16-byte boundaries.
template <bool FULL>
__global__ void __launch_bounds__(kRecBlock) k_records(const uint8_t* __restrict__ packed, uint64_t n, uint32_t stride,
                                                       uint32_t n_sh, double alpha_min,
                                                       const double* __restrict__ act64, const IcoVerts iv,
                                                       uint32_t* __restrict__ flags, float4* __restrict__ shade,
                                                       float4* __restrict__ sh, float4* __restrict__ params,
                                                       float4* __restrict__ w2o, float* __restrict__ box,
                                                       uint32_t* bounds_ord) {
  extern __shared__ float rows[];
  __shared__ uint32_t kept_s[kRecBlock];
  // the words of a record that are read: the head and the SH rows present
  const uint32_t words = FULL ? 16u : min(stride / 4u, 16u + 4u * n_sh), pitch = words | 1u;
  const uint64_t p0 = (uint64_t)blockIdx.x * kRecBlock;
  const uint32_t cnt = (uint32_t)min((uint64_t)kRecBlock, n - p0);
  const uint8_t* src = packed + p0 * stride;
  if (FULL) {
    // 20 quads a record, ten loads of a thread in flight at a time.  Four
    // lanes hold four quads of one record: its head (quads 0-3), which goes
    // to shared memory, or four coefficients, three floats each of 12 that
    // leave as three quads.
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
      float4 v[10];
#pragma unroll
      for (uint32_t i = 0; i < 10; ++i) {
        const uint32_t at = (h * 10 + i) * kRecBlock + threadIdx.x;
        v[i] = at < cnt * 20u ? __ldcs(reinterpret_cast<const float4*>(src) + at) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (uint32_t i = 0; i < 10; ++i) {
        const uint32_t at = (h * 10 + i) * kRecBlock + threadIdx.x;
        const uint32_t r = at / 20u, q = at % 20u, g = q / 4u, l = q % 4u;
        const float nx = __shfl_down_sync(0xFFFFFFFFu, v[i].x, 1), ny = __shfl_down_sync(0xFFFFFFFFu, v[i].y, 1),
                    nz = __shfl_down_sync(0xFFFFFFFFu, v[i].z, 1);
        if (at >= cnt * 20u) continue;
        if (g == 0) {
          float* d = rows + r * pitch + 4u * l;
          d[0] = v[i].x;
          d[1] = v[i].y;
          d[2] = v[i].z;
          d[3] = v[i].w;
        } else if (l < 3u) {
          sh[12 * (p0 + r) + 3u * (g - 1u) + l] = l == 0   ? make_float4(v[i].x, v[i].y, v[i].z, nx)
                                                  : l == 1 ? make_float4(v[i].y, v[i].z, nx, ny)
                                                           : make_float4(v[i].z, nx, ny, nz);
        }
      }
    }
  } else {
    for (uint32_t i = threadIdx.x; i < cnt * words; i += kRecBlock) {
      const uint32_t r = i / words, w = i - r * words;
      rows[r * pitch + w] = __ldg(reinterpret_cast<const float*>(src + (size_t)r * stride) + w);
    }
  }
  __syncthreads();
  const uint64_t p = p0 + threadIdx.x;
  float cmin[3] = {CUDART_INF_F, CUDART_INF_F, CUDART_INF_F}, cmax[3] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
  float bmag = 0.0f;
  bool kept = false;
  if (threadIdx.x < cnt) {
    const float* rec = rows + threadIdx.x * pitch;
    const Act64 act = activation(rec, act64, p);
    kept = act.o > alpha_min;
    flags[p] = kept ? 1u : 0u;
    if (kept) {
      const float q[4] = {rec[8], rec[9], rec[10], rec[11]};
      const float sc[3] = {rec[4], rec[5], rec[6]};
      float A[3][3];
      precision_matrix(q, sc, A);
      shade[3 * p] = make_float4(rec[0], rec[1], rec[2], rec[12]);
      shade[3 * p + 1] = make_float4(A[0][0], A[1][0], A[2][0], A[1][1]);
      shade[3 * p + 2] = make_float4(A[2][1], A[2][2], 0.f, 0.f);
      params[2 * p] = make_float4(sc[0], sc[1], sc[2], 0.f);
      params[2 * p + 1] = make_float4(q[0], q[1], q[2], q[3]);
      float M[12], W[12];
      proxy_o2w(rec, act, alpha_min, M);
      affine_inverse(M, W);
      w2o[3 * p] = make_float4(W[0], W[1], W[2], W[3]);
      w2o[3 * p + 1] = make_float4(W[4], W[5], W[6], W[7]);
      w2o[3 * p + 2] = make_float4(W[8], W[9], W[10], W[11]);
      Affine T;
#pragma unroll
      for (int c = 0; c < 12; ++c) T.m[c] = M[c];
      float lo[3] = {CUDART_INF_F, CUDART_INF_F, CUDART_INF_F}, hi[3] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
      for (int v = 0; v < 12; ++v) {
        V3 w = xpoint(T, mk(iv.v[3 * v], iv.v[3 * v + 1], iv.v[3 * v + 2]));
        lo[0] = fminf(lo[0], w.x); lo[1] = fminf(lo[1], w.y); lo[2] = fminf(lo[2], w.z);
        hi[0] = fmaxf(hi[0], w.x); hi[1] = fmaxf(hi[1], w.y); hi[2] = fmaxf(hi[2], w.z);
      }
      float ext = fmaxf(fmaxf(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
      float mag = 0.0f;
#pragma unroll
      for (int a = 0; a < 3; ++a) mag = fmaxf(mag, fmaxf(fabsf(lo[a]), fabsf(hi[a])));
      // conservative padding for the rounding of the vertex transform
      float pad = __fmaf_rn(1e-5f, ext, 2e-6f * (mag + 1.0f));
      float* b = box + 6 * p;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float b0 = lo[a] - pad, b1 = hi[a] + pad;
        b[a] = b0;
        b[3 + a] = b1;
        float c = 0.5f * (b0 + b1);
        cmin[a] = c;
        cmax[a] = c;
        bmag = fmaxf(bmag, fmaxf(fabsf(b0), fabsf(b1)));
      }
    }
  }
  if (!FULL) {
    kept_s[threadIdx.x] = kept ? 1u : 0u;
    __syncthreads();
    // SH rows: float 3k + ch of a row is coefficient k, channel ch
    for (uint32_t i = threadIdx.x; i < cnt * 12u; i += kRecBlock) {
      const uint32_t r = i / 12u, q = i - 12u * r;
      if (!kept_s[r]) continue;
      const float* rec = rows + r * pitch + 16;
      float v[4];
#pragma unroll
      for (uint32_t c = 0; c < 4; ++c) {
        const uint32_t f = 4 * q + c, k = f / 3u, ch = f - 3u * k;
        v[c] = k < n_sh ? rec[4 * k + ch] : 0.0f;
      }
      sh[12 * (p0 + r) + q] = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
  // the block's centre bounds, and atomics only for those that move the
  // totals (an atomic of every warp on one sector takes longer than the pass)
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      cmin[a] = fminf(cmin[a], __shfl_xor_sync(0xFFFFFFFFu, cmin[a], off));
      cmax[a] = fmaxf(cmax[a], __shfl_xor_sync(0xFFFFFFFFu, cmax[a], off));
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) bmag = fmaxf(bmag, __shfl_xor_sync(0xFFFFFFFFu, bmag, off));
  if ((threadIdx.x & 31) == 0 && cmin[0] <= cmax[0]) {
    const uint4 now0 = __ldcg(reinterpret_cast<const uint4*>(bounds_ord)),
                now1 = __ldcg(reinterpret_cast<const uint4*>(bounds_ord) + 1);
    const uint32_t now[7] = {now0.x, now0.y, now0.z, now0.w, now1.x, now1.y, now1.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (f2ord(cmin[a]) < now[a]) atomicMin(&bounds_ord[a], f2ord(cmin[a]));
      if (f2ord(cmax[a]) > now[3 + a]) atomicMax(&bounds_ord[3 + a], f2ord(cmax[a]));
    }
    if (f2ord(bmag) > now[6]) atomicMax(&bounds_ord[6], f2ord(bmag));
  }
}

__device__ __forceinline__ uint32_t spread10(uint32_t v) {
  v &= 0x3FFu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

// The range of the centres that the Morton grid divides, per axis: all of it, or,
// where a few proxies far out stretch it to four times what most of them need and
// more, that part (kCore of the 1024 cells; the rest is shared out outside it).
// From 256 samples: between the 3rd and the 97th percentile, a quarter more on
// either side.  (1M Gaussians in clusters and eight at a distance of 3,500, 200x150
// from radius 60 by a warp per ray: 1.91 ms over the whole range, whose cells are
// larger than the clusters, 0.52 so.)
constexpr int kCoreSamples = 256;
constexpr float kCore = 896.0f;
__global__ void __launch_bounds__(kCoreSamples) k_core(const float* box, uint64_t n, const uint32_t* flags,
                                                       const uint32_t* bounds_ord, float* core) {
  __shared__ float c[kCoreSamples];
  const int a = blockIdx.x, i = threadIdx.x;  // a block an axis
  const uint64_t p = i * ((n + kCoreSamples - 1) / kCoreSamples);
  float x = CUDART_INF_F;
  if (p < n && flags[p]) x = 0.5f * (box[6 * p + a] + box[6 * p + 3 + a]);
  if (!(fabsf(x) < 1e30f)) x = CUDART_INF_F;
  c[i] = x;
  const int m = __syncthreads_count(x < 1e30f);
  for (int k = 2; k <= kCoreSamples; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      const int o = i ^ j;
      if (o > i && (c[i] > c[o]) == ((i & k) == 0)) {
        const float t = c[i];
        c[i] = c[o];
        c[o] = t;
      }
      __syncthreads();
    }
  if (i == 0) {
    float lo = ord2f(bounds_ord[a]), hi = ord2f(bounds_ord[3 + a]);
    if (m >= 32) {
      const float q0 = c[m * 3 / 100], q1 = c[m - 1 - m * 3 / 100], more = 0.25f * (q1 - q0);
      const float l = fmaxf(lo, q0 - more), h = fminf(hi, q1 + more);
      if (h > l && 4.0f * (h - l) < hi - lo) {
        lo = l;
        hi = h;
      }
    }
    core[a] = lo;
    core[3 + a] = hi;
  }
}

// Morton code of every kept particle's box centre, with the particle's index.
__global__ void k_morton(const float* box, uint64_t n, const uint32_t* flags, const uint32_t* slots,
                         const uint32_t* bounds_ord, const float* core, uint32_t* keys, uint32_t* vals) {
  const uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (p >= n || !flags[p]) return;
  uint32_t code = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float lo = ord2f(bounds_ord[a]), hi = ord2f(bounds_ord[3 + a]);
    float c = 0.5f * (box[6 * p + a] + box[6 * p + 3 + a]);
    float e = hi - lo;
    float u = e > 0.0f ? (c - lo) / e : 0.0f;
    u = fminf(fmaxf(u, 0.0f), 1.0f);
    uint32_t q = (uint32_t)(u * 1023.0f);
    const float l = core[a], h = core[3 + a];
    if (l > lo || h < hi) {  // below, in and above the core
      constexpr float kSide = 0.5f * (1024.0f - kCore);
      const float x = c < l ? kSide * (c - lo) / (l - lo)
                            : c < h ? kSide + kCore * (c - l) / (h - l) : kSide + kCore + kSide * (c - h) / (hi - h);
      q = (uint32_t)fminf(fmaxf(x, 0.0f), 1023.0f);
    }
    code |= spread10(q) << (2 - a);
  }
  keys[slots[p]] = code;
  vals[slots[p]] = (uint32_t)p;
}

// ------------------------------------------------------------------ scan
constexpr int kScanBlock = 512;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanBlock * kScanItems;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_sums[32];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int nw = blockDim.x >> 5;
    uint32_t s = lane < nw ? warp_sums[lane] : 0u;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, off);
      if (lane >= off) s += y;
    }
    warp_sums[lane] = s;
  }
  __syncthreads();
  uint32_t base = warp ? warp_sums[warp - 1] : 0u;
  if (total) *total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return base + x - v;
}

__global__ void k_scan_tiles(const uint32_t* in, uint32_t* out, uint64_t n, uint32_t* tile_sums) {
  uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = (base + i < n) ? in[base + i] : 0u;
    sum += v[i];
  }
  uint32_t total;
  uint32_t pre = block_exclusive_scan(sum, &total);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i < n) out[base + i] = pre;
    pre += v[i];
  }
  if (threadIdx.x == 0 && tile_sums) tile_sums[blockIdx.x] = total;
}

__global__ void k_scan_add(uint32_t* out, uint64_t n, const uint32_t* tile_offsets) {
  uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
  uint32_t add = tile_offsets[blockIdx.x];
#pragma unroll
  for (int i = 0; i < kScanItems; ++i)
    if (base + i < n) out[base + i] += add;
}

// Exclusive scan of n uint32 values (in may equal out).  Temporaries are
// stream-ordered allocations.
Err scan_exclusive(const uint32_t* in, uint32_t* out, uint64_t n, cudaStream_t st, uint64_t* launches) {
  if (n == 0) return Err{};
  uint64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles == 1) {
    k_scan_tiles<<<1, kScanBlock, 0, st>>>(in, out, n, nullptr);
    ++*launches;
    GT_CUDA_TRY(cudaGetLastError());
    return Err{};
  }
  uint32_t* sums = nullptr;
  GT_CUDA_TRY(cudaMallocAsync(&sums, tiles * sizeof(uint32_t), st));
  k_scan_tiles<<<(unsigned)tiles, kScanBlock, 0, st>>>(in, out, n, sums);
  ++*launches;
  Err e = scan_exclusive(sums, sums, tiles, st, launches);
  if (e.code == GT_OK) {
    k_scan_add<<<(unsigned)tiles, kScanBlock, 0, st>>>(out, n, sums);
    ++*launches;
  }
  cudaFreeAsync(sums, st);
  if (e.code != GT_OK) return e;
  GT_CUDA_TRY(cudaGetLastError());
  return Err{};
}

// ------------------------------------------------------------ radix sort
// Stable sort of (key, value) pairs by the low 30 bits of the key (Morton codes),
// 10 bits a pass, in one cooperative launch.  A block owns one stretch of the
// array and each of its warps a part of it, so a pass is: counts per warp and
// digit in shared memory, the blocks' counts to global memory, a grid barrier,
// every block its own offsets from these (1024 digits, one a thread, times the
// blocks), and the warps' parts to their places.  Bound by latencies (barriers,
// the chain of a warp's steps).  Four passes of five launches each took 115 us for
// 65k pairs and 162 us for 1M, this 50 and 118 us (at 1M the blocks read one
// another's counts, 90 MB a pass from L2).
constexpr int kRsBits = 10, kRsDigits = 1 << kRsBits, kRsPasses = 3, kRsThreads = 1024, kRsWarps = kRsThreads / 32;
static_assert(kRsDigits == kRsThreads, "one digit a thread");

__global__ void __launch_bounds__(kRsThreads) k_radix_sort(uint32_t* ka, uint32_t* va, uint32_t* kb, uint32_t* vb,
                                                           uint32_t n, uint32_t per_warp, uint32_t* hist) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  extern __shared__ uint32_t cnt[];  // [warp][digit]
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d = threadIdx.x;
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t* mine = cnt + warp * kRsDigits;
  const uint64_t first = ((uint64_t)blockIdx.x * kRsWarps + warp) * per_warp;
  const uint32_t begin = (uint32_t)(first < n ? first : n), end = min(n - begin, per_warp) + begin;
  for (int pass = 0; pass < kRsPasses; ++pass) {
    const int shift = pass * kRsBits;
    for (uint32_t q = lane; q < kRsDigits; q += 32) mine[q] = 0;
    __syncwarp();
#pragma unroll 4
    for (uint32_t i = begin + lane; i < end; i += 32)
      atomicAdd(&mine[(__ldcg(ka + i) >> shift) & (kRsDigits - 1)], 1u);
    __syncthreads();
    uint32_t sum = 0;
#pragma unroll 8
    for (int w = 0; w < kRsWarps; ++w) {
      const uint32_t x = cnt[w * kRsDigits + d];
      cnt[w * kRsDigits + d] = sum;
      sum += x;
    }
    hist[blockIdx.x * kRsDigits + d] = sum;
    grid.sync();
    uint32_t before = 0, total = 0;
#pragma unroll 8
    for (uint32_t b = 0; b < gridDim.x; ++b) {
      const uint32_t x = __ldcg(hist + b * kRsDigits + d);
      if (b < blockIdx.x) before += x;
      total += x;
    }
    before += block_exclusive_scan(total, nullptr);
#pragma unroll 8
    for (int w = 0; w < kRsWarps; ++w) cnt[w * kRsDigits + d] += before;
    __syncthreads();
    uint32_t next_key = 0, next_val = 0;  // loaded a step ahead
    if (begin + lane < end) {
      next_key = __ldcg(ka + begin + lane);
      next_val = __ldcg(va + begin + lane);
    }
    for (uint32_t i0 = begin; i0 < end; i0 += 32) {
      const uint32_t i = i0 + lane, key = next_key, val = next_val;
      if (i < end && end - i > 32) {
        next_key = __ldcg(ka + i + 32);
        next_val = __ldcg(va + i + 32);
      }
      const uint32_t digit = i < end ? (key >> shift) & (kRsDigits - 1) : kRsDigits;  // kRsDigits: no item
      const uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
      const uint32_t rank = __popc(peers & lt_mask);
      uint32_t at = 0;
      if (i < end) at = mine[digit] + rank;
      __syncwarp();
      if (i < end) {
        if (rank == 0) mine[digit] = at + __popc(peers);
        kb[at] = key;
        vb[at] = val;
      }
      __syncwarp();
    }
    grid.sync();
    uint32_t* t = ka;
    ka = kb;
    kb = t;
    t = va;
    va = vb;
    vb = t;
  }
}

// Sorts in place of keys and vals, which may come back as other buffers of n.
static Err radix_sort(uint32_t*& keys, uint32_t*& vals, uint32_t n, cudaStream_t st, uint64_t* launches) {
  if (n <= 1) return Err{};
  int dev = 0, sms = 0;
  GT_CUDA_TRY(cudaGetDevice(&dev));
  GT_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const size_t smem = sizeof(uint32_t) * kRsWarps * kRsDigits;
  GT_CUDA_TRY(cudaFuncSetAttribute(k_radix_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const uint32_t grid = std::min<uint32_t>((uint32_t)std::max(1, sms), (n + kRsThreads - 1) / kRsThreads);
  uint32_t per_warp = (uint32_t)(((uint64_t)n + (uint64_t)grid * kRsThreads - 1) / ((uint64_t)grid * kRsThreads)) * 32u;
  uint32_t *k2 = nullptr, *v2 = nullptr, *hist = nullptr;
  GT_CUDA_TRY(cudaMallocAsync(&k2, (size_t)n * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&v2, (size_t)n * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&hist, (size_t)grid * kRsDigits * 4, st));
  void* args[] = {(void*)&keys, (void*)&vals, (void*)&k2, (void*)&v2, (void*)&n, (void*)&per_warp, (void*)&hist};
  const cudaError_t e =
      cudaLaunchCooperativeKernel((const void*)k_radix_sort, dim3(grid), dim3(kRsThreads), args, smem, st);
  ++*launches;
  if (kRsPasses % 2) {  // the sorted pairs are in the second buffers
    std::swap(keys, k2);
    std::swap(vals, v2);
  }
  cudaFreeAsync(k2, st);
  cudaFreeAsync(v2, st);
  cudaFreeAsync(hist, st);
  GT_CUDA_TRY(e);
  return Err{};
}

// -------------------------------------------------------------- hierarchy
__device__ __forceinline__ int kdelta(const uint32_t* k, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  uint32_t a = k[i], b = k[j];
  if (a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
  return __clz(a ^ b);
}

// Karras 2012, "Maximizing parallelism in the construction of BVHs, octrees
// and k-d trees": internal node i covers a key range found by one exponential
// and two binary searches on the longest common prefix.
__global__ void k_karras(const uint32_t* keys, int n, float4* nodes, uint32_t* parent_int, uint32_t* parent_leaf) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  int d = (kdelta(keys, n, i, i + 1) - kdelta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  int dmin = kdelta(keys, n, i, i - d);
  int lmax = 2;
  while (kdelta(keys, n, i, i + lmax * d) > dmin) lmax *= 2;
  int l = 0;
  for (int t = lmax / 2; t >= 1; t /= 2)
    if (kdelta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  int j = i + l * d;
  int dnode = kdelta(keys, n, i, j);
  int s = 0, t = l;
  do {
    t = (t + 1) / 2;
    if (kdelta(keys, n, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  int gamma = i + s * d + min(d, 0);
  int lo = min(i, j), hi = max(i, j);
  uint32_t c0 = (lo == gamma) ? (kLeafBit | (uint32_t)gamma) : (uint32_t)gamma;
  uint32_t c1 = (hi == gamma + 1) ? (kLeafBit | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
  nodes[4 * (size_t)i + 3] = make_float4(__uint_as_float(c0), __uint_as_float(c1), 0.f, 0.f);
  if (c0 & kLeafBit) parent_leaf[gamma] = (uint32_t)i; else parent_int[gamma] = (uint32_t)i;
  if (c1 & kLeafBit) parent_leaf[gamma + 1] = (uint32_t)i; else parent_int[gamma + 1] = (uint32_t)i;
  if (i == 0) parent_int[0] = kInvalid;
}

// Leaf records in leaf order: world-to-object map, particle index, box.
__global__ void k_leaves(const uint32_t* sorted_pidx, uint32_t m, const float4* w2o_by_particle,
                         const float* box_by_particle, float4* w2o, uint32_t* leaf_pidx, float* leaf_box) {
  uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint32_t p = sorted_pidx[j];
#pragma unroll
  for (int q = 0; q < 3; ++q) w2o[3 * (size_t)j + q] = __ldg(w2o_by_particle + 3 * (size_t)p + q);
  leaf_pidx[j] = p;
  const float2* b = reinterpret_cast<const float2*>(box_by_particle) + 3 * (size_t)p;
  float2* o = reinterpret_cast<float2*>(leaf_box) + 3 * (size_t)j;
#pragma unroll
  for (int a = 0; a < 3; ++a) o[a] = __ldg(b + a);
}

__device__ __forceinline__ void child_box(uint32_t ref, const float* leaf_box, const float* ibox, float b[6]) {
  const float* src = (ref & kLeafBit) ? leaf_box + 6 * (size_t)(ref & ~kLeafBit) : ibox + 6 * (size_t)ref;
#pragma unroll
  for (int a = 0; a < 6; ++a) b[a] = __ldcg(src + a);
}

// Bottom-up refit: the second child to arrive at a node writes its boxes.
__global__ void k_refit(uint32_t m, const float* leaf_box, float* ibox, float4* nodes, const uint32_t* parent_int,
                        const uint32_t* parent_leaf, uint32_t* arrive) {
  uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  uint32_t node = parent_leaf[j];
  uint32_t guard = 0;
  while (node != kInvalid && guard++ < 4096u) {
    __threadfence();
    if (atomicAdd(&arrive[node], 1u) == 0u) return;
    float4 f3 = __ldcg(nodes + 4 * (size_t)node + 3);
    uint32_t c0 = __float_as_uint(f3.x), c1 = __float_as_uint(f3.y);
    float b0[6], b1[6];
    child_box(c0, leaf_box, ibox, b0);
    child_box(c1, leaf_box, ibox, b1);
    nodes[4 * (size_t)node + 0] = make_float4(b0[0], b0[3], b0[1], b0[4]);
    nodes[4 * (size_t)node + 1] = make_float4(b1[0], b1[3], b1[1], b1[4]);
    nodes[4 * (size_t)node + 2] = make_float4(b0[2], b0[5], b1[2], b1[5]);
    float* ib = ibox + 6 * (size_t)node;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      ib[a] = fminf(b0[a], b1[a]);
      ib[3 + a] = fmaxf(b0[3 + a], b1[3 + a]);
    }
    node = parent_int[node];
  }
}

// Tree check before any traversal: every child reference in range and every
// node reached by exactly one parent (the root by none).
__global__ void k_check_children(uint32_t m, const float4* nodes, uint32_t* refcount, const uint32_t* root,
                                 uint32_t* bad) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i + 1 >= m) return;
  float4 f3 = nodes[4 * (size_t)i + 3];
  uint32_t c[2] = {__float_as_uint(f3.x), __float_as_uint(f3.y)};
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint32_t r = c[q];
    if (r & kLeafBit) {
      uint32_t j = r & ~kLeafBit;
      if (j >= m) atomicOr(bad, 1u); else atomicAdd(&refcount[(m - 1) + j], 1u);
    } else {
      if (r >= m - 1 || r == *root) atomicOr(bad, 2u); else atomicAdd(&refcount[r], 1u);
    }
  }
}
__global__ void k_check_counts(uint32_t total, const uint32_t* refcount, const uint32_t* root, uint32_t* bad) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  uint32_t expect = i == *root ? 0u : 1u;
  if (refcount[i] != expect) atomicOr(bad, 4u);
}

__global__ void k_depth(uint32_t m, const uint32_t* parent_int, const uint32_t* parent_leaf, uint32_t* depth) {
  uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  uint32_t d = 0, node = parent_leaf[j];
  while (node != kInvalid && d < 100000u) {
    ++d;
    node = parent_int[node];
  }
  atomicMax(depth, d);
}

// ------------------------------------------------------------- BVH8 collapse
// Greedy collapse of the binary hierarchy into 8-wide nodes: a node starts
// with the two children of a binary node and repeatedly opens its internal
// entry of largest surface area until it holds 8 entries or only leaves.
// Each binary internal node ends up inside exactly one 8-wide node, and
// every 8-wide node opens at least one binary node, so there are fewer
// 8-wide nodes than binary internal nodes.
//
// 8-wide node layout: 8 child records of 32 bytes (2 float4):
//   f0 = (lo.x, lo.y, lo.z, hi.x), f1 = (hi.y, hi.z, ref, 0)
// ref = kLeafBit | j for leaf j, an 8-wide node index, or kInvalid (empty
// slot, with an empty box).
__device__ __forceinline__ float half_area(const float b[6]) {
  float x = b[3] - b[0], y = b[4] - b[1], z = b[5] - b[2];
  return x * y + y * z + z * x;
}

// Child c (0 or 1) of binary node i.
__device__ __forceinline__ void binary_child(const float4* bn, uint32_t i, uint32_t c, float b[6], uint32_t& ref) {
  const float4 xy = __ldg(bn + 4 * (size_t)i + c), z = __ldg(bn + 4 * (size_t)i + 2), r = __ldg(bn + 4 * (size_t)i + 3);
  b[0] = xy.x;
  b[3] = xy.y;
  b[1] = xy.z;
  b[4] = xy.w;
  b[2] = c ? z.z : z.x;
  b[5] = c ? z.w : z.y;
  ref = __float_as_uint(c ? r.y : r.x);
}

// The whole collapse in one cooperative launch: level by level, eight lanes a
// node (one entry each), the grid in step between levels.  The nodes of a
// level follow each other, so a node's index is also its place in the work
// list; bin_of[i] is the binary node 8-wide node i starts from.  counts: how
// many nodes a level has made so far, three in turn.  Bound by the dependent
// loads of up to six openings a node.  (B200, 1M proxies: a thread a node and a
// launch and a host round trip a level took 312 us of kernels in 15 launches;
// this takes 215 us in one.)
__global__ void __launch_bounds__(128) k_collapse8(const float4* __restrict__ bn, float4* __restrict__ nodes8,
                                                   const float* __restrict__ ibox, const uint32_t* root, float* root_box,
                                                   uint32_t* bin_of, uint32_t* counts, uint32_t* out,
                                                   uint32_t max_nodes8) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31, gl = lane & 7, g0 = lane & 24;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, n_warps = (gridDim.x * blockDim.x) >> 5;
  if (blockIdx.x == 0 && threadIdx.x < 6) root_box[threadIdx.x] = ibox[6 * (size_t)*root + threadIdx.x];
  uint32_t start = 0, end = 1;
  for (uint32_t level = 0; start < end; ++level) {
    if (blockIdx.x == 0 && threadIdx.x == 0) counts[(level + 1) % 3] = 0;
    uint32_t* made = &counts[level % 3];
    for (uint32_t first = start + 4 * warp; first < end; first += 4 * n_warps) {
      const uint32_t i = first + (lane >> 3);
      const bool on = i < end;
      float b[6] = {1e30f, 1e30f, 1e30f, -1e30f, -1e30f, -1e30f};
      uint32_t ref = kInvalid;
      const uint32_t bi = i == 0 ? *root : on ? __ldcg(bin_of + i) : 0u;
      if (on && gl < 2) binary_child(bn, bi, gl, b, ref);
      uint32_t cnt = 2;
      for (int open = 0; open < 6; ++open) {
        float area = ref == kInvalid || (ref & kLeafBit) ? -1.0f : half_area(b);
        if (!(area >= 0.0f)) area = -1.0f;
        uint32_t at = gl;
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) {
          const float oa = __shfl_xor_sync(kAll, area, off);
          const uint32_t ob = __shfl_xor_sync(kAll, at, off);
          if (oa > area || (oa == area && ob < at)) {
            area = oa;
            at = ob;
          }
        }
        const uint32_t parent = __shfl_sync(kAll, ref, g0 + at);
        if (area >= 0.0f) {
          if (gl == at) binary_child(bn, parent, 0, b, ref);
          if (gl == cnt) binary_child(bn, parent, 1, b, ref);
          ++cnt;
        }
        if (!__any_sync(kAll, area >= 0.0f)) break;
      }
      const bool inner = on && ref != kInvalid && !(ref & kLeafBit);
      const uint32_t im = __ballot_sync(kAll, inner);
      uint32_t base = 0;
      if (lane == 0 && im) base = atomicAdd(made, (uint32_t)__popc(im));
      base = __shfl_sync(kAll, base, 0);
      if (inner) {
        const uint32_t child = end + base + __popc(im & lt_mask);
        if (child >= max_nodes8) {
          out[1] = 1u;
          ref = 0u;
        } else {
          __stcg(bin_of + child, ref);
          ref = child;
        }
      }
      if (on) {
        float4* o = nodes8 + 16 * (size_t)i + 2 * gl;
        o[0] = make_float4(b[0], b[1], b[2], b[3]);
        o[1] = make_float4(b[4], b[5], __uint_as_float(ref), 0.f);
      }
    }
    __threadfence();
    grid.sync();
    start = end;
    end = min(end + *reinterpret_cast<volatile uint32_t*>(made), max_nodes8);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[0] = end;
}

// Collapses the binary hierarchy (m leaves) into `*out8` (exactly sized).
static Err collapse_bvh8(const float4* bn, const float* ibox, const float* leaf_box, uint32_t m, uint32_t* bounds,
                         cudaStream_t st, float4** out8, uint32_t* n_nodes8, uint64_t* launches) {
  uint32_t cap = std::max<uint32_t>(m > 1 ? m - 1 : 1, 1);
  float4* tmp = nullptr;
  uint32_t* buf = nullptr;  // 5 words: level counts, result; then bin_of
  GT_CUDA_TRY(cudaMallocAsync(&tmp, (size_t)cap * 16 * sizeof(float4), st));
  GT_CUDA_TRY(cudaMallocAsync(&buf, ((size_t)cap + 8) * 4, st));
  uint32_t total = 1;
  if (m == 1) {
    float lb[6];
    GT_CUDA_TRY(cudaMemcpyAsync(lb, leaf_box, sizeof lb, cudaMemcpyDeviceToHost, st));
    GT_CUDA_TRY(cudaStreamSynchronize(st));
    auto bits = [](uint32_t u) {
      float f;
      memcpy(&f, &u, 4);
      return f;
    };
    float4 host[16];
    host[0] = make_float4(lb[0], lb[1], lb[2], lb[3]);
    host[1] = make_float4(lb[4], lb[5], bits(kLeafBit | 0u), 0.f);
    for (int q = 1; q < 8; ++q) {
      host[2 * q] = make_float4(1e30f, 1e30f, 1e30f, -1e30f);
      host[2 * q + 1] = make_float4(-1e30f, -1e30f, bits(kInvalid), 0.f);
    }
    GT_CUDA_TRY(cudaMemcpyAsync(tmp, host, sizeof host, cudaMemcpyHostToDevice, st));
  } else {
    GT_CUDA_TRY(cudaMemsetAsync(buf, 0, 8 * 4, st));  // counts and result
    int dev = 0, sms = 0, per_sm = 0;
    GT_CUDA_TRY(cudaGetDevice(&dev));
    GT_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_collapse8, 128, 0));
    // (a level has at most m / 4 or so nodes, 16 a block)
    const unsigned grid =
        (unsigned)std::max<uint32_t>(1, std::min<uint32_t>((uint32_t)(sms * std::min(per_sm, 8)), m / 64 + 1));
    uint32_t* counts = buf;
    uint32_t* out = buf + 4;
    uint32_t* bin_of = buf + 8;
    const uint32_t* root = bounds + 8;
    float* root_box = reinterpret_cast<float*>(bounds + 9);
    void* args[] = {(void*)&bn, (void*)&tmp, (void*)&ibox, (void*)&root, (void*)&root_box, (void*)&bin_of, (void*)&counts, (void*)&out, (void*)&cap};
    GT_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)k_collapse8, dim3(grid), dim3(128), args, 0, st));
    ++*launches;
    uint32_t c[2];
    GT_CUDA_TRY(cudaMemcpyAsync(c, out, sizeof c, cudaMemcpyDeviceToHost, st));
    GT_CUDA_TRY(cudaStreamSynchronize(st));
    if (c[1]) return Err{GT_ERR_CUDA, "internal error: 8-wide collapse exceeded its node bound"};
    total = c[0];
  }
  GT_CUDA_TRY(cudaMallocAsync(out8, (size_t)total * 16 * sizeof(float4), st));
  GT_CUDA_TRY(cudaMemcpyAsync(*out8, tmp, (size_t)total * 16 * sizeof(float4), cudaMemcpyDeviceToDevice, st));
  cudaFreeAsync(tmp, st);
  cudaFreeAsync(buf, st);
  *n_nodes8 = total;
  return Err{};
}

// -------------------------------------------------------------- driver
// The scene's buffers come from the device's stream-ordered pool (which the
// context keeps from releasing), so a scene built after another was freed
// reuses its memory instead of mapping new pages.
void free_scene(SceneBuffers* b, cudaStream_t st) {
  for (void* p : {(void*)b->nodes, (void*)b->nodes8, (void*)b->w2o, (void*)b->leaf_pidx, (void*)b->shade,
                  (void*)b->sh, (void*)b->params})
    if (p) cudaFreeAsync(p, st);
  *b = SceneBuffers{};
}

static inline unsigned grid_for(uint64_t n, unsigned block) { return (unsigned)((n + block - 1) / block); }

Err build_scene(const void* packed_dev, uint64_t n, uint32_t stride, double alpha_min, cudaStream_t st,
                SceneBuffers* out, uint64_t* launches, bool fast_build, const double* act64) {
  SceneBuffers b;
  b.n_sh = std::min<uint32_t>(16u, (stride - 64u) / 16u);
  const uint8_t* packed = static_cast<const uint8_t*>(packed_dev);
  if (n == 0) {
    *out = b;
    return Err{};
  }
  if (n >= (1ull << 31)) return Err{GT_ERR_INVALID_ARG, "scene larger than 2^31 particles"};
  // shading records (every particle slot; only kept ones are written/read)
  GT_CUDA_TRY(cudaMallocAsync(&b.shade, n * 3 * sizeof(float4), st));
  GT_CUDA_TRY(cudaMallocAsync(&b.sh, n * 12 * sizeof(float4), st));
  GT_CUDA_TRY(cudaMallocAsync(&b.params, n * 2 * sizeof(float4), st));
  b.bytes += n * 17 * sizeof(float4);
  uint32_t *flags = nullptr, *slots = nullptr, *bounds = nullptr;
  float *box = nullptr;
  float4* w2o_p = nullptr;
  GT_CUDA_TRY(cudaMallocAsync(&flags, n * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&slots, n * 4, st));
  // centre bounds [0, 6), largest coordinate [6], tree check [7], binary root [8], its box [9, 15), core [16, 22)
  GT_CUDA_TRY(cudaMallocAsync(&bounds, 32 * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&box, n * 6 * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&w2o_p, n * 3 * sizeof(float4), st));
  const unsigned B = 256;
  {
    uint32_t init[16] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
    GT_CUDA_TRY(cudaMemcpyAsync(bounds, init, sizeof init, cudaMemcpyHostToDevice, st));
  }
  IcoVerts iv;
  ico_vertices(iv.v);
  if (stride == 320 && (uintptr_t)packed % 16 == 0) {
    k_records<true><<<grid_for(n, kRecBlock), kRecBlock, kRecBlock * 17 * sizeof(float), st>>>(
        packed, n, stride, b.n_sh, alpha_min, act64, iv, flags, b.shade, b.sh, b.params, w2o_p, box, bounds);
  } else {
    const size_t smem = (size_t)kRecBlock * (std::min(stride / 4u, 16u + 4u * b.n_sh) | 1u) * sizeof(float);
    k_records<false><<<grid_for(n, kRecBlock), kRecBlock, smem, st>>>(
        packed, n, stride, b.n_sh, alpha_min, act64, iv, flags, b.shade, b.sh, b.params, w2o_p, box, bounds);
  }
  ++*launches;
  GT_CUDA_TRY(cudaGetLastError());
  Err e = scan_exclusive(flags, slots, n, st, launches);
  if (e.code != GT_OK) return e;
  uint32_t last_flag = 0, last_slot = 0;
  GT_CUDA_TRY(cudaMemcpyAsync(&last_flag, flags + (n - 1), 4, cudaMemcpyDeviceToHost, st));
  GT_CUDA_TRY(cudaMemcpyAsync(&last_slot, slots + (n - 1), 4, cudaMemcpyDeviceToHost, st));
  GT_CUDA_TRY(cudaStreamSynchronize(st));
  uint32_t m = last_slot + last_flag;
  b.n_kept = m;
  auto drop_first = [&]() {
    cudaFreeAsync(flags, st);
    cudaFreeAsync(slots, st);
    cudaFreeAsync(bounds, st);
    cudaFreeAsync(box, st);
    cudaFreeAsync(w2o_p, st);
  };
  if (m == 0) {
    drop_first();
    GT_CUDA_TRY(cudaStreamSynchronize(st));
    *out = b;
    return Err{};
  }
  uint32_t *keys = nullptr, *vals = nullptr;
  GT_CUDA_TRY(cudaMallocAsync(&keys, (size_t)m * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&vals, (size_t)m * 4, st));
  float* core = reinterpret_cast<float*>(bounds + 16);
  k_core<<<3, kCoreSamples, 0, st>>>(box, n, flags, bounds, core);
  k_morton<<<grid_for(n, B), B, 0, st>>>(box, n, flags, slots, bounds, core, keys, vals);
  *launches += 2;
  GT_CUDA_TRY(cudaGetLastError());
  e = radix_sort(keys, vals, m, st, launches);
  if (e.code != GT_OK) return e;
  // scene records
  uint32_t n_int = m > 1 ? m - 1 : 0;
  GT_CUDA_TRY(cudaMallocAsync(&b.w2o, (size_t)m * 3 * sizeof(float4), st));
  GT_CUDA_TRY(cudaMallocAsync(&b.leaf_pidx, (size_t)m * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&b.nodes, (size_t)std::max<uint32_t>(n_int, 1) * 4 * sizeof(float4), st));
  b.bytes += (uint64_t)m * (3 * sizeof(float4) + 4) + (uint64_t)std::max<uint32_t>(n_int, 1) * 4 * sizeof(float4);
  float *leaf_box = nullptr, *ibox = nullptr;
  uint32_t *parent_int = nullptr, *parent_leaf = nullptr, *arrive = nullptr, *depth = nullptr;
  GT_CUDA_TRY(cudaMallocAsync(&leaf_box, (size_t)m * 6 * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&ibox, (size_t)std::max<uint32_t>(n_int, 1) * 6 * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&parent_int, (size_t)std::max<uint32_t>(n_int, 1) * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&parent_leaf, (size_t)m * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&arrive, (size_t)std::max<uint32_t>(n_int, 1) * 4, st));
  GT_CUDA_TRY(cudaMallocAsync(&depth, 4, st));
  GT_CUDA_TRY(cudaMemsetAsync(arrive, 0, (size_t)std::max<uint32_t>(n_int, 1) * 4, st));
  GT_CUDA_TRY(cudaMemsetAsync(depth, 0, 4, st));
  k_leaves<<<grid_for(m, B), B, 0, st>>>(vals, m, w2o_p, box, b.w2o, b.leaf_pidx, leaf_box);
  ++*launches;
  if (m > 1) {
    if (fast_build) {
      k_karras<<<grid_for(n_int, B), B, 0, st>>>(keys, (int)m, b.nodes, parent_int, parent_leaf);
      k_refit<<<grid_for(m, B), B, 0, st>>>(m, leaf_box, ibox, b.nodes, parent_int, parent_leaf, arrive);
      *launches += 2;
    } else {
      Err pe = build_ploc(keys, leaf_box, m, st, b.nodes, ibox, parent_int, parent_leaf, bounds + 8, launches);
      if (pe.code != GT_OK) return pe;
    }
    k_depth<<<grid_for(m, B), B, 0, st>>>(m, parent_int, parent_leaf, depth);
    *launches += 1;
    // structural check: refcount over [internal 0..m-2 | leaves 0..m-1]
    uint32_t* refc = nullptr;
    GT_CUDA_TRY(cudaMallocAsync(&refc, (size_t)(2 * m - 1) * 4, st));
    GT_CUDA_TRY(cudaMemsetAsync(refc, 0, (size_t)(2 * m - 1) * 4, st));
    k_check_children<<<grid_for(n_int, B), B, 0, st>>>(m, b.nodes, refc, bounds + 8, bounds + 7);
    k_check_counts<<<grid_for(2 * m - 1, B), B, 0, st>>>(2 * m - 1, refc, bounds + 8, bounds + 7);
    *launches += 2;
    cudaFreeAsync(refc, st);
    b.root = 0;
  } else {
    b.root = kLeafBit | 0u;
  }
  GT_CUDA_TRY(cudaGetLastError());
  {
    Err ce = collapse_bvh8(b.nodes, ibox, leaf_box, m, bounds, st, &b.nodes8, &b.n_nodes8, launches);
    if (ce.code != GT_OK) return ce;
    b.bytes += (uint64_t)b.n_nodes8 * 16 * sizeof(float4);
    // traversal reads only the 8-wide nodes: the binary hierarchy goes
    cudaFreeAsync(b.nodes, st);
    b.nodes = nullptr;
    b.bytes -= (uint64_t)std::max<uint32_t>(n_int, 1) * 4 * sizeof(float4);
  }
  float rb[6];
  uint32_t bo[16];
  if (m == 1) GT_CUDA_TRY(cudaMemcpyAsync(rb, leaf_box, sizeof rb, cudaMemcpyDeviceToHost, st));
  GT_CUDA_TRY(cudaMemcpyAsync(&b.depth, depth, 4, cudaMemcpyDeviceToHost, st));
  GT_CUDA_TRY(cudaMemcpyAsync(bo, bounds, sizeof bo, cudaMemcpyDeviceToHost, st));
  GT_CUDA_TRY(cudaStreamSynchronize(st));
  if (m > 1) memcpy(rb, bo + 9, sizeof rb);
  for (int a = 0; a < 6; ++a) b.bounds[a] = rb[a];
  float mag = 0.0f;
  for (int a = 0; a < 6; ++a) mag = std::max(mag, std::fabs(rb[a]));
  b.scene_mag = mag;
  drop_first();
  cudaFreeAsync(keys, st);
  cudaFreeAsync(vals, st);
  cudaFreeAsync(leaf_box, st);
  cudaFreeAsync(ibox, st);
  cudaFreeAsync(parent_int, st);
  cudaFreeAsync(parent_leaf, st);
  cudaFreeAsync(arrive, st);
  cudaFreeAsync(depth, st);
  GT_CUDA_TRY(cudaStreamSynchronize(st));
  if (bo[7] != 0) {
    free_scene(&b, st);
    return Err{GT_ERR_CUDA, "internal error: the built hierarchy is not a tree"};
  }
  if (b.depth > kMaxDepth) {
    free_scene(&b, st);
    // (the radix tree is at most 30 code bits and 31 index bits deep)
    if (!fast_build) return build_scene(packed_dev, n, stride, alpha_min, st, out, launches, true, act64);
    return Err{GT_ERR_UNSUPPORTED, "BVH deeper than the traversal stack allows"};
  }
  *out = b;
  return Err{};
}

}  // namespace gt
