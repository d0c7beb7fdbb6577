// gt_warp.cuh — warp-cooperative traversal of the 8-wide BVH, shared by the
// forward tracer (gt_trace.cu) and the adjoint (gt_backward.cu).
//
//   * traversal: up to 4 nodes are popped at once and their 32 children are
//     box-tested by the 32 lanes; hit inner children are sorted by entry
//     distance (warp bitonic sort) and pushed far-to-near onto a per-warp
//     stack in shared memory; hit leaves go to a per-warp leaf queue;
//   * leaves: 32 queued proxies at a time go through the bounding-sphere
//     filter, one per lane; those that pass wait in a second queue, and
//     kSurvivors of them at a time get the exact object-space face tests of
//     the reference (gt_trace_common.cuh), one per lane;
//   * k-buffer: lane i holds the i-th closest hit (t, particle) found so far;
//     a hit is inserted with one ballot and one shuffle.
#pragma once

#include <math_constants.h>

#include "gt_device.cuh"
#include "gt_internal.cuh"
#include "gt_trace_common.cuh"

namespace gt {

constexpr int kWarpsPerBlock = 4;
constexpr int kLeafQueue = 96;   // leaf queue entries per warp (<= 63 in use)
constexpr int kMaxHitsPerProxy = 6;
constexpr int kSurvivors = 24;   // face-test batch of the two-phase leaf test
constexpr uint32_t kFull = 0xFFFFFFFFu;

struct WarpScratch {
  uint32_t snode[kWarpStack];
  float st[kWarpStack];
  uint32_t leafq[kLeafQueue];
  float leaft[kLeafQueue];
  uint32_t svj[64];  // proxies that passed the sphere filter, waiting for the face tests
  float svt[64];     // (< kSurvivors + 32 in use)
  uint32_t pop[4];  // nodes taken by the current pop (lanes 8s..8s+7 test pop[s])
  float hq[kMaxHitsPerProxy][32];  // hits of each lane's proxy, column per lane
  RayStats stats;                  // the warp's work counters (lane 0 writes)
  FaceRows faces;                  // the caller fills them
  float rs[4];                     // warp-uniform ray state parked during a traversal
  uint32_t ru[8];
};

struct HitOut {
  uint32_t* pidx;   // [slot][max_entries]
  float* t;
  float* alpha;
  uint32_t* count;  // [slot]
  uint32_t* rounds; // [slot]
  float4* rgba;     // [slot] or null
  uint32_t max_entries;
};

// Sorts lanes [0, w) ascending by key, w = the power of two >= m (m <= 32);
// keys of lanes >= m are +inf.
__device__ __forceinline__ void warp_sort_prefix(float& key, uint32_t& val, uint32_t lane, int m) {
  const int w = m <= 2 ? 2 : m <= 4 ? 4 : m <= 8 ? 8 : m <= 16 ? 16 : 32;
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1) {
    if (k > w) break;
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      float ok = __shfl_xor_sync(kFull, key, j);
      uint32_t ov = __shfl_xor_sync(kFull, val, j);
      bool up = (lane & k) == 0;
      bool lower = (lane & j) == 0;
      bool take = (lower == up) ? (ok < key) : (ok > key);
      if (take) {
        key = ok;
        val = ov;
      }
    }
  }
}

// Warp k-buffer of 32*NB entries ascending in (t, particle index): entry
// 32*j + lane lives in lane `lane`, slot j.  Unused entries are (t_max,
// kInvalid), which sort after every hit.
template <int NB>
struct KBuf {
  float t[NB];
  uint32_t p[NB];
};

template <int NB>
__device__ __forceinline__ void kbuf_init(KBuf<NB>& b, float t_max) {
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    b.t[j] = t_max;
    b.p[j] = kInvalid;
  }
}

// Value of entry idx (warp-uniform idx < 32*NB), broadcast to all lanes.
// (One shuffle per slot: selecting the slot first with a runtime index made
// the compiler move the whole buffer to local memory.)
template <int NB>
__device__ __forceinline__ float kbuf_t_at(const KBuf<NB>& b, int idx) {
  float v = __shfl_sync(kFull, b.t[0], idx & 31);
#pragma unroll
  for (int j = 1; j < NB; ++j) {
    const float x = __shfl_sync(kFull, b.t[j], idx & 31);
    v = (idx >> 5) == j ? x : v;
  }
  return v;
}

// Inserts (t, p): entries greater than the hit form a suffix that moves up
// by one position (the last entry drops out).
template <int NB>
__device__ __forceinline__ void kbuf_insert(KBuf<NB>& b, float t, uint32_t p, uint32_t lane) {
  bool moved = false;  // warp-uniform: the hit went into an earlier slot
  float ct = 0.f;      // lane 31's entry of the previous slot, before the move
  uint32_t cp = 0;
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    if (moved) {
      float ut = __shfl_up_sync(kFull, b.t[j], 1);
      uint32_t up = __shfl_up_sync(kFull, b.p[j], 1);
      if (j + 1 < NB) {
        const float nt = __shfl_sync(kFull, b.t[j], 31);
        const uint32_t np = __shfl_sync(kFull, b.p[j], 31);
        if (lane == 0) {
          ut = ct;
          up = cp;
        }
        ct = nt;
        cp = np;
      } else if (lane == 0) {
        ut = ct;
        up = cp;
      }
      b.t[j] = ut;
      b.p[j] = up;
    } else {
      const bool after = t < b.t[j] || (t == b.t[j] && p < b.p[j]);
      const uint32_t m = __ballot_sync(kFull, after);
      if (m) {
        const int pos = __ffs(m) - 1;
        if (j + 1 < NB) {
          ct = __shfl_sync(kFull, b.t[j], 31);
          cp = __shfl_sync(kFull, b.p[j], 31);
        }
        const float ut = __shfl_up_sync(kFull, b.t[j], 1);
        const uint32_t up = __shfl_up_sync(kFull, b.p[j], 1);
        if ((int)lane > pos) {
          b.t[j] = ut;
          b.p[j] = up;
        }
        if ((int)lane == pos) {
          b.t[j] = t;
          b.p[j] = p;
        }
        moved = true;
      }
    }
  }
}

// Modes of one traversal.
enum TraverseMode { kCollect = 0, kClosestAny = 1, kCountFront = 2 };

// Warp-cooperative traversal from the root with interval (tlo, t_max).
//   kCollect:    the closest front-face hits go into the k-buffer kb
//   kClosestAny: the closest hit of any facing goes into entry 0 of kb
//   kCountFront: every front-face hit is counted into st.anyhits
// Far bound of the box tests: entry kbuf-1 of the buffer (kCollect; the
// entries past it are not exact), entry 0 (kClosestAny) or t_max
// (kCountFront).  leaf_batch: queued leaves that trigger a batch of proxy
// tests (<= 32).
template <int MODE, int NB>
__device__ __forceinline__ void traverse8(const SceneDev& S, const FaceTable& F, WarpScratch& W, V3 o, V3 d,
                                          const BoxRay& br, float tlo, float t_max, KBuf<NB>& kb,
                                          RayStats& st, uint32_t& status, uint32_t lane,
                                          int kbuf = 32 * NB, int leaf_batch = 32) {
  if (S.n_kept == 0) return;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const int cull = MODE == kClosestAny ? 0 : kbuf - 1;  // the entry that bounds the search
  int sp = 0, nq = 0;
  int ns = 0;  // proxies that passed the sphere filter, waiting for the face tests
  if (lane == 0) {
    W.snode[0] = 0;
    W.st[0] = -CUDART_INF_F;
  }
  sp = 1;
  __syncwarp();
  float thi = MODE == kCountFront ? t_max : kbuf_t_at(kb, cull);
  uint32_t iters = 0;
  const uint32_t max_iters = min(4u * S.n_kept + 64u, F.lim_steps);
  while (true) {
    if (++iters > max_iters) {
      status |= kStatusVisitCap;
      return;
    }
    // pop: lanes 0..7 read the top 8 stack entries at once and the first
    // (top-most) entries still in range are taken, up to 4 in all, through a
    // 4-slot array in shared memory; out-of-range entries above the last one
    // taken are dropped (the far bound only shrinks).  __fns is avoided: it is
    // a software loop and made this step slower than a serial pop.
    int np = 0;
    while (np < 4 && sp > 0) {
      const int avail = sp < 8 ? sp : 8;
      bool ok = false;
      uint32_t en = 0;
      if ((int)lane < avail) {
        const float et = W.st[sp - 1 - (int)lane];
        en = W.snode[sp - 1 - (int)lane];
        ok = et <= thi;
      }
      const uint32_t okm = __ballot_sync(kFull, ok);
      const int r = np + __popc(okm & lt_mask);
      if (ok && r < 4) W.pop[r] = en;
      const uint32_t m4 = __ballot_sync(kFull, ok && r == 3);
      sp -= m4 ? __ffs(m4) : avail;
      np = np + __popc(okm) < 4 ? np + __popc(okm) : 4;
    }
    __syncwarp();
    if (np > 0) {
      const int slot = (int)(lane >> 3);
      const bool valid = slot < np;
      const uint32_t node = W.pop[slot];
      float tnear = CUDART_INF_F;
      uint32_t ref = kInvalid;
      bool hit = false;
      if (valid) {
        const float4* rec = S.nodes8 + 16 * (size_t)node + 2 * (lane & 7);
        float4 a = __ldg(rec), b = __ldg(rec + 1);
        ref = __float_as_uint(b.z);
        float x0 = __fmaf_rn(a.x, br.ix, -br.ox), x1 = __fmaf_rn(a.w, br.ix, -br.ox);
        float y0 = __fmaf_rn(a.y, br.iy, -br.oy), y1 = __fmaf_rn(b.x, br.iy, -br.oy);
        float z0 = __fmaf_rn(a.z, br.iz, -br.oz), z1 = __fmaf_rn(b.y, br.iz, -br.oz);
        float tn = fmaxf(fmaxf(fminf(x0, x1) - br.px, fminf(y0, y1) - br.py), fmaxf(fminf(z0, z1) - br.pz, tlo));
        float tf = fminf(fminf(fmaxf(x0, x1) + br.px, fmaxf(y0, y1) + br.py), fminf(fmaxf(z0, z1) + br.pz, thi));
        hit = ref != kInvalid && tn <= tf;
        tnear = tn;
      }
      if (lane == 0) st.node_visits += (unsigned)np;
      const bool leaf = (ref & kLeafBit) != 0;
      const uint32_t lmask = __ballot_sync(kFull, hit && leaf);
      const uint32_t imask = __ballot_sync(kFull, hit && !leaf);
      if (lmask) {
        if (hit && leaf) {
          int q = nq + __popc(lmask & lt_mask);
          W.leafq[q] = ref & ~kLeafBit;
          W.leaft[q] = tnear;
        }
        nq += __popc(lmask);
      }
      if (imask) {
        const int m = __popc(imask);
        if (sp + m > (int)F.lim_stack) {
          status |= kStatusStackOverflow;
          return;
        }
        // the m hit children are written to stack slots sp..sp+m-1 in lane
        // order, then read back into lanes 0..m-1, sorted and stored far-to-near
        if (hit && !leaf) {
          const int r = __popc(imask & lt_mask);
          W.snode[sp + r] = ref;
          W.st[sp + r] = tnear;
        }
        __syncwarp();
        if (m > 1) {
          float key = CUDART_INF_F;
          uint32_t val = 0;
          if ((int)lane < m) {
            key = W.st[sp + (int)lane];
            val = W.snode[sp + (int)lane];
          }
          warp_sort_prefix(key, val, lane, m);
          __syncwarp();
          if ((int)lane < m) {
            W.snode[sp + m - 1 - (int)lane] = val;
            W.st[sp + m - 1 - (int)lane] = key;
          }
        }
        sp += m;
      }
      __syncwarp();
    }
    const bool drain = sp == 0;
    // kCollect tests leaves in two phases: the bounding-sphere filter on each
    // batch of 32 queued leaves, then the face tests on batches of kSurvivors
    // proxies that passed it.  The face tests then run with (nearly) every
    // lane busy instead of the ~60 % the filter leaves: 4 % faster on the 1M
    // view although the far bound tightens a little later (3 % more tests).
    if (MODE == kCollect) {
      if (nq >= leaf_batch || (drain && nq > 0)) {
        const int nb = nq < 32 ? nq : 32;
        uint32_t j = 0;
        float lt = 0.f;
        bool have = (int)lane < nb;
        if (have) {
          j = W.leafq[lane];
          lt = W.leaft[lane];
          have = lt <= thi;
        }
        __syncwarp();
        if (nq > nb) {
          uint32_t qj = 0;
          float qt = 0.f;
          bool mv = (int)lane < nq - nb;
          if (mv) {
            qj = W.leafq[nb + lane];
            qt = W.leaft[nb + lane];
          }
          __syncwarp();
          if (mv) {
            W.leafq[lane] = qj;
            W.leaft[lane] = qt;
          }
          __syncwarp();
        }
        nq -= nb;
        const uint32_t tested = __ballot_sync(kFull, have);
        if (lane == 0) st.proxy_tests += (unsigned)__popc(tested);
        const bool surv = have && proxy_sphere(F, S.w2o, j, o, d);
        const uint32_t sm = __ballot_sync(kFull, surv);
        if (surv) {
          const int r = ns + __popc(sm & lt_mask);
          W.svj[r] = j;
          W.svt[r] = lt;
        }
        ns += __popc(sm);
        __syncwarp();
      }
      const bool all_queued = sp == 0 && nq == 0;
      if (ns >= kSurvivors || (all_queued && ns > 0)) {
        const int nb = ns < 32 ? ns : 32;
        uint32_t j = 0;
        bool have = (int)lane < nb;
        if (have) {
          j = W.svj[lane];
          have = W.svt[lane] <= thi;
        }
        __syncwarp();
        if (ns > nb) {
          uint32_t qj = 0;
          float qt = 0.f;
          bool mv = (int)lane < ns - nb;
          if (mv) {
            qj = W.svj[nb + lane];
            qt = W.svt[nb + lane];
          }
          __syncwarp();
          if (mv) {
            W.svj[lane] = qj;
            W.svt[lane] = qt;
          }
          __syncwarp();
        }
        ns -= nb;
        int nh = 0;
        if (have) {
          const float tb = fminf(next_up(thi), t_max);
          auto on_hit = [&](float t, int) {
            if (nh < kMaxHitsPerProxy) W.hq[nh][lane] = t;
            ++nh;
          };
          proxy_faces(F, W.faces, S.w2o, j, o, d, tlo, tb, on_hit);
          if (nh > kMaxHitsPerProxy) {
            status |= kStatusHitOverflow;
            nh = kMaxHitsPerProxy;
          }
        }
        const uint32_t found = __reduce_add_sync(kFull, (uint32_t)nh);
        if (lane == 0) st.anyhits += found;
        if (found) {
          __syncwarp();
          const uint32_t p = nh ? __ldg(S.leaf_pidx + j) : 0u;
          while (true) {
            const uint32_t pend = __ballot_sync(kFull, nh > 0);
            if (!pend) break;
            const int src = __ffs(pend) - 1;
            const int slot = __shfl_sync(kFull, nh, src) - 1;
            const float t = W.hq[slot][src];
            const uint32_t pp = __shfl_sync(kFull, p, src);
            if ((int)lane == src) --nh;
            kbuf_insert(kb, t, pp, lane);
          }
          thi = kbuf_t_at(kb, cull);
        }
      }
      if (sp == 0 && nq == 0 && ns == 0) break;
      continue;
    }
    if (nq >= leaf_batch || (drain && nq > 0)) {
      const int nb = nq < 32 ? nq : 32;
      uint32_t j = 0;
      bool have = (int)lane < nb;
      if (have) {
        j = W.leafq[lane];
        have = W.leaft[lane] <= thi;
      }
      __syncwarp();
      if (nq > nb) {  // keep the rest (at most 31 entries) at the front of the queue
        uint32_t qj = 0;
        float qt = 0.f;
        bool mv = (int)lane < nq - nb;
        if (mv) {
          qj = W.leafq[nb + lane];
          qt = W.leaft[nb + lane];
        }
        __syncwarp();
        if (mv) {
          W.leafq[lane] = qj;
          W.leaft[lane] = qt;
        }
        __syncwarp();
      }
      nq -= nb;
      // one proxy per lane; its hits go to the lane's column of the hit queue
      // in shared memory (registers are the kernel's scarcest resource)
      int nh = 0;
      const uint32_t tested = __ballot_sync(kFull, have);
      if (lane == 0) st.proxy_tests += (unsigned)__popc(tested);
      if (have) {
        const float tb = MODE == kCountFront ? t_max : fminf(next_up(thi), t_max);
        auto on_hit = [&](float t, int) {
          if (nh < kMaxHitsPerProxy) W.hq[nh][lane] = t;
          ++nh;
        };
        if (proxy_sphere(F, S.w2o, j, o, d)) {
          if (MODE == kClosestAny)
            proxy_any_face(F, S.w2o, j, o, d, tlo, tb, on_hit);
          else
            proxy_faces(F, W.faces, S.w2o, j, o, d, tlo, tb, on_hit);
        }
        if (nh > kMaxHitsPerProxy) {
          status |= kStatusHitOverflow;
          nh = kMaxHitsPerProxy;
        }
      }
      const uint32_t found = __reduce_add_sync(kFull, (uint32_t)nh);
      if (lane == 0) st.anyhits += found;
      if (MODE != kCountFront && found) {
        __syncwarp();
        const uint32_t p = nh ? __ldg(S.leaf_pidx + j) : 0u;
        while (true) {
          const uint32_t pend = __ballot_sync(kFull, nh > 0);
          if (!pend) break;
          const int src = __ffs(pend) - 1;
          const int slot = __shfl_sync(kFull, nh, src) - 1;
          const float t = W.hq[slot][src];
          const uint32_t pp = __shfl_sync(kFull, p, src);
          if ((int)lane == src) --nh;
          kbuf_insert(kb, t, pp, lane);
        }
        thi = kbuf_t_at(kb, cull);
      }
    }
    if (sp == 0 && nq == 0) break;
  }
}

}  // namespace gt
