// gt_ploc.cu — binary hierarchy by hierarchical parallel locally-ordered
// clustering.
//
// PLOC (Meister and Bittner, "Parallel Locally-Ordered Clustering for
// Bounding Volume Hierarchy Construction", IEEE TVCG 2018) merges clusters
// with their nearest neighbour in Morton order (the distance is the surface
// area of the merged box).  Run over the whole array, every iteration is
// several launches and a host round trip (117 iterations for 1M proxies).
// H-PLOC (Benthin et al., "H-PLOC: Hierarchical Parallel Locally-Ordered
// Clustering for Bounding Volume Hierarchy Construction", 2024) does the same
// merges bottom-up over the radix tree of the Morton codes: a node's clusters
// are those its two children left over, at most kPlocKeep each, and the warp
// that reaches it merges mutual nearest neighbours until at most kPlocKeep
// remain (one at the root).  One launch, no host round trip.
//
// The warp's 32 lanes each climb from one leaf (Apetrei, "Fast and Simple
// Agglomerative LBVH Construction", 2014: the second child to arrive at a
// node goes on); when a lane's node holds more than kPlocKeep leaves, the
// whole warp merges its clusters, one per lane, by shuffles.
//
// Determinism: which clusters merge depends only on the codes, a tie in area
// goes to the smaller index.  A cluster is labelled by a leaf (the left
// cluster's label stays), so the label a merge retires numbers its node: the
// tree and its layout are the same on every run, and no counter is shared (with
// one atomic counter: 726 us).
//
// Bound by the instructions of the climb and of the neighbour search (48 % of
// issue slots, 29 % of warps resident: most lanes stop after a few nodes).
// B200, 1M proxies: the clustering loop took about 8 ms (3.5 ms of kernels and
// 117 host round trips), this kernel takes 660 us; rays visit as many nodes.
#include <math_constants.h>

#include <algorithm>

#include "gt_internal.cuh"

namespace gt {

constexpr uint32_t kPlocKeep = 16;   // clusters a node leaves to its parent
constexpr uint32_t kPlocRadius = 8;  // neighbours searched on either side
constexpr int kPlocBlock = 64;

struct PlocWarp {
  float b[6][32];
  uint32_t ref[32], label[32];
};

__device__ __forceinline__ unsigned long long ploc_delta(const uint32_t* __restrict__ keys, uint32_t i) {
  // codes made distinct by their position
  return ((unsigned long long)(keys[i] ^ keys[i + 1]) << 32) | (i ^ (i + 1));
}

__global__ void __launch_bounds__(kPlocBlock) k_hploc(const uint32_t* __restrict__ keys, uint32_t m,
                                                      const float* __restrict__ leaf_box, uint2* cluster,
                                                      uint32_t* link, float4* nodes, float* ibox,
                                                      uint32_t* parent_int, uint32_t* parent_leaf, uint32_t* root) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  __shared__ PlocWarp scratch[kPlocBlock / 32];
  PlocWarp& S = scratch[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  bool active = j < m;
  uint32_t lo = j, hi = j, split = 0;
  // (every pass moves each active lane one node up: at most m of them)
  while (__any_sync(kAll, active)) {
    if (active) {
      uint32_t other;
      if (lo == 0 || (hi != m - 1 && ploc_delta(keys, hi) < ploc_delta(keys, lo - 1))) {
        other = atomicExch(&link[hi], lo);  // this node is the left child
        if (other != kInvalid) {
          split = hi + 1;
          hi = other;
        }
      } else {
        other = atomicExch(&link[lo - 1], hi);
        if (other != kInvalid) {
          split = lo;
          lo = other;
        }
      }
      if (other == kInvalid) active = false;  // its sibling goes on
    }
    uint32_t todo = __ballot_sync(kAll, active && (hi - lo + 1 > kPlocKeep || hi - lo + 1 == m));
    if (todo) __threadfence();  // the arrivals before the reads of what they announced
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t L = __shfl_sync(kAll, lo, src), H = __shfl_sync(kAll, hi, src), P = __shfl_sync(kAll, split, src);
      const uint32_t keep = H - L + 1 == m ? 1u : kPlocKeep;
      // the children's clusters, left then right, one per lane
      uint32_t ref = kInvalid, label = 0;
      const uint32_t nl_max = min(P - L, kPlocKeep), nr_max = min(H - P + 1, kPlocKeep);
      if (lane < nl_max) {
        const uint2 c = __ldcg(cluster + L + lane);
        ref = c.x;
        label = c.y;
      }
      const uint32_t nl = __popc(__ballot_sync(kAll, ref != kInvalid));
      if (lane >= nl) {
        const uint2 c = lane - nl < nr_max ? __ldcg(cluster + P + (lane - nl)) : make_uint2(kInvalid, 0u);
        ref = c.x;
        label = c.y;
      }
      uint32_t n = __popc(__ballot_sync(kAll, ref != kInvalid));
      float b[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (lane < n) {
        const float* s = (ref & kLeafBit) ? leaf_box + 6 * (size_t)(ref & ~kLeafBit) : ibox + 6 * (size_t)ref;
#pragma unroll
        for (int a = 0; a < 6; ++a) b[a] = __ldcg(s + a);
      }
      while (n > keep) {
        // nearest neighbour within the radius (a tie keeps the smaller index)
        float best = CUDART_INF_F;
        uint32_t nn = lane > 0 ? lane - 1 : 1u;
#pragma unroll
        for (uint32_t r = kPlocRadius; r >= 1; --r) {
          float o[6];
#pragma unroll
          for (int a = 0; a < 6; ++a) o[a] = __shfl_down_sync(kAll, b[a], r);
          const float x = fmaxf(b[3], o[3]) - fminf(b[0], o[0]), y = fmaxf(b[4], o[4]) - fminf(b[1], o[1]),
                      z = fmaxf(b[5], o[5]) - fminf(b[2], o[2]);
          const float d = x * y + y * z + z * x;
          const float e = __shfl_up_sync(kAll, d, r);  // the pair (lane - r, lane)
          if (lane + r < n && (d < best || (d == best && lane + r < nn))) {
            best = d;
            nn = lane + r;
          }
          if (lane >= r && lane < n && (e < best || (e == best && lane - r < nn))) {
            best = e;
            nn = lane - r;
          }
        }
        const uint32_t back = __shfl_sync(kAll, nn, nn & 31u);
        bool mutual = lane < n && nn < n && back == lane;
        if (__ballot_sync(kAll, mutual) == 0) {  // (no order among the areas, as with NaN: the first two)
          mutual = lane < 2;
          nn = lane ^ 1u;
        }
        const bool merge = mutual && lane < nn, gone = mutual && nn < lane;
        // the partner's box and reference
        float o[6];
#pragma unroll
        for (int a = 0; a < 6; ++a) o[a] = __shfl_sync(kAll, b[a], nn & 31u);
        const uint32_t rb = __shfl_sync(kAll, ref, nn & 31u);
        const uint32_t retired = __shfl_sync(kAll, label, nn & 31u);
        if (merge) {
          const uint32_t id = retired - 1u;  // (label 0 is never retired)
          // binary node: child boxes as (lo.x, hi.x, lo.y, hi.y) x 2, (lo.z, hi.z) x 2, refs
          nodes[4 * (size_t)id + 0] = make_float4(b[0], b[3], b[1], b[4]);
          nodes[4 * (size_t)id + 1] = make_float4(o[0], o[3], o[1], o[4]);
          nodes[4 * (size_t)id + 2] = make_float4(b[2], b[5], o[2], o[5]);
          nodes[4 * (size_t)id + 3] = make_float4(__uint_as_float(ref), __uint_as_float(rb), 0.f, 0.f);
          if (ref & kLeafBit) parent_leaf[ref & ~kLeafBit] = id; else parent_int[ref] = id;
          if (rb & kLeafBit) parent_leaf[rb & ~kLeafBit] = id; else parent_int[rb] = id;
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            b[a] = fminf(b[a], o[a]);
            b[3 + a] = fmaxf(b[3 + a], o[3 + a]);
          }
#pragma unroll
          for (int a = 0; a < 6; ++a) ibox[6 * (size_t)id + a] = b[a];
          ref = id;
        }
        // close the gaps, in order
        const uint32_t km = __ballot_sync(kAll, lane < n && !gone);
        if (lane < n && !gone) {
          const uint32_t q = __popc(km & lt_mask);
#pragma unroll
          for (int a = 0; a < 6; ++a) S.b[a][q] = b[a];
          S.ref[q] = ref;
          S.label[q] = label;
        }
        n = __popc(km);
        __syncwarp();
        if (lane < n) {
#pragma unroll
          for (int a = 0; a < 6; ++a) b[a] = S.b[a][lane];
          ref = S.ref[lane];
          label = S.label[lane];
        }
        __syncwarp();
      }
      if (keep == 1u) {
        if (lane == 0) {
          *root = ref;
          parent_int[ref] = kInvalid;
        }
      } else if (lane < kPlocKeep && L + lane <= H) {
        cluster[L + lane] = make_uint2(lane < n ? ref : kInvalid, label);
      }
      __threadfence();  // the clusters before the next arrival
      __syncwarp();
    }
  }
}

__global__ void k_hploc_init(uint32_t m, uint2* cluster, uint32_t* link) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  cluster[j] = make_uint2(kLeafBit | j, j);
  link[j] = kInvalid;
}

Err build_ploc(const uint32_t* keys, const float* leaf_box, uint32_t m, cudaStream_t st, float4* nodes, float* ibox,
               uint32_t* parent_int, uint32_t* parent_leaf, uint32_t* root, uint64_t* launches) {
  if (m < 2) return Err{};
  uint2* cluster = nullptr;  // m clusters, then m links
  GT_CUDA_TRY(cudaMallocAsync(&cluster, (size_t)m * 12, st));
  uint32_t* link = reinterpret_cast<uint32_t*>(cluster + m);
  k_hploc_init<<<(m + 255) / 256, 256, 0, st>>>(m, cluster, link);
  k_hploc<<<(m + kPlocBlock - 1) / kPlocBlock, kPlocBlock, 0, st>>>(keys, m, leaf_box, cluster, link, nodes, ibox,
                                                                   parent_int, parent_leaf, root);
  *launches += 2;
  cudaError_t e = cudaGetLastError();
  cudaFreeAsync(cluster, st);
  GT_CUDA_TRY(e);
  return Err{};
}

}  // namespace gt
