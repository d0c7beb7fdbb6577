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
// The nodes of more than kPlocKeep leaves whose children have no more, at most
// m / (kPlocKeep + 1), each start a warp, which merges the node's clusters, one
// per lane, and climbs (Apetrei, "Fast and Simple Agglomerative LBVH
// Construction", 2014: the second child to arrive at a node goes on).
//
// Determinism: which clusters merge depends only on the codes and boxes, a tie in
// area goes to the smaller index.  A cluster is labelled by a leaf (the left
// cluster's label stays), so the label a merge retires numbers its node: the
// tree and its layout are the same on every run, and no counter is shared (with
// one atomic counter: 726 us).
//
// Bound by instructions while all tasks run and by the longest climb after that
// (25 nodes, 144 rounds of merges, about 1 us each).  B200, 1M proxies: a
// clustering loop over the array took about 8 ms (3.5 ms of kernels and 117 host
// round trips).  One warp for 32 leaves that climbed lane by lane, boxes passed by
// shuffles: 650 us (a warp's lanes wait for one another, SMs idle 40 %); a warp
// for each task: 529 us; boxes read from shared memory, the nearest neighbour as
// the least of 16 integer keys, clusters stored with their boxes: 366 us, and
// 16 us to find the tasks.
#include <math_constants.h>

#include <algorithm>

#include "gt_internal.cuh"

namespace gt {

constexpr uint32_t kPlocKeep = 16;   // clusters a node leaves to its parent
constexpr uint32_t kPlocRadius = 8;  // neighbours searched on either side
constexpr int kPlocBlock = 32;  // (a warp's work varies: 64 threads 583 us, 32 threads 529)

// The warp's clusters in shared memory: (lo, hi.x), (hi.yz), (reference, label).
// Rows from the number of clusters on hold a box too large to merge with.
struct PlocWarp {
  float4 b0[32 + kPlocRadius];
  float2 b1[32 + kPlocRadius];
  uint2 id[32];
};
constexpr float kPlocFar = 1e30f;  // squared: infinity

__device__ __forceinline__ unsigned long long ploc_delta(const uint32_t* __restrict__ keys, uint32_t i) {
  // codes made distinct by their position
  return ((unsigned long long)(keys[i] ^ keys[i + 1]) << 32) | (i ^ (i + 1));
}

// One thread a boundary i | i + 1: the radix tree's node that splits there spans
// the leaves around it whose deltas are smaller, found by at most kPlocKeep + 1
// steps to either side.  A node of more than kPlocKeep leaves (or the root) whose
// children have no more each is a task, (lo, hi, split); a child that small whose
// sibling is larger counts as arrived.
constexpr int kFindBlock = 256;
__global__ void __launch_bounds__(kFindBlock) k_hploc_find(const uint32_t* __restrict__ keys, uint32_t m,
                                                           uint32_t* link, uint4* tasks, uint32_t* count) {
  constexpr int kHalo = (int)kPlocKeep + 1;
  __shared__ unsigned long long delta[kFindBlock + 2 * kHalo];  // ~0 past the ends
  const int64_t first = (int64_t)blockIdx.x * kFindBlock - kHalo;
  for (int x = threadIdx.x; x < kFindBlock + 2 * kHalo; x += kFindBlock) {
    const int64_t b = first + x;
    delta[x] = b >= 0 && b + 1 < (int64_t)m ? ploc_delta(keys, (uint32_t)b) : ~0ull;
  }
  __syncthreads();
  const uint32_t i = blockIdx.x * kFindBlock + threadIdx.x;
  bool found = false;
  uint32_t nl = 1, nr = 1;  // leaves on either side, kPlocKeep + 1 for more than kPlocKeep
  if (i + 1 < m) {
    const unsigned long long* at = delta + kHalo + threadIdx.x;
    const unsigned long long mine = *at;
    while (nl <= kPlocKeep && at[-(int)nl] < mine) ++nl;
    while (nr <= kPlocKeep && at[nr] < mine) ++nr;
    const bool sl = nl <= kPlocKeep, sr = nr <= kPlocKeep;
    found = sl && sr && (nl + nr > kPlocKeep || nl + nr == m);
    link[i] = sl == sr ? kInvalid : sl ? i + 1 - nl : i + nr;
  }
  // places in the block, then one atomic a block (one a warp: 31 us for 1M leaves)
  __shared__ uint32_t in_block, base;
  if (threadIdx.x == 0) in_block = 0;
  __syncthreads();
  uint32_t place = 0;
  if (found) place = atomicAdd(&in_block, 1u);
  __syncthreads();
  if (threadIdx.x == 0 && in_block) base = atomicAdd(count, in_block);
  __syncthreads();
  if (found) tasks[base + place] = make_uint4(i + 1 - nl, i + nr, i + 1, 0u);
}

__global__ void __launch_bounds__(kPlocBlock) k_hploc(const uint32_t* __restrict__ keys, uint32_t m,
                                                      const float* __restrict__ leaf_box, float4* cluster,
                                                      uint32_t* link, const uint4* __restrict__ tasks,
                                                      const uint32_t* __restrict__ count, float4* nodes, float* ibox,
                                                      uint32_t* parent_int, uint32_t* parent_leaf, uint32_t* root) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  __shared__ PlocWarp scratch[kPlocBlock / 32];
  PlocWarp& S = scratch[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t task = blockIdx.x * (kPlocBlock / 32) + (threadIdx.x >> 5);
  if (task >= *count) return;
  uint32_t L = tasks[task].x, H = tasks[task].y, P = tasks[task].z;
  if (lane < kPlocRadius) {
    S.b0[32 + lane] = make_float4(-kPlocFar, -kPlocFar, -kPlocFar, kPlocFar);
    S.b1[32 + lane] = make_float2(kPlocFar, kPlocFar);
  }
  uint32_t back_code[kPlocRadius];  // of the neighbour r before; larger than any area where there is none
#pragma unroll
  for (uint32_t r = 1; r <= kPlocRadius; ++r) back_code[r - 1] = (kPlocRadius - r) | (lane < r ? 0x7FFFFFF0u : 0u);
  // (every pass moves the warp one node up: at most m of them)
  while (true) {
    // which child of its parent the node is
    const bool left = L == 0 || (H != m - 1 && ploc_delta(keys, H) < ploc_delta(keys, L - 1));
    const uint32_t keep = H - L + 1 == m ? 1u : kPlocKeep;
    // the children's clusters: the left child's by lanes 0..15, the right one's by
    // 16..31.  A child of at most kPlocKeep leaves has these for clusters.
    uint32_t ref = kInvalid, label = 0, n;
    float4 b0;
    float2 b1;
    {
      const uint32_t from = lane < kPlocKeep ? L : P, to = lane < kPlocKeep ? P : H + 1;
      const uint32_t at = from + (lane & (kPlocKeep - 1u));
      if (to - from > kPlocKeep) {
        const float4 v0 = __ldcg(cluster + 2 * (size_t)at), v1 = __ldcg(cluster + 2 * (size_t)at + 1);
        ref = __float_as_uint(v0.x);
        label = __float_as_uint(v0.y);
        b0 = make_float4(v0.z, v0.w, v1.x, v1.y);
        b1 = make_float2(v1.z, v1.w);
      } else if (at < to) {
        const float2* s = reinterpret_cast<const float2*>(leaf_box + 6 * (size_t)at);
        const float2 v0 = __ldg(s), v1 = __ldg(s + 1);
        ref = kLeafBit | at;
        label = at;
        b0 = make_float4(v0.x, v0.y, v1.x, v1.y);
        b1 = __ldg(s + 2);
      }
      const uint32_t have = __ballot_sync(kAll, ref != kInvalid);
      n = __popc(have);
      __syncwarp();
      if (ref != kInvalid) {
        const uint32_t q = __popc(have & lt_mask);
        S.b0[q] = b0;
        S.b1[q] = b1;
        S.id[q] = make_uint2(ref, label);
      }
      if (lane >= n) {
        S.b0[lane] = make_float4(-kPlocFar, -kPlocFar, -kPlocFar, kPlocFar);
        S.b1[lane] = make_float2(kPlocFar, kPlocFar);
      }
      __syncwarp();
      b0 = S.b0[lane];
      b1 = S.b1[lane];
      ref = S.id[lane].x;
      label = S.id[lane].y;
    }
    while (n > keep) {
      // Nearest neighbour within the radius: the least of 16 keys, a merged area
      // (not negative, so its bits are in order) with the low four bits replaced by
      // the neighbour's place, earlier first.
      uint32_t near = 0x7FFFFFFFu, d[kPlocRadius];
#pragma unroll
      for (uint32_t r = 1; r <= kPlocRadius; ++r) {
        const float4 o0 = S.b0[lane + r];
        const float2 o1 = S.b1[lane + r];
        const float x = fmaxf(b0.w, o0.w) - fminf(b0.x, o0.x), y = fmaxf(b1.x, o1.x) - fminf(b0.y, o0.y),
                    z = fmaxf(b1.y, o1.y) - fminf(b0.z, o0.z);
        d[r - 1] = __float_as_uint(__fmaf_rn(x, y, __fmaf_rn(y, z, z * x)));
        near = min(near, (d[r - 1] & ~15u) | (kPlocRadius - 1 + r));
      }
#pragma unroll
      for (uint32_t r = 1; r <= kPlocRadius; ++r)
        near = min(near, (__shfl_up_sync(kAll, d[r - 1], r) & ~15u) | back_code[r - 1]);
      uint32_t nn = lane + (near & 15u) - kPlocRadius;
      if ((near & 15u) >= kPlocRadius) ++nn;
      const uint32_t back = __shfl_sync(kAll, nn, nn & 31u);
      bool mutual = lane < n && nn < n && back == lane;
      if (__ballot_sync(kAll, mutual) == 0) {  // (no order among the areas, as with NaN: the first two)
        mutual = lane < 2;
        nn = lane ^ 1u;
      }
      const bool merge = mutual && lane < nn, gone = mutual && nn < lane;
      if (merge) {
        const float4 o0 = S.b0[nn];
        const float2 o1 = S.b1[nn];
        const uint2 other = S.id[nn];
        const uint32_t id = other.y - 1u;  // the label retired (label 0 never is)
        // binary node: child boxes as (lo.x, hi.x, lo.y, hi.y) x 2, (lo.z, hi.z) x 2, refs
        nodes[4 * (size_t)id + 0] = make_float4(b0.x, b0.w, b0.y, b1.x);
        nodes[4 * (size_t)id + 1] = make_float4(o0.x, o0.w, o0.y, o1.x);
        nodes[4 * (size_t)id + 2] = make_float4(b0.z, b1.y, o0.z, o1.y);
        nodes[4 * (size_t)id + 3] = make_float4(__uint_as_float(ref), __uint_as_float(other.x), 0.f, 0.f);
        if (ref & kLeafBit) parent_leaf[ref & ~kLeafBit] = id; else parent_int[ref] = id;
        if (other.x & kLeafBit) parent_leaf[other.x & ~kLeafBit] = id; else parent_int[other.x] = id;
        b0 = make_float4(fminf(b0.x, o0.x), fminf(b0.y, o0.y), fminf(b0.z, o0.z), fmaxf(b0.w, o0.w));
        b1 = make_float2(fmaxf(b1.x, o1.x), fmaxf(b1.y, o1.y));
        float2* s = reinterpret_cast<float2*>(ibox + 6 * (size_t)id);
        s[0] = make_float2(b0.x, b0.y);
        s[1] = make_float2(b0.z, b0.w);
        s[2] = b1;
        ref = id;
      }
      // close the gaps, in order
      const uint32_t km = __ballot_sync(kAll, lane < n && !gone);
      __syncwarp();
      if (lane < n && !gone) {
        const uint32_t q = __popc(km & lt_mask);
        S.b0[q] = b0;
        S.b1[q] = b1;
        S.id[q] = make_uint2(ref, label);
      }
      n = __popc(km);
      if (lane >= n) {
        S.b0[lane] = make_float4(-kPlocFar, -kPlocFar, -kPlocFar, kPlocFar);
        S.b1[lane] = make_float2(kPlocFar, kPlocFar);
      }
      __syncwarp();
      b0 = S.b0[lane];
      b1 = S.b1[lane];
      ref = S.id[lane].x;
      label = S.id[lane].y;
    }
    if (keep == 1u) {
      if (lane == 0) {
        *root = ref;
        parent_int[ref] = kInvalid;
      }
      return;
    }
    if (lane < kPlocKeep) {  // (the node has more leaves than that)
      float4* o = cluster + 2 * (size_t)(L + lane);
      o[0] = make_float4(__uint_as_float(lane < n ? ref : kInvalid), __uint_as_float(label), b0.x, b0.y);
      o[1] = make_float4(b0.z, b0.w, b1.x, b1.y);
    }
    __threadfence();  // the clusters and boxes before the arrival
    __syncwarp();
    // the first child to arrive at the parent leaves its far end there
    uint32_t other = 0;
    if (lane == 0) other = left ? atomicExch(link + H, L) : atomicExch(link + L - 1, H);
    other = __shfl_sync(kAll, other, 0);
    if (other == kInvalid) return;  // its sibling goes on
    P = left ? H + 1 : L;
    if (left) H = other; else L = other;
    __threadfence();  // the arrival before the reads of what it announced
  }
}

Err build_ploc(const uint32_t* keys, const float* leaf_box, uint32_t m, cudaStream_t st, float4* nodes, float* ibox,
               uint32_t* parent_int, uint32_t* parent_leaf, uint32_t* root, uint64_t* launches) {
  if (m < 2) return Err{};
  const uint32_t most = m / (kPlocKeep + 1) + 1;  // tasks: their nodes are disjoint (one when m <= kPlocKeep)
  uint4* tasks = nullptr;  // `most` tasks, m clusters (reference, label, box), m links, the count
  GT_CUDA_TRY(cudaMallocAsync(&tasks, (size_t)most * 16 + (size_t)m * 36 + 4, st));
  float4* cluster = reinterpret_cast<float4*>(tasks + most);
  uint32_t* link = reinterpret_cast<uint32_t*>(cluster + 2 * (size_t)m);
  uint32_t* count = link + m;
  GT_CUDA_TRY(cudaMemsetAsync(count, 0, 4, st));
  k_hploc_find<<<(m + kFindBlock - 1) / kFindBlock, kFindBlock, 0, st>>>(keys, m, link, tasks, count);
  const uint32_t warps = kPlocBlock / 32;
  k_hploc<<<(most + warps - 1) / warps, kPlocBlock, 0, st>>>(keys, m, leaf_box, cluster, link, tasks, count, nodes,
                                                             ibox, parent_int, parent_leaf, root);
  *launches += 2;
  cudaError_t e = cudaGetLastError();
  cudaFreeAsync(tasks, st);
  GT_CUDA_TRY(e);
  return Err{};
}

}  // namespace gt
