/*
 * bvh_gpu.cu - BVH8 builder on the GPU (replaces the OptiX "Trbvh" build the
 * reference requests for every group, e.g. host_includes/scenes.hpp:32).
 *
 *  1. k_bounds      padded world AABB and centroid of every primitive record
 *  2. k_morton      30-bit Morton code of the centroid (10 bits per axis, one
 *                   scale for all axes: the centroid box's longest side)
 *  3. radix sort    CUB DeviceRadixSort over (code, primitive) pairs
 *  4. k_ploc        (triangle meshes) binary tree by locally-ordered clustering
 *                   and the cost of every subtree as slots of wide nodes, in
 *                   one launch (H-PLOC, HPG 2024)
 *     k_karras      (other scenes) binary radix tree, Karras, "Maximizing
 *                   Parallelism in the Construction of BVHs, Octrees, and k-d
 *                   Trees", HPG 2012; then k_bottom_up: bounds and SAH cost
 *                   bottom-up (atomic arrival counters); at every node with
 *                   >= 7 primitives below it the treelet of up to 7 leaves is
 *                   rebuilt optimally for SAH by dynamic programming over leaf
 *                   subsets (Karras & Aila, "Fast Parallel Construction of
 *                   High-Quality BVHs", HPG 2013), one warp per treelet; a
 *                   first pass without restructuring, then one per treelet
 *                   round
 *  5. k_collapse    one launch per level: each binary node becomes a wide
 *                   node, cut by the costs of k_ploc, or by expanding its
 *                   largest child until 8 children (or the requested width);
 *                   subtrees of <= 3 primitives become leaf slots; child
 *                   boxes are quantised to 8 bits (node format: pt_types.h)
 *  6. k_check_*     structural check of the finished tree before any
 *                   traversal runs on it (check_node8 on every node, every
 *                   leaf position covered once, leaf_of_id a permutation)
 * The result is order independent for rendering (closest hit is the minimum
 * of (t, primitive id)), so the atomics that place nodes do not change images.
 */
#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>
#include <stdint.h>
#include <vector>

#include "bvh_build.h"
#include "pt_device.cuh"
#include "pt_internal.h"

#ifndef PT_TREELET_ROUNDS
#define PT_TREELET_ROUNDS 2  /* SAH treelet restructuring passes */
#endif

namespace {

constexpr uint32_t LEAF_BIT = 0x80000000u;
constexpr uint32_t NONE = 0xffffffffu;
constexpr float C_INNER = 1.2f, C_TRI = 1.0f;

struct GBox {
  float lo[3], hi[3];
};

__device__ __forceinline__ GBox box_union(const GBox& a, const GBox& b) {
  GBox r;
  for (int k = 0; k < 3; k++) {
    r.lo[k] = fminf(a.lo[k], b.lo[k]);
    r.hi[k] = fmaxf(a.hi[k], b.hi[k]);
  }
  return r;
}
__device__ __forceinline__ float box_area(const GBox& b) {
  float x = b.hi[0] - b.lo[0], y = b.hi[1] - b.lo[1], z = b.hi[2] - b.lo[2];
  return x * y + y * z + z * x;
}
__device__ __forceinline__ void box_store(float4* lo, float4* hi, uint32_t i, const GBox& b,
                                          float w0, float w1) {
  lo[i] = make_float4(b.lo[0], b.lo[1], b.lo[2], w0);
  hi[i] = make_float4(b.hi[0], b.hi[1], b.hi[2], w1);
}
__device__ __forceinline__ GBox box_load(const float4* lo, const float4* hi, uint32_t i) {
  float4 a = lo[i], b = hi[i];
  GBox r;
  r.lo[0] = a.x; r.lo[1] = a.y; r.lo[2] = a.z;
  r.hi[0] = b.x; r.hi[1] = b.y; r.hi[2] = b.z;
  return r;
}
// Loads of tree data that other threads write during the same kernel
// (k_ploc, k_bottom_up): L2 only (ld.global.cg), so no stale L1 line is read.
__device__ __forceinline__ GBox box_load_cg(const float4* lo, const float4* hi, uint32_t i) {
  float4 a = __ldcg(lo + i), b = __ldcg(hi + i);
  GBox r;
  r.lo[0] = a.x; r.lo[1] = a.y; r.lo[2] = a.z;
  r.hi[0] = b.x; r.hi[1] = b.y; r.hi[2] = b.z;
  return r;
}

// Padded world AABB of one primitive record (the host builder's padding).
__global__ void k_bounds(const float4* __restrict__ rec, const float4* __restrict__ xforms,
                         uint32_t n, float cam_t0, float cam_t1, float4* lo, float4* hi,
                         unsigned int* cbox) {
  GBox c;
  for (int k = 0; k < 3; k++) {
    c.lo[k] = 3.0e38f;
    c.hi[k] = -3.0e38f;
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float4 r0 = rec[3 * i], r1 = rec[3 * i + 1], r2 = rec[3 * i + 2];
    uint32_t tag = __float_as_uint(r0.w);
    int type = tag & 3, axis = (tag >> 2) & 3, xf = (int)(tag >> 8) - 1;
    float f[9] = {r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r2.x, r2.y, r2.z};
    GBox b;
    if (type == PT_PRIM_TRIANGLE) {
      for (int a = 0; a < 3; a++) {
        b.lo[a] = fminf(fminf(f[a], f[3 + a]), f[6 + a]);
        b.hi[a] = fmaxf(fmaxf(f[a], f[3 + a]), f[6 + a]);
      }
    } else if (type == PT_PRIM_SPHERE && (tag & PT_PRIM_MOVING)) {
      pt::moving_sphere_box(f, cam_t0, cam_t1, b.lo, b.hi);
    } else if (type == PT_PRIM_SPHERE) {
      for (int a = 0; a < 3; a++) {
        b.lo[a] = f[a] - f[3];
        b.hi[a] = f[a] + f[3];
      }
    } else if (type == PT_PRIM_RECT) {
      int ia = axis == 0 ? 1 : 0, ib = axis == 2 ? 1 : 2;
      b.lo[axis] = b.hi[axis] = f[4];
      b.lo[ia] = f[0];
      b.hi[ia] = f[1];
      b.lo[ib] = f[2];
      b.hi[ib] = f[3];
    } else {
      for (int a = 0; a < 3; a++) {
        b.lo[a] = f[a];
        b.hi[a] = f[3 + a];
      }
    }
    if (xf >= 0) {
      const float4* M = xforms + 6 * xf;
      GBox w;
      for (int k = 0; k < 3; k++) {
        w.lo[k] = 3.0e38f;
        w.hi[k] = -3.0e38f;
      }
      for (int cc = 0; cc < 8; cc++) {
        ptd::V3 q = ptd::v3((cc & 1) ? b.hi[0] : b.lo[0], (cc & 2) ? b.hi[1] : b.lo[1],
                            (cc & 4) ? b.hi[2] : b.lo[2]);
        ptd::V3 p = ptd::xpoint(M, q);
        float pw[3] = {p.x, p.y, p.z};
        for (int k = 0; k < 3; k++) {
          w.lo[k] = fminf(w.lo[k], pw[k]);
          w.hi[k] = fmaxf(w.hi[k], pw[k]);
        }
      }
      b = w;
    }
    for (int a = 0; a < 3; a++) {
      float mag = fmaxf(1.0f, fmaxf(fabsf(b.lo[a]), fabsf(b.hi[a])));
      float pad = mag * 9.5367431640625e-07f * (xf >= 0 ? 16.f : 1.f);
      b.lo[a] -= pad;
      b.hi[a] += pad;
    }
    lo[i] = make_float4(b.lo[0], b.lo[1], b.lo[2], 0.f);
    hi[i] = make_float4(b.hi[0], b.hi[1], b.hi[2], 0.f);
    for (int a = 0; a < 3; a++) {
      const float m = 0.5f * (b.lo[a] + b.hi[a]);
      c.lo[a] = fminf(c.lo[a], m);
      c.hi[a] = fmaxf(c.hi[a], m);
    }
  }
  // centroid bounds: warp reductions, then ordered-int atomics (the grid is a
  // few blocks per SM: an atomic per warp of all primitives took 0.28 ms for
  // 2.1 M)
  for (int a = 0; a < 3; a++) {
    for (int o = 16; o > 0; o >>= 1) {
      c.lo[a] = fminf(c.lo[a], __shfl_xor_sync(0xffffffffu, c.lo[a], o));
      c.hi[a] = fmaxf(c.hi[a], __shfl_xor_sync(0xffffffffu, c.hi[a], o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
    for (int a = 0; a < 3; a++) {
      // monotone float -> uint mapping
      uint32_t u = __float_as_uint(c.lo[a]);
      u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
      atomicMin(&cbox[a], u);
      uint32_t v = __float_as_uint(c.hi[a]);
      v = (v & 0x80000000u) ? ~v : (v | 0x80000000u);
      atomicMax(&cbox[3 + a], v);
    }
  }
}

__device__ __forceinline__ float unmap(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ uint32_t spread10(uint32_t v) {
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

__global__ void k_morton(const float4* __restrict__ lo, const float4* __restrict__ hi, uint32_t n,
                         const unsigned int* cbox, uint32_t* keys, uint32_t* vals) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 a = lo[i], b = hi[i];
  float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
  // one scale for all axes (the centroid box's longest side): a flat scene
  // (a heightfield) is not split along its thin axis as often as along the
  // wide ones, which would give siblings that overlap over their whole area
  float e = 0.f;
  for (int k = 0; k < 3; k++) e = fmaxf(e, unmap(cbox[3 + k]) - unmap(cbox[k]));
  uint32_t code = 0;
  for (int k = 0; k < 3; k++) {
    float l = unmap(cbox[k]);
    float t = e > 0.f ? (c[k] - l) / e : 0.5f;
    uint32_t q = (uint32_t)fminf(fmaxf(t * 1024.f, 0.f), 1023.f);
    code |= spread10(q) << (2 - k);
  }
  keys[i] = code;
  vals[i] = i;
}

// ---------------------------------------------------------- binary tree ----
// Internal nodes 0..n-2; references with LEAF_BIT are leaves in Morton order.
struct Tree {
  uint32_t *left, *right;
  uint32_t *parent_int, *parent_leaf, *flags;  // treelet builder
  float4 *ilo, *ihi;        // internal bounds; ilo.w = SAH cost (treelet builder),
                            // ihi.w = primitive count
  const float4 *llo, *lhi;  // leaf bounds (sorted order)
  float4* cost;             // 2 per node, of nodes that are clusters between merges: WideCost
  uint32_t* plan;           // per node: how it is cut into wide nodes (wide_cost); null: by area
  uint32_t root;
  bool guard;               // encode_node_dev
};

// Cost of a subtree as at most i + 1 slots of a wide node, by dynamic
// programming over the binary tree (Ylitie, Karras & Laine, HPG 2017, sec. 3):
// one slot holds a leaf of up to 3 primitives or a wide node of its own, more
// slots are shared between the two children.
#ifndef PT_COST_NODE
#define PT_COST_NODE 1.0f
#endif
#ifndef PT_COST_PRIM
#define PT_COST_PRIM 0.3f
#endif
struct WideCost {
  float c[7];
};

// The costs of a node from its children's and its plan: bits 3j..3j+2 (j =
// 0..6): the left child's slots when the node has j + 2 (0: it takes fewer);
// bit 21: as one slot it is a leaf.
__device__ __forceinline__ WideCost wide_cost(const WideCost& l, const WideCost& r, float area,
                                              float count, int width, uint32_t& plan) {
  WideCost o;
  float dist[7];
  plan = 0;
#pragma unroll
  for (int j = 2; j <= 8; j++) {
    float best = 3.0e38f;
    uint32_t k = 1;
#pragma unroll
    for (int i = 1; i < j; i++) {
      if (j - i > 7 || i > 7) continue;
      const float v = l.c[i - 1] + r.c[j - i - 1];
      if (v < best) {
        best = v;
        k = (uint32_t)i;
      }
    }
    dist[j - 2] = best;
    plan |= k << (3 * (j - 2));
  }
  float whole = dist[6];
#pragma unroll
  for (int j = 2; j < 8; j++)
    if (j == width) whole = dist[j - 2];
  o.c[0] = PT_COST_NODE * area + whole;
  if (count <= 3.f && PT_COST_PRIM * area * count <= o.c[0]) {
    o.c[0] = PT_COST_PRIM * area * count;
    plan |= 1u << 21;
  }
#pragma unroll
  for (int j = 2; j <= 7; j++) {
    o.c[j - 1] = dist[j - 2];
    if (j == width) continue;  // a full node is always shared out
    if (o.c[j - 2] <= o.c[j - 1]) {
      o.c[j - 1] = o.c[j - 2];
      plan &= ~(7u << (3 * (j - 2)));
    }
  }
  return o;
}

__device__ __forceinline__ GBox ref_box(const Tree& T, uint32_t r) {
  return (r & LEAF_BIT) ? box_load(T.llo, T.lhi, r & ~LEAF_BIT) : box_load(T.ilo, T.ihi, r);
}
__device__ __forceinline__ float ref_count(const Tree& T, uint32_t r) {
  return (r & LEAF_BIT) ? 1.f : T.ihi[r].w;
}

// Where the Morton codes of positions i and i + 1 differ (equal codes: where
// the positions do); smaller = closer.
__device__ __forceinline__ unsigned long long code_gap(const uint32_t* __restrict__ keys, uint32_t i) {
  const unsigned long long a = ((unsigned long long)keys[i] << 32) | i;
  const unsigned long long b = ((unsigned long long)keys[i + 1] << 32) | (i + 1);
  return a ^ b;
}

// Clusters kept per code range, and places searched on each side.  The radius
// is small: with 1 / 2 / 3 / 4 / 8 / 16 a 2.1 M-triangle terrain took 7.28 /
// 7.30 / 7.26 / 7.43 / 7.48 / - node fetches per ray, one of 0.5 M 6.60 /
// 6.59 / 6.79 / 6.86 / 7.16 / - (greedy collapse, 8 / 16: 7.66 / 8.03 and
// 7.45 / 7.54): on regular meshes the Morton order already is the good tree.
constexpr uint32_t PLOC_KEEP = 16, PLOC_RADIUS = 2;

// A lane's cluster while a warp merges.
struct Cluster {
  uint32_t ref;
  GBox box;
  float count;
  WideCost w;
};

__device__ __forceinline__ Cluster shfl_cluster(const Cluster& c, int src) {
  Cluster r;
  r.ref = __shfl_sync(0xffffffffu, c.ref, src);
  for (int a = 0; a < 3; a++) {
    r.box.lo[a] = __shfl_sync(0xffffffffu, c.box.lo[a], src);
    r.box.hi[a] = __shfl_sync(0xffffffffu, c.box.hi[a], src);
  }
  r.count = __shfl_sync(0xffffffffu, c.count, src);
  for (int k = 0; k < 7; k++) r.w.c[k] = __shfl_sync(0xffffffffu, c.w.c[k], src);
  return r;
}

// Merges the clusters of the code ranges [L, split) and [split, R] (at most
// PLOC_KEEP each, at the front of their range's entries of `cluster`) until at
// most PLOC_KEEP are left (one at the root): each cluster finds the neighbour
// within PLOC_RADIUS places whose union with it has the least area, and
// mutual nearest neighbours become one node.  All lanes call it together.
__device__ void ploc_merge(const Tree& T, uint32_t* cluster, uint32_t* counter, uint32_t L,
                           uint32_t split, uint32_t R, bool top, int width, uint8_t* map, int lane) {
  const uint32_t nl = min(PLOC_KEEP, split - L), nr = min(PLOC_KEEP, R + 1 - split);
  Cluster c;
  c.ref = NONE;
  if ((uint32_t)lane < nl) c.ref = __ldcg(cluster + L + lane);
  if ((uint32_t)lane >= PLOC_KEEP && (uint32_t)lane - PLOC_KEEP < nr)
    c.ref = __ldcg(cluster + split + (lane - PLOC_KEEP));
  const uint32_t valid = __ballot_sync(0xffffffffu, c.ref != NONE);
  const int cl = __popc(valid & ((1u << PLOC_KEEP) - 1u));
  int num = __popc(valid);
  c.ref = __shfl_sync(0xffffffffu, c.ref, lane < cl ? lane : (lane - cl + (int)PLOC_KEEP) & 31);
  if (lane >= num) c.ref = NONE;
  c.count = 1.f;
  for (int a = 0; a < 3; a++) c.box.lo[a] = c.box.hi[a] = 0.f;
  for (int k = 0; k < 7; k++) c.w.c[k] = 0.f;
  if (c.ref != NONE) {
    if (c.ref & LEAF_BIT) {
      c.box = box_load(T.llo, T.lhi, c.ref & ~LEAF_BIT);
      for (int k = 0; k < 7; k++) c.w.c[k] = PT_COST_PRIM * box_area(c.box);
    } else {
      c.box = box_load_cg(T.ilo, T.ihi, c.ref);
      const float4 w0 = __ldcg(T.cost + 2 * (size_t)c.ref), w1 = __ldcg(T.cost + 2 * (size_t)c.ref + 1);
      c.w.c[0] = w0.x; c.w.c[1] = w0.y; c.w.c[2] = w0.z; c.w.c[3] = w0.w;
      c.w.c[4] = w1.x; c.w.c[5] = w1.y; c.w.c[6] = w1.z;
      c.count = w1.w;
    }
  }
  const int goal = top ? 1 : (int)PLOC_KEEP;
  for (int it = 0; it < 32 && num > goal; it++) {  // each step merges a pair at least
    // nearest neighbour: the area's bits (it is not negative) with the lane in
    // the low 5; the pair of least (area, lanes) is always mutual
    uint32_t best = NONE;
#pragma unroll
    for (int r = 1; r <= (int)PLOC_RADIUS; r++) {
      GBox o;
      for (int a = 0; a < 3; a++) {
        o.lo[a] = __shfl_down_sync(0xffffffffu, c.box.lo[a], r);
        o.hi[a] = __shfl_down_sync(0xffffffffu, c.box.hi[a], r);
      }
      uint32_t d = NONE;
      if (lane + r < num) {
        d = __float_as_uint(fmaxf(box_area(box_union(c.box, o)), 0.f)) & ~31u;
        best = min(best, d | (uint32_t)(lane + r));
      }
      const uint32_t up = __shfl_up_sync(0xffffffffu, d, r);
      if (lane >= r && lane < num) best = min(best, up | (uint32_t)(lane - r));
    }
    const int nn = lane < num ? (int)(best & 31u) : lane;
    const int back = __shfl_sync(0xffffffffu, nn, nn);  // every lane takes part
    const bool mutual = lane < num && back == lane;
    const bool merges = mutual && lane < nn;
    const uint32_t mm = __ballot_sync(0xffffffffu, merges);
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(counter, (uint32_t)__popc(mm));
    base = __shfl_sync(0xffffffffu, base, 0);
    const Cluster o = shfl_cluster(c, nn);
    if (merges) {
      const uint32_t node = base + (uint32_t)__popc(mm & ((1u << lane) - 1u));
      T.left[node] = c.ref;
      T.right[node] = o.ref;
      c.box = box_union(c.box, o.box);
      c.count += o.count;
      box_store(T.ilo, T.ihi, node, c.box, 0.f, c.count);
      uint32_t plan;
      c.w = wide_cost(c.w, o.w, box_area(c.box), c.count, width, plan);
      T.plan[node] = plan;
      c.ref = node;
    }
    const bool keep = lane < num && !(mutual && lane > nn);
    const uint32_t km = __ballot_sync(0xffffffffu, keep);
    if (keep) map[__popc(km & ((1u << lane) - 1u))] = (uint8_t)lane;
    __syncwarp();
    num = __popc(km);
    c = shfl_cluster(c, lane < num ? map[lane] : lane);
    __syncwarp();
    if (lane >= num) c.ref = NONE;
  }
  if ((uint32_t)lane < PLOC_KEEP && L + lane <= R) {
    cluster[L + lane] = c.ref;
    if (!(c.ref & LEAF_BIT)) {  // NONE has the bit too
      T.cost[2 * (size_t)c.ref] = make_float4(c.w.c[0], c.w.c[1], c.w.c[2], c.w.c[3]);
      T.cost[2 * (size_t)c.ref + 1] = make_float4(c.w.c[4], c.w.c[5], c.w.c[6], c.count);
    }
  }
  __threadfence();  // nodes and entries before any lane of this warp reports the range upward
  __syncwarp();
}

// Bottom-up over the Morton order (H-PLOC: Benthin, Meister, Barczak, Mehalwal,
// Tsakok & Kensler, "H-PLOC: Hierarchical Parallel Locally-Ordered Clustering
// for Bounding Volume Hierarchy Construction", HPG 2024): a thread's code
// range joins its sibling's (the second to arrive goes on), and ranges of more
// than PLOC_KEEP primitives are merged to PLOC_KEEP clusters by the whole
// warp.  ends: per gap between codes, the outer end of the range that arrived
// first (NONE before).  Launched with 256 threads.
__global__ void __launch_bounds__(256) k_ploc(Tree T, const uint32_t* __restrict__ keys, uint32_t n,
                                              uint32_t* cluster, uint32_t* ends,
                                              uint32_t* counter, int width) {
  __shared__ uint8_t maps[8][32];
  const int lane = threadIdx.x & 31;
  uint32_t L = blockIdx.x * blockDim.x + threadIdx.x, R = L, split = L;
  bool alive = L < n;
  while (__any_sync(0xffffffffu, alive)) {
    if (alive) {
      // the parent range: towards the smaller gap
      const bool right = L == 0 || (R != n - 1 && code_gap(keys, R) < code_gap(keys, L - 1));
      __threadfence();
      const uint32_t other = atomicExch(&ends[right ? R : L - 1], right ? L : R);
      if (other == NONE) {
        alive = false;  // the sibling range is not done: its thread continues
      } else if (right) {
        split = R + 1;
        R = other;
      } else {
        split = L;
        L = other;
      }
      __threadfence();
    }
    const bool top = alive && L == 0 && R == n - 1;
    uint32_t m = __ballot_sync(0xffffffffu, alive && (R - L + 1 > PLOC_KEEP || top));
    while (m) {
      const int src = __ffs(m) - 1;
      m &= m - 1;
      ploc_merge(T, cluster, counter, __shfl_sync(0xffffffffu, L, src),
                 __shfl_sync(0xffffffffu, split, src), __shfl_sync(0xffffffffu, R, src),
                 __shfl_sync(0xffffffffu, top ? 1 : 0, src) != 0, width, maps[threadIdx.x >> 5], lane);
    }
    if (top) alive = false;
  }
}

// ------------------------------------------------------ treelet builder ----
__device__ __forceinline__ int delta(const uint32_t* keys, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  uint32_t a = keys[i], b = keys[j];
  if (a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
  return __clz(a ^ b);
}

// internal node i of the radix tree over sorted keys (Karras 2012, fig. 4)
__global__ void k_karras(const uint32_t* __restrict__ keys, int n, uint32_t* left, uint32_t* right,
                         uint32_t* parent_int, uint32_t* parent_leaf) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  int dmin = delta(keys, n, i, i - d);
  int lmax = 2;
  while (delta(keys, n, i, i + lmax * d) > dmin) lmax *= 2;
  int l = 0;
  for (int t = lmax / 2; t >= 1; t /= 2)
    if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  int j = i + l * d;
  int dnode = delta(keys, n, i, j);
  int s = 0;
  for (int div = 2;; div *= 2) {
    int t = (l + div - 1) / div;
    if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    if (t <= 1) break;
  }
  int gamma = i + s * d + min(d, 0);
  int lo = min(i, j), hi = max(i, j);
  uint32_t lc = (lo == gamma) ? ((uint32_t)gamma | LEAF_BIT) : (uint32_t)gamma;
  uint32_t rc = (hi == gamma + 1) ? ((uint32_t)(gamma + 1) | LEAF_BIT) : (uint32_t)(gamma + 1);
  left[i] = lc;
  right[i] = rc;
  if (lc & LEAF_BIT) parent_leaf[lc & ~LEAF_BIT] = (uint32_t)i;
  else parent_int[lc] = (uint32_t)i;
  if (rc & LEAF_BIT) parent_leaf[rc & ~LEAF_BIT] = (uint32_t)i;
  else parent_int[rc] = (uint32_t)i;
  if (i == 0) parent_int[0] = 0xffffffffu;
}

// Internal-node data (boxes, costs, counts, links) is written by other
// threads of k_bottom_up while it runs, so it is read through L2 only; leaf
// boxes come from an earlier kernel.
__device__ __forceinline__ GBox ref_box_cg(const Tree& T, uint32_t r) {
  return (r & LEAF_BIT) ? box_load(T.llo, T.lhi, r & ~LEAF_BIT) : box_load_cg(T.ilo, T.ihi, r);
}
__device__ __forceinline__ float ref_cost(const Tree& T, uint32_t r) {
  return (r & LEAF_BIT) ? C_TRI * box_area(box_load(T.llo, T.lhi, r & ~LEAF_BIT))
                        : __ldcg(&T.ilo[r].w);
}
__device__ __forceinline__ float ref_count_cg(const Tree& T, uint32_t r) {
  return (r & LEAF_BIT) ? 1.f : __ldcg(&T.ihi[r].w);
}
__device__ __forceinline__ uint32_t left_of(const Tree& T, uint32_t x) { return __ldcg(T.left + x); }
__device__ __forceinline__ uint32_t right_of(const Tree& T, uint32_t x) { return __ldcg(T.right + x); }
__device__ __forceinline__ void set_parent(const Tree& T, uint32_t r, uint32_t p) {
  if (r & LEAF_BIT) T.parent_leaf[r & ~LEAF_BIT] = p;
  else T.parent_int[r] = p;
}

// Dynamic-programming state of one treelet, one per warp in shared memory.
struct TreeletDP {
  float cost[128];    // SAH cost of the best subtree over each leaf subset
  float box[6][128];  // bounds of each leaf subset (lo xyz, hi xyz)
  uint8_t split[128]; // the subset's best first part
};

// Rebuilds the treelet rooted at internal node `root` (up to 7 leaves) with
// the SAH-optimal topology; the treelet's internal nodes are reused.  Called
// by all 32 lanes of a warp together: every lane forms the same treelet (the
// same loads), the lanes share the subsets of each size of the dynamic
// program, and lane 0 writes the new topology.
__device__ void optimize_treelet(const Tree& T, uint32_t root, TreeletDP& dp, int lane) {
  uint32_t leaves[7], inner[6];
  int nl = 2, ni = 1;
  leaves[0] = left_of(T, root);
  leaves[1] = right_of(T, root);
  inner[0] = root;
  while (nl < 7) {
    int best = -1;
    float ba = -1.f;
    for (int k = 0; k < nl; k++) {
      if (leaves[k] & LEAF_BIT) continue;
      float a = box_area(box_load_cg(T.ilo, T.ihi, leaves[k]));
      if (a > ba) {
        ba = a;
        best = k;
      }
    }
    if (best < 0) break;
    uint32_t x = leaves[best];
    inner[ni++] = x;
    leaves[best] = left_of(T, x);
    leaves[nl++] = right_of(T, x);
  }
  if (nl < 3) return;  // the same for every lane
  const int full = (1 << nl) - 1;
  if (lane < nl) {
    GBox b = ref_box_cg(T, leaves[lane]);
    const int S = 1 << lane;
    for (int a = 0; a < 3; a++) {
      dp.box[a][S] = b.lo[a];
      dp.box[3 + a][S] = b.hi[a];
    }
    dp.cost[S] = ref_cost(T, leaves[lane]);
  }
  __syncwarp();
  // subsets by size: every proper subset of S is complete before S
  for (int size = 2; size <= nl; size++) {
    for (int S = lane + 1; S <= full; S += 32) {
      if (__popc(S) != size) continue;
      const int low = S & -S;
      GBox b;
      for (int a = 0; a < 3; a++) {
        b.lo[a] = fminf(dp.box[a][S ^ low], dp.box[a][low]);
        b.hi[a] = fmaxf(dp.box[3 + a][S ^ low], dp.box[3 + a][low]);
        dp.box[a][S] = b.lo[a];
        dp.box[3 + a][S] = b.hi[a];
      }
      // subsets P of S containing the lowest bit, P != S
      float best = 3.0e38f;
      int bp = low;
      const int rest = S ^ low;
      for (int Q = (rest - 1) & rest;; Q = (Q - 1) & rest) {
        const int P = Q | low;  // P ranges over low + proper subsets of rest
        float c = dp.cost[P] + dp.cost[S ^ P];
        if (c < best) {
          best = c;
          bp = P;
        }
        if (Q == 0) break;
      }
      dp.cost[S] = C_INNER * box_area(b) + best;
      dp.split[S] = (uint8_t)bp;
    }
    __syncwarp();
  }
  if (lane == 0) {
    // rewrite: assign internal node indices top-down (root keeps its index)
    struct Item {
      int S;
      uint32_t node;
    };
    Item stk[8];
    int sp = 0, next_inner = 1;
    stk[sp++] = {full, root};
    while (sp) {
      Item it = stk[--sp];
      int P = dp.split[it.S], R = it.S ^ P;
      uint32_t ch[2];
      int sets[2] = {P, R};
      for (int c = 0; c < 2; c++) {
        int X = sets[c];
        if ((X & (X - 1)) == 0) {
          int k = __ffs(X) - 1;
          ch[c] = leaves[k];
        } else {
          ch[c] = inner[next_inner++];
          stk[sp++] = {X, ch[c]};
        }
        set_parent(T, ch[c], it.node);
      }
      T.left[it.node] = ch[0];
      T.right[it.node] = ch[1];
      float cnt = 0.f;
      // count = sum of leaf counts in S
      for (int k = 0; k < nl; k++)
        if (it.S & (1 << k)) cnt += ref_count_cg(T, leaves[k]);
      GBox b;
      for (int a = 0; a < 3; a++) {
        b.lo[a] = dp.box[a][it.S];
        b.hi[a] = dp.box[3 + a][it.S];
      }
      box_store(T.ilo, T.ihi, it.node, b, dp.cost[it.S], cnt);
    }
    __threadfence();  // before any lane of this warp reports the root upward
  }
  __syncwarp();
}

// Bounds, costs and counts bottom-up (the second thread to arrive at a node
// processes it); optionally treelet restructuring, done by the whole warp
// for each of its lanes' nodes in turn.  Launched with 256 threads.
__global__ void __launch_bounds__(256) k_bottom_up(Tree T, int n, int optimize) {
  __shared__ TreeletDP dps[8];
  const int lane = threadIdx.x & 31;
  TreeletDP& dp = dps[threadIdx.x >> 5];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool alive = i < n;
  uint32_t node = alive ? T.parent_leaf[i] : 0xffffffffu;
  while (__any_sync(0xffffffffu, alive)) {
    bool need = false;
    if (alive) {
      if (node == 0xffffffffu) {
        alive = false;
      } else {
        __threadfence();
        if (atomicAdd(&T.flags[node], 1u) == 0) {
          alive = false;  // the sibling subtree is not done: its thread continues
        } else {
          __threadfence();
          uint32_t l = left_of(T, node), r = right_of(T, node);
          GBox b = box_union(ref_box_cg(T, l), ref_box_cg(T, r));
          float cnt = ref_count_cg(T, l) + ref_count_cg(T, r);
          float cost = C_INNER * box_area(b) + ref_cost(T, l) + ref_cost(T, r);
          box_store(T.ilo, T.ihi, node, b, cost, cnt);
          need = optimize && cnt >= 7.f;
        }
      }
    }
    uint32_t m = __ballot_sync(0xffffffffu, need);
    while (m) {
      const int src = __ffs(m) - 1;
      m &= m - 1;
      optimize_treelet(T, __shfl_sync(0xffffffffu, node, src), dp, lane);
    }
    if (alive) {
      __threadfence();
      node = __ldcg(T.parent_int + node);
    }
  }
}

struct CollapseOut {
  uint4* nodes;           // 5 per node
  float4* rec_out;        // leaf-ordered primitive records
  uint32_t* leaf_of_id;
  uint32_t* counters;     // [0] nodes, [1] primitives, [2] error
  uint32_t n;             // primitives = capacity of nodes, records and queues
};

// gathers the primitives of a subtree with <= 3 of them
__device__ __forceinline__ int gather_small(const Tree& T, const uint32_t* sorted_prim, uint32_t r,
                                            uint32_t* out) {
  int cnt = 0;
  uint32_t stk[4];
  int sp = 0;
  stk[sp++] = r;
  while (sp) {
    uint32_t x = stk[--sp];
    if (x & LEAF_BIT) {
      if (cnt < 3) out[cnt] = sorted_prim[x & ~LEAF_BIT];
      cnt++;
    } else if (sp < 3) {
      stk[sp++] = T.right[x];
      stk[sp++] = T.left[x];
    }
  }
  return cnt;
}

// One wide node: it.x the binary subtree, it.y its index.
__device__ __forceinline__ void collapse_node(const Tree& T, const uint32_t* __restrict__ sorted_prim,
                                              const float4* __restrict__ rec_in, uint2 it,
                                              uint2* qout, uint32_t* qout_len,
                                              const CollapseOut& out, int width) {
  uint32_t kids[8];
  uint32_t slots = 0;  // 4 bits per kid: the slots its subtree may take (0: it is one slot)
  int nk = 0;
  if (it.x & LEAF_BIT) {  // a single-primitive scene
    kids[nk++] = it.x;
  } else if (!T.plan) {
    kids[nk++] = T.left[it.x];
    kids[nk++] = T.right[it.x];
    // the child of largest area is expanded, at most 6 times (2 -> 8 children);
    // a fixed trip count keeps the per-thread arrays in registers
#pragma unroll
    for (int ex = 0; ex < 6; ex++) {
      if (nk >= width) break;
      int best = -1;
      float ba = -1.f;
      for (int k = 0; k < nk; k++) {
        if ((kids[k] & LEAF_BIT) || ref_count(T, kids[k]) <= 3.f) continue;
        float a = box_area(box_load(T.ilo, T.ihi, kids[k]));
        if (a > ba) {
          ba = a;
          best = k;
        }
      }
      if (best < 0) break;
      uint32_t x = kids[best];
      kids[best] = T.left[x];
      kids[nk++] = T.right[x];
    }
  } else {
    // the node's children, then every child with slots to share out in turn:
    // at most 6 more; a fixed trip count keeps the arrays in registers
    const uint32_t k = (__ldg(T.plan + it.x) >> (3 * (width - 2))) & 7u;
    kids[0] = T.left[it.x];
    kids[1] = T.right[it.x];
    slots = k | (((uint32_t)width - k) << 4);
    nk = 2;
#pragma unroll
    for (int ex = 0; ex < 6; ex++) {
      int at = -1;
      uint32_t share = 0, have = 0;
      for (int q = 0; q < nk; q++) {
        if (at >= 0) break;
        uint32_t j = (slots >> (4 * q)) & 15u;
        if (j < 2 || (kids[q] & LEAF_BIT)) continue;
        const uint32_t plan = __ldg(T.plan + kids[q]);
        while (j >= 2 && !((plan >> (3 * (j - 2))) & 7u)) j--;
        if (j < 2) {
          slots &= ~(15u << (4 * q));
          continue;
        }
        at = q;
        have = j;
        share = (plan >> (3 * (j - 2))) & 7u;
      }
      if (at < 0) break;
      const uint32_t x = kids[at];
      kids[at] = T.left[x];
      kids[nk] = T.right[x];
      slots = (slots & ~(15u << (4 * at))) | (share << (4 * at)) | ((have - share) << (4 * nk));
      nk++;
    }
  }
  // classify and allocate
  int n_int = 0;
  uint32_t nprim = 0;
  uint32_t cnts[8];
  for (int k = 0; k < nk; k++) {
    float c = ref_count(T, kids[k]);
    if (!(kids[k] & LEAF_BIT) && (T.plan ? !((__ldg(T.plan + kids[k]) >> 21) & 1u) : c > 3.f)) {
      n_int++;
      cnts[k] = 0;
    } else if (c >= 1.f && c <= 3.f) {
      cnts[k] = (uint32_t)c;
      nprim += cnts[k];
    } else {  // a count a valid tree cannot have: flag it, write nothing
      atomicOr(&out.counters[2], 1u);
      return;
    }
  }
  uint32_t child_base = n_int ? atomicAdd(&out.counters[0], (uint32_t)n_int) : 0;
  uint32_t prim_base = nprim ? atomicAdd(&out.counters[1], nprim) : 0;
  uint32_t qbase = n_int ? atomicAdd(qout_len, (uint32_t)n_int) : 0;
  if (it.y >= out.n || child_base + (uint32_t)n_int > out.n || prim_base + nprim > out.n ||
      qbase + (uint32_t)n_int > out.n) {
    atomicOr(&out.counters[2], 2u);  // would overrun the buffers: the host rejects the tree
    return;
  }
  pt::WideChild wc[8];
  GBox parent;
  for (int a = 0; a < 3; a++) {
    parent.lo[a] = 3.0e38f;
    parent.hi[a] = -3.0e38f;
  }
  uint32_t off = 0, rank = 0;
  for (int k = 0; k < nk; k++) {
    GBox b = ref_box(T, kids[k]);
    parent = box_union(parent, b);
    for (int a = 0; a < 3; a++) {
      wc[k].box.lo[a] = b.lo[a];
      wc[k].box.hi[a] = b.hi[a];
    }
    if (cnts[k] == 0) {
      wc[k].internal = true;
      wc[k].count = 0;
      wc[k].prim_off = 0;
      qout[qbase + rank] = make_uint2(kids[k], child_base + rank);
      rank++;
    } else {
      wc[k].internal = false;
      wc[k].count = cnts[k];
      wc[k].prim_off = off;
      uint32_t pr[3];
      if (gather_small(T, sorted_prim, kids[k], pr) != (int)cnts[k]) {
        atomicOr(&out.counters[2], 4u);
        return;
      }
      for (uint32_t q = 0; q < cnts[k]; q++) {
        uint32_t dst = prim_base + off + q;
        out.rec_out[3 * dst] = rec_in[3 * pr[q]];
        out.rec_out[3 * dst + 1] = rec_in[3 * pr[q] + 1];
        out.rec_out[3 * dst + 2] = rec_in[3 * pr[q] + 2];
        out.leaf_of_id[pr[q]] = dst;
      }
      off += cnts[k];
    }
  }
  pt::Box pb;
  for (int a = 0; a < 3; a++) {
    pb.lo[a] = parent.lo[a];
    pb.hi[a] = parent.hi[a];
  }
  uint32_t words[20];
  pt::encode_node_dev(pb, wc, nk, child_base, prim_base, words, T.guard);
  uint4* dst = out.nodes + 5 * (size_t)it.y;
  for (int w = 0; w < 5; w++)
    dst[w] = make_uint4(words[4 * w], words[4 * w + 1], words[4 * w + 2], words[4 * w + 3]);
}

// One level of the wide tree; its length and the next level's are on the device.
__global__ void k_collapse(Tree T, const uint32_t* __restrict__ sorted_prim,
                           const float4* __restrict__ rec_in, const uint2* __restrict__ qin,
                           const uint32_t* __restrict__ qlen, uint2* qout, uint32_t* qout_len,
                           CollapseOut out, int width) {
  // an earlier level met an inconsistency, or the binary tree is incomplete: the
  // queue is not to be trusted
  const uint32_t err = __ldcg(out.counters + 2), made = __ldcg(out.counters + 3);
  if (err || (T.plan && out.n > 1 && made != out.n - 1)) return;
  const uint32_t nq = min(*qlen, out.n);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nq; t += gridDim.x * blockDim.x)
    collapse_node(T, sorted_prim, rec_in, qin[t], qout, qout_len, out, width);
}

// Leaf boxes in sorted (Morton) order, every leaf a cluster of its own, and
// the first entry of the collapse queue.
__global__ void k_gather_boxes(const float4* lo, const float4* hi, const uint32_t* order, uint32_t n,
                               float4* slo, float4* shi, uint32_t* cluster, uint2* queue,
                               uint32_t root) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t p = order[i];
  slo[i] = lo[p];
  shi[i] = hi[p];
  if (cluster) cluster[i] = i | LEAF_BIT;
  if (i == 0) queue[0] = make_uint2(root, 0u);
}

// Carves the builder's scratch arrays out of one device arena that persists
// across builds (grown only when a scene needs more), so a commit makes no
// allocation once the arena fits.
struct Carve {
  unsigned char* base;
  size_t off;
  template <typename T>
  void take(T** p, size_t n) {
    off = (off + 255) & ~(size_t)255;
    *p = base ? (T*)(base + off) : nullptr;
    off += (n ? n : 1) * sizeof(T);
  }
};

// Structural check, per node: the rules of check_node8, counting in cover
// how often each leaf position is referenced.
__global__ void __launch_bounds__(256) k_check_nodes(const uint4* __restrict__ nodes,
                                                     uint32_t nn, uint32_t n,
                                                     uint32_t* __restrict__ cover,
                                                     uint32_t* err) {
  const uint32_t k = blockIdx.x * 256u + threadIdx.x;
  if (k >= nn) return;
  const uint4 a = nodes[5 * (size_t)k], b = nodes[5 * (size_t)k + 1];
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};  // words 3..7 are read
  const bool ok = pt::check_node8(w, k, nn, n, [cover](uint64_t pi) {
    atomicAdd(&cover[pi], 1u);
    return true;
  });
  if (!ok) atomicOr(err, 8u);
}

// Counts in ids how often each leaf position is some primitive's position.
__global__ void __launch_bounds__(256) k_check_ids(const uint32_t* __restrict__ leaf_of_id,
                                                   uint32_t n, uint32_t* __restrict__ ids,
                                                   uint32_t* err) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= n) return;
  const uint32_t p = leaf_of_id[i];
  if (p >= n)
    atomicOr(err, 8u);
  else
    atomicAdd(&ids[p], 1u);
}

// Every leaf position must be covered by exactly one leaf slot and be the
// position of exactly one primitive.
__global__ void __launch_bounds__(256) k_check_cover(const uint32_t* __restrict__ cover,
                                                     const uint32_t* __restrict__ ids, uint32_t n,
                                                     uint32_t* err) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i < n && (cover[i] != 1u || ids[i] != 1u)) atomicOr(err, 8u);
}

}  // namespace

namespace pt {

// Builds the BVH8 of n primitive records (call order, on the device) into
// d_nodes / d_rec_out / d_leaf_of_id (allocated by the caller: n nodes,
// n records, n ids).  Returns the number of nodes and the depth (depth < 0:
// the collapse met an inconsistent tree and stopped before overrunning a
// buffer; -depth: 1 bad count, 2 capacity, 4 leaf gather mismatch; 8: the
// finished tree broke a structural rule; 16: incomplete or too deep).
// cluster: the tree is clustered, else rebuilt in treelets; guard: guarded
// grids (encode_node_dev).  Triangle meshes take both.  GB300, 2.1 M-triangle terrain: pt_commit 16.0 -> 4.3 ms (the
// treelet passes took 12.6), 64 frames at 1920x1080 76.9 -> 76.3 ms, a batch of
// eight terrains 72.0 -> 71.1 ms.  Scenes with other shapes keep the treelet
// tree and with it their images: see encode_node_dev on node boundaries.
cudaError_t build_bvh8_gpu(const float4* d_rec, const float4* d_xforms, uint32_t n,
                           uint4* d_nodes, float4* d_rec_out, uint32_t* d_leaf_of_id,
                           uint32_t* out_nodes, int* out_depth, int width, bool cluster, bool guard,
                           float cam_t0, float cam_t1, BuildArena* arena, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  if (width < 2 || width > 8) width = 8;
  float4 *lo = nullptr, *hi = nullptr, *ilo = nullptr, *ihi = nullptr, *slo = nullptr,
         *shi = nullptr, *cost = nullptr;
  uint32_t* plan = nullptr;
  uint32_t *keys = nullptr, *vals = nullptr, *keys2 = nullptr, *vals2 = nullptr, *left = nullptr,
           *right = nullptr, *entry = nullptr, *ends = nullptr, *counters = nullptr;
  uint32_t *pint = nullptr, *pleaf = nullptr, *flags = nullptr;
  unsigned int* cbox = nullptr;
  uint2 *qa = nullptr, *qb = nullptr;
  void* tmp = nullptr;
  size_t tmp_bytes = 0;
  uint32_t ni = n > 1 ? n - 1 : 1;
  int depth = 0;
  // nodes, primitives, error, tree nodes; then the queue length of each level
  constexpr int kLevels = 252;
  uint32_t h_cnt[4 + kLevels] = {1, 0, 0, 0, 1};
  unsigned int h_cbox[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
#define BV(x)                         \
  do {                                \
    e = (x);                          \
    if (e != cudaSuccess) goto done;  \
  } while (0)
  // the radix sort's temporary size (a query: no sorting, no allocation)
  BV(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, keys, keys2, vals, vals2, (int)n, 0, 30,
                                     st));
  {
    Carve cv{nullptr, 0};
    for (int pass = 0; pass < 2; pass++) {
      cv.off = 0;
      cv.take(&lo, n);
      cv.take(&hi, n);
      cv.take(&slo, n);
      cv.take(&shi, n);
      cv.take(&ilo, ni);
      cv.take(&ihi, ni);
      cv.take(&keys, n);
      cv.take(&vals, n);
      cv.take(&keys2, n);
      cv.take(&vals2, n);
      cv.take(&left, ni);
      cv.take(&right, ni);
      if (cluster) {
        cv.take(&entry, n);
        cv.take(&ends, n);
        cv.take(&cost, 2 * (size_t)ni);
        cv.take(&plan, ni);
      } else {
        cv.take(&pint, ni);
        cv.take(&pleaf, n);
        cv.take(&flags, ni);
      }
      cv.take(&counters, 4 + kLevels);
      cv.take(&cbox, 6);
      cv.take(&qa, n);
      cv.take(&qb, n);
      unsigned char* t8 = nullptr;
      cv.take(&t8, tmp_bytes);
      tmp = t8;
      if (pass == 0 && cv.off > arena->bytes) {  // grow the arena
        if (arena->p) cudaFree(arena->p);
        arena->p = nullptr;
        arena->bytes = 0;
        BV(cudaMalloc(&arena->p, cv.off));
        arena->bytes = cv.off;
      }
      cv.base = (unsigned char*)arena->p;
    }
  }
  BV(cudaMemcpyAsync(cbox, h_cbox, sizeof(h_cbox), cudaMemcpyHostToDevice, st));
  {
    uint32_t g = (n + 255) / 256;
    k_bounds<<<g < 608u ? g : 608u, 256, 0, st>>>(d_rec, d_xforms, n, cam_t0, cam_t1, lo, hi, cbox);
    k_morton<<<g, 256, 0, st>>>(lo, hi, n, cbox, keys, vals);
    BV(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, keys, keys2, vals, vals2, (int)n, 0, 30, st));
    // leaf bounds in sorted order
    Tree T;
    T.left = left;
    T.right = right;
    T.ilo = ilo;
    T.ihi = ihi;
    T.llo = slo;
    T.lhi = shi;
    T.cost = cost;
    T.plan = plan;
    T.parent_int = pint;
    T.parent_leaf = pleaf;
    T.flags = flags;
    T.root = n == 1 ? (0u | LEAF_BIT) : (cluster ? n - 2 : 0u);
    T.guard = guard;
    BV(cudaMemcpyAsync(counters, h_cnt, sizeof(h_cnt), cudaMemcpyHostToDevice, st));
    k_gather_boxes<<<g, 256, 0, st>>>(lo, hi, vals2, n, slo, shi, entry, qa, T.root);
    if (n > 1 && cluster) {
      BV(cudaMemsetAsync(ends, 0xff, (size_t)n * 4, st));
      k_ploc<<<g, 256, 0, st>>>(T, keys2, n, entry, ends, counters + 3, width);
    } else if (n > 1) {
      BV(cudaMemsetAsync(pint, 0xff, ni * 4, st));
      BV(cudaMemsetAsync(pleaf, 0xff, (size_t)n * 4, st));
      k_karras<<<(ni + 255) / 256, 256, 0, st>>>(keys2, (int)n, left, right, pint, pleaf);
      for (int round = 0; round <= PT_TREELET_ROUNDS; round++) {
        BV(cudaMemsetAsync(flags, 0, ni * 4, st));
        k_bottom_up<<<g, 256, 0, st>>>(T, (int)n, round > 0 ? 1 : 0);
      }
    }
    // collapse level by level; the host looks every few levels whether one is left
    CollapseOut co{d_nodes, d_rec_out, d_leaf_of_id, counters, n};
    const uint32_t cg = g < 2048u ? g : 2048u;
    while (true) {
      const int last = depth + 6 < kLevels - 1 ? depth + 6 : kLevels - 1;
      for (; depth < last; depth++) {
        k_collapse<<<cg, 128, 0, st>>>(T, vals2, d_rec, qa, counters + 4 + depth, qb,
                                       counters + 5 + depth, co, width);
        uint2* tq = qa;
        qa = qb;
        qb = tq;
      }
      BV(cudaMemcpyAsync(h_cnt, counters, sizeof(h_cnt), cudaMemcpyDeviceToHost, st));
      BV(cudaStreamSynchronize(st));
      if (h_cnt[2] || !h_cnt[4 + depth]) break;
      if (depth == kLevels - 1) {
        h_cnt[2] = 16;
        break;
      }
    }
    depth = 0;
    while (depth < kLevels && h_cnt[4 + depth]) depth++;
    if (cluster && n > 1 && !h_cnt[2] && h_cnt[3] != n - 1) h_cnt[2] = 16;
    // structural check of the result (keys and vals are free by now)
    if (!h_cnt[2] && n > 0) {
      const uint32_t nn = h_cnt[0];
      if (nn == 0 || nn > n) {
        h_cnt[2] = 8;
      } else {
        BV(cudaMemsetAsync(keys, 0, (size_t)n * 4, st));
        BV(cudaMemsetAsync(vals, 0, (size_t)n * 4, st));
        k_check_nodes<<<(nn + 255) / 256, 256, 0, st>>>(d_nodes, nn, n, keys, counters + 2);
        k_check_ids<<<g, 256, 0, st>>>(d_leaf_of_id, n, vals, counters + 2);
        k_check_cover<<<g, 256, 0, st>>>(keys, vals, n, counters + 2);
        BV(cudaMemcpyAsync(&h_cnt[2], counters + 2, 4, cudaMemcpyDeviceToHost, st));
        BV(cudaStreamSynchronize(st));
      }
    }
    BV(cudaGetLastError());
    *out_nodes = h_cnt[2] ? 0u : h_cnt[0];
    *out_depth = h_cnt[2] ? -(int)h_cnt[2] : depth;  // < 0: the collapse found an inconsistent tree
  }
done:
#undef BV
  return e;
}

}  // namespace pt
