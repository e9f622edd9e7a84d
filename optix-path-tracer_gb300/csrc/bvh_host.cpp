/*
 * bvh_host.cpp - host BVH8 builder: binned-SAH binary BVH, collapsed to
 * 8-wide nodes with 8-bit quantised child boxes (the node format of
 * pt_types.h).  Replaces the OptiX "Trbvh" acceleration the reference
 * requests for every group (e.g. host_includes/scenes.hpp:32,
 * host_includes/transforms.hpp:59).  The GPU builder (bvh_gpu.cu) produces
 * the same node format; this one serves small scenes and cross-checks.
 */
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>
#include "bvh_build.h"

namespace pt {

namespace {

// Four floats (x, y, z, unused): bounds are merged, binned and quantised a
// vector at a time, in the scalar order of operations.
typedef float f4 __attribute__((vector_size(16)));
typedef int i4 __attribute__((vector_size(16)));

struct VBox {
  f4 lo, hi;
};
struct BNode {
  VBox box;
  int left, right;    // internal children; left -1: a leaf
  int first, nprims;  // the subtree's primitives in `order`
};

inline f4 splat(float v) { return f4{v, v, v, v}; }
inline f4 vmin(f4 a, f4 b) { return b < a ? b : a; }
inline f4 vmax(f4 a, f4 b) { return a < b ? b : a; }
inline VBox merge(const VBox& a, const VBox& b) {
  return {vmin(a.lo, b.lo), vmax(a.hi, b.hi)};
}
inline float half_area(const VBox& a) {
  const f4 e = a.hi - a.lo;
  if (e[0] < 0) return 0.f;
  return e[0] * e[1] + e[1] * e[2] + e[2] * e[0];
}
inline VBox empty_box() { return {splat(FLT_MAX), splat(-FLT_MAX)}; }
inline Box to_box(const VBox& v) {
  Box b;
  for (int a = 0; a < 3; a++) {
    b.lo[a] = v.lo[a];
    b.hi[a] = v.hi[a];
  }
  return b;
}

// Binary tree by binned SAH.  One pass bins a node's primitives along all axes
// and keeps their bins for the partition; the sweeps visit the bins in use (an
// empty one repeats its neighbour's cost), of which a small node has few.
struct Bvh2 {
  static const int NB = 32;
  std::vector<VBox> boxes;
  std::vector<f4> cen;
  std::vector<uint32_t> bin;  // per primitive: its bins in the node at hand, a byte an axis
  std::vector<int> wrong;     // split: positions in the wrong part
  std::vector<uint32_t>& order;
  std::vector<BNode> nodes;
  const int leaf;  // most primitives of a leaf
  Bvh2(const std::vector<Box>& b, std::vector<uint32_t>& o, int most)
      : boxes(b.size()), cen(b.size()), bin(b.size()), wrong(2 * b.size() + 2), order(o), leaf(most) {
    for (size_t i = 0; i < b.size(); i++) {
      boxes[i] = {f4{b[i].lo[0], b[i].lo[1], b[i].lo[2], 0.f},
                  f4{b[i].hi[0], b[i].hi[1], b[i].hi[2], 0.f}};
      cen[i] = 0.5f * (boxes[i].lo + boxes[i].hi);
    }
    nodes.reserve(2 * b.size());
    build(0, (int)b.size(), bounds(0, (int)b.size()));
  }
  VBox bounds(int begin, int end) const {
    VBox bb = empty_box();
    for (int k = begin; k < end; k++) bb = merge(bb, boxes[order[k]]);
    return bb;
  }

  int build(int begin, int end, const VBox& bb) {
    const int ni = (int)nodes.size();
    const int n = end - begin;
    nodes.push_back({bb, -1, -1, begin, n});
    if (n <= leaf) return ni;
    int mid = begin;
    VBox lb, rb;
    if (n > 3) {
      mid = split(begin, end, lb, rb);
    } else if (n == 3) {  // leaf 1: the pair with the smaller box
      uint32_t* q = &order[begin];
      const float a01 = half_area(merge(boxes[q[0]], boxes[q[1]]));
      const float a02 = half_area(merge(boxes[q[0]], boxes[q[2]]));
      const float a12 = half_area(merge(boxes[q[1]], boxes[q[2]]));
      if (a12 < a01 && a12 <= a02) std::swap(q[0], q[2]);
      else if (a02 < a01) std::swap(q[1], q[2]);
    }
    if (mid == begin) {  // no plane separates the centroids: in the middle, or a pair and one
      mid = n > 3 ? begin + n / 2 : end - 1;
      lb = bounds(begin, mid);
      rb = bounds(mid, end);
    }
    const int l = build(begin, mid, lb), r = build(mid, end, rb);
    nodes[ni].left = l;
    nodes[ni].right = r;
    return ni;
  }

  // Partitions order[begin, end) at the cheapest plane between bins: the first
  // of the second part and the parts' boxes (begin: there is no plane).  Not
  // inlined: its bins would be part of every frame of build's recursion.
  __attribute__((noinline)) int split(int begin, int end, VBox& lb, VBox& rb) {
    const int n = end - begin;
    const int nb = leaf == 1 ? std::min((int)NB, 2 * n) : NB;  // few for few
    VBox cb = empty_box();
    for (int k = begin; k < end; k++) {
      const f4 c = cen[order[k]];
      cb.lo = vmin(cb.lo, c);
      cb.hi = vmax(cb.hi, c);
    }
    const f4 ext = cb.hi - cb.lo, scale = splat((float)nb) / ext;
    VBox bins[3][NB];
    int cnt[3][NB];
    for (int a = 0; a < 3; a++)
      for (int q = 0; q < nb; q++) {
        bins[a][q] = empty_box();
        cnt[a][q] = 0;
      }
    const i4 zero = {0, 0, 0, 0}, top = {nb - 1, nb - 1, nb - 1, nb - 1};
    for (int k = begin; k < end; k++) {
      const uint32_t p = order[k];
      i4 b = __builtin_convertvector((cen[p] - cb.lo) * scale, i4);
      b = b < zero ? zero : b;
      b = b > top ? top : b;
      bin[p] = (uint32_t)b[0] | (uint32_t)b[1] << 8 | (uint32_t)b[2] << 16;
      for (int a = 0; a < 3; a++) {
        bins[a][b[a]] = merge(bins[a][b[a]], boxes[p]);
        cnt[a][b[a]]++;
      }
    }
    float best = FLT_MAX;
    int best_ax = -1, best_bin = -1, best_n = 0;
    for (int ax = 0; ax < 3; ax++) {
      if (!(ext[ax] > 0.f)) continue;
      int at[NB], lc[NB], m = 0, c = 0;  // the bins in use, primitives up to each
      float la[NB];                      // and the area of their box
      VBox acc = empty_box();
      for (int q = 0; q < nb; q++) {
        if (!cnt[ax][q]) continue;
        acc = merge(acc, bins[ax][q]);
        c += cnt[ax][q];
        at[m] = q;
        lc[m] = c;
        la[m++] = half_area(acc);
      }
      acc = empty_box();
      for (int k = m - 1; k > 0; k--) {
        acc = merge(acc, bins[ax][at[k]]);
        const float cost = la[k - 1] * lc[k - 1] + half_area(acc) * (n - lc[k - 1]);
        if (cost < best) {
          best = cost;
          best_ax = ax;
          best_bin = at[k];
          best_n = lc[k - 1];
        }
      }
    }
    if (best_ax < 0) return begin;
    lb = rb = empty_box();
    for (int q = 0; q < nb; q++) (q < best_bin ? lb : rb) = merge(q < best_bin ? lb : rb, bins[best_ax][q]);
    // what lies in the wrong part, from either end, changes places (std::partition's
    // order, without a branch on each primitive)
    const int mid = begin + best_n, shift = 8 * best_ax;
    int *out = wrong.data(), *in = out + best_n + 1, no = 0, nin = 0;
    for (int k = begin; k < mid; k++) {
      out[no] = k;
      no += (int)((bin[order[k]] >> shift) & 255u) >= best_bin;
    }
    for (int k = end - 1; k >= mid; k--) {
      in[nin] = k;
      nin += (int)((bin[order[k]] >> shift) & 255u) < best_bin;
    }
    for (int k = 0; k < no; k++) std::swap(order[out[k]], order[in[k]]);
    return mid;
  }
};

// Wide nodes by cost.  The cost of a subtree is that of its wide nodes (one
// each) and of its leaves' primitives (kCostPrim each), times the area of the
// box that a ray is tested against before it reaches them: the child's box as
// it is quantised in its parent's grid.  That is the point of it: where a
// scene's bounds are much larger than most of its primitives, the root's step
// is as large as they are, and children cut small under the root would all be
// hit by every ray that comes near them.  By this cost they go into a node of
// their own with a fine grid (random spheres on a ground sphere of radius
// 1000: the root's step is 8, the spheres' diameter 0.4).
// GB300, by area -> by cost: 488 spheres 8.6 -> 3.9 node fetches a ray,
// 1920x1080 128 frames 155.8 -> 106 ms (28 refill lanes), one frame 2.03 -> 1.48 ms; 104 moving
// ones 1.60 -> 1.26 ms; the textures scene 2.14 -> 2.02 ms.
// A primitive test against a node step: 0.15 / 0.2 / 0.3 / 0.4 / 0.6 gave
// 110.6 / 110.7 / 109.7 / 111.5 / 112.1 ms on the spheres.
#ifndef PT_FIT_PRIM
#define PT_FIT_PRIM 0.3f
#endif
constexpr float kCostPrim = PT_FIT_PRIM;

// Every node with all its descendants down to seven levels is a sub-problem, so
// that is where the builder's time goes: loops of fixed length (a subtree of
// fewer primitives than slots repeats its last cost), and the choices noted only
// for the nodes that become wide nodes.  pt_commit on the GB300's host, ms, trees
// by area with scalar loops / by cost with scalar loops / this: 488 spheres 0.31 /
// 0.45 / 0.23, 1940 spheres 1.33 / 1.90 / 0.96, 2000 boxes 2.23 / 2.84 / 1.08.
struct Fit {
  const std::vector<BNode>& B;
  const int width;
  std::vector<float> inner;   // a node's cost below itself, as a wide node (more than 3 primitives)
  std::vector<uint8_t> split; // per node under the current wide node: slots of its left child by
                              // its own slots (0: it takes one)
  f4 p, step, inv;            // the current wide node's grid

  Fit(const std::vector<BNode>& b, int w) : B(b), width(w), inner(w ? b.size() : 0, 0.f),
                                         split(9 * inner.size(), 0) {
    for (size_t k = inner.size(); k-- > 1;)  // children come after their parents; the root is no child
      if (b[k].nprims > 3) inner[k] = open<false>((int)k, nullptr);
  }
  void set_grid(const VBox& b) {
    for (int a = 0; a < 3; a++) {
      float o;
      const int ex = box_grid(b.lo[a], b.hi[a], true, o);
      p[a] = o;
      step[a] = exp2i(ex);
      inv[a] = exp2i(-ex);
    }
  }
  float area(int c) const {  // of its box in the current wide node's grid (at steps 0..255)
    const VBox& b = B[c].box;
    const f4 l = (b.lo - p) * inv - splat(PT_BOX_SLACK), h = (b.hi - p) * inv + splat(PT_BOX_SLACK);
    const f4 top = splat(256.f), none = splat(0.f), hc = vmin(vmax(none, h), top);
    const f4 lo = whole(vmin(vmax(none, l), top)), ht = whole(hc);
    const f4 e = ((ht < hc ? ht + splat(1.f) : ht) - lo) * step;
    return e[0] * e[1] + e[1] * e[2] + e[2] * e[0];
  }
  static f4 whole(f4 v) { return __builtin_convertvector(__builtin_convertvector(v, i4), f4); }
  // as one child of the current wide node: a leaf (3 primitives cost less than
  // one more node), or a wide node of its own
  float slot(int c) const {
    const float a = area(c);
    return B[c].nprims <= 3 ? kCostPrim * a * (float)B[c].nprims : a + inner[c];
  }
  // cost[k]: the subtree of c in at most k slots of the current wide node, k =
  // 1..M.  NOTE: with the choices.
  template <int M, bool NOTE>
  void share(int c, float* cost) {
    const BNode& b = B[c];
    uint8_t* s = &split[9 * (size_t)c];
    cost[1] = slot(c);
    if (NOTE) s[1] = 0;
    if (M == 1) return;
    if (b.nprims <= 2) {
      const float two = b.nprims == 1 ? cost[1] : slot(b.left) + slot(b.right);
      for (int k = 2; k <= M; k++) cost[k] = std::min(cost[1], two);
      if (NOTE) {
        for (int k = 2; k <= M; k++) s[k] = two < cost[1] ? 1 | (2 << 4) : 0;
        if (b.nprims == 2) split[9 * (size_t)b.left + 1] = split[9 * (size_t)b.right + 1] = 0;
      }
      return;
    }
    float l[9], r[9];
    constexpr int N = M > 1 ? M - 1 : 1;
    share<N, NOTE>(b.left, l);
    share<N, NOTE>(b.right, r);
    for (int k = 2; k <= M; k++) {
      float best = cost[k - 1];
      int at = NOTE ? s[k - 1] : 0;
      for (int i = 1; i < k; i++) {
        const float v = l[i] + r[k - i];
        if (NOTE && v < best) at = i | (k << 4);
        best = v < best ? v : best;
      }
      cost[k] = best;
      if (NOTE) s[k] = (uint8_t)at;
    }
  }
  // the cost of node x's children where it is a wide node of at most M; NOTE:
  // into kids
  template <int M, bool NOTE>
  float open_as(int x, std::vector<int>* kids) {
    set_grid(B[x].box);
    float l[9], r[9];
    share<M - 1, NOTE>(B[x].left, l);
    share<M - 1, NOTE>(B[x].right, r);
    float best = FLT_MAX;
    int li = 1, ri = 1;  // where no cost is a number
    for (int k = NOTE ? 2 : M; k <= M; k++)
      for (int i = 1; i < k; i++) {
        const float v = l[i] + r[k - i];
        if (NOTE && v < best) {
          li = i;
          ri = k - i;
        }
        best = v < best ? v : best;
      }
    if (NOTE) {
      take(B[x].left, li, *kids);
      take(B[x].right, ri, *kids);
    }
    return best;
  }
  template <bool NOTE>
  float open(int x, std::vector<int>* kids) {
    switch (std::min(width, B[x].nprims)) {
      case 2: return open_as<2, NOTE>(x, kids);
      case 3: return open_as<3, NOTE>(x, kids);
      case 4: return open_as<4, NOTE>(x, kids);
      case 5: return open_as<5, NOTE>(x, kids);
      case 6: return open_as<6, NOTE>(x, kids);
      case 7: return open_as<7, NOTE>(x, kids);
      default: return open_as<8, NOTE>(x, kids);
    }
  }
  void take(int c, int k, std::vector<int>& kids) const {
    const uint8_t s = split[9 * (size_t)c + k];
    if (s == 0) {
      kids.push_back(c);
      return;
    }
    take(B[c].left, s & 15, kids);
    take(B[c].right, (s >> 4) - (s & 15), kids);
  }
};

}  // namespace

// The quantisation grid of encode_node extends the parent box upward by up
// to 255 steps; the parent itself must cover the children, which the caller
// guarantees (parent = union of children).
int build_bvh8_host(const std::vector<Box>& boxes, Bvh8Out& out, int width, bool fit) {
  if (width < 2 || width > 8) width = 8;
  size_t n = boxes.size();
  out.nodes.clear();
  out.leaf_order.clear();
  out.depth = 0;
  if (n == 0) return 0;
  std::vector<uint32_t> order(n);
  for (size_t i = 0; i < n; i++) order[i] = (uint32_t)i;
  Bvh2 b2(boxes, order, fit ? 1 : 3);
  const std::vector<BNode>& B = b2.nodes;
  Fit cost(B, fit ? width : 0);

  // breadth-first emission of wide nodes; each wide node records the binary
  // node it expands
  struct Pending {
    int bnode;
    int depth;
  };
  std::vector<Pending> queue;
  queue.push_back({0, 1});
  out.nodes.resize(20);  // root
  size_t head = 0;
  while (head < queue.size()) {
    Pending pd = queue[head];
    uint32_t self = (uint32_t)head;
    head++;
    out.depth = std::max(out.depth, pd.depth);
    // gather up to `width` children by expanding the largest internal child
    std::vector<int> kids;
    const BNode& bn = B[pd.bnode];
    if (bn.left < 0) {
      kids.push_back(pd.bnode);  // single-leaf root
    } else if (fit) {
      cost.open<true>(pd.bnode, &kids);  // the root has two primitives at least
    } else {
      kids.push_back(bn.left);
      kids.push_back(bn.right);
      while ((int)kids.size() < width) {
        int best = -1;
        float best_area = -1.f;
        for (size_t k = 0; k < kids.size(); k++) {
          const BNode& c = B[kids[k]];
          if (c.left < 0 || c.nprims <= 3) continue;  // leaf or small enough for one slot
          float a = half_area(c.box);
          if (a > best_area) {
            best_area = a;
            best = (int)k;
          }
        }
        if (best < 0) break;
        int bi = kids[best];
        kids[best] = B[bi].left;
        kids.push_back(B[bi].right);
      }
    }
    WideChild wc[8];
    int nch = (int)kids.size();
    uint32_t child_base = (uint32_t)queue.size();
    uint32_t prim_base = (uint32_t)out.leaf_order.size();
    uint32_t off = 0;
    VBox parent = empty_box();
    for (int k = 0; k < nch; k++) {
      const BNode& c = B[kids[k]];
      wc[k].box = to_box(c.box);
      parent = merge(parent, c.box);
      if (c.nprims <= 3) {
        wc[k].internal = false;
        wc[k].count = (uint32_t)c.nprims;
        wc[k].prim_off = off;
        for (int q = 0; q < c.nprims; q++) out.leaf_order.push_back(order[c.first + q]);
        off += (uint32_t)c.nprims;
      } else {
        wc[k].internal = true;
        wc[k].count = 0;
        wc[k].prim_off = 0;
        queue.push_back({kids[k], pd.depth + 1});
      }
    }
    out.nodes.resize(queue.size() * 20);
    encode_node(to_box(parent), wc, nch, child_base, prim_base, &out.nodes[(size_t)self * 20], fit);
  }
  return 0;
}

// Structural check of a BVH8 before it is uploaded: every internal child
// index lies after its parent and inside the node array, internal children
// fill the low slots with dense ranks (slot == rank),
// leaf ranges lie inside the primitive array and cover each primitive once.
bool validate_bvh8(const Bvh8Out& b, size_t num_prims) {
  size_t nn = b.nodes.size() / 20;
  if (num_prims == 0) return nn == 0 && b.leaf_order.empty();
  if (nn == 0 || b.leaf_order.size() != num_prims) return false;
  std::vector<uint8_t> seen(num_prims, 0);
  auto cover = [&](uint64_t pi) {
    const uint32_t id = b.leaf_order[pi];
    return id < num_prims && seen[id]++ == 0;
  };
  for (size_t k = 0; k < nn; k++)
    if (!check_node8(&b.nodes[k * 20], k, nn, num_prims, cover)) return false;
  for (uint8_t v : seen)
    if (v != 1) return false;
  return true;
}

}  // namespace pt
