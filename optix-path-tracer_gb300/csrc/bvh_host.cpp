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

struct BNode {
  Box box;
  int left = -1, right = -1;  // internal children
  int first = 0, count = 0;   // range in `order` (count: leaves only)
  int nprims = 0;             // primitives in the subtree
};

inline Box merge(const Box& a, const Box& b) {
  Box r;
  for (int k = 0; k < 3; k++) {
    r.lo[k] = std::min(a.lo[k], b.lo[k]);
    r.hi[k] = std::max(a.hi[k], b.hi[k]);
  }
  return r;
}
inline float half_area(const Box& a) {
  float ex = a.hi[0] - a.lo[0], ey = a.hi[1] - a.lo[1], ez = a.hi[2] - a.lo[2];
  if (ex < 0) return 0.f;
  return ex * ey + ey * ez + ez * ex;
}
inline Box empty_box() {
  Box b;
  for (int k = 0; k < 3; k++) {
    b.lo[k] = FLT_MAX;
    b.hi[k] = -FLT_MAX;
  }
  return b;
}

struct Bvh2 {
  const std::vector<Box>& boxes;
  std::vector<float> cx, cy, cz;
  std::vector<uint32_t>& order;
  std::vector<BNode> nodes;
  const int leaf;  // most primitives of a leaf
  Bvh2(const std::vector<Box>& b, std::vector<uint32_t>& o, int most)
      : boxes(b), order(o), leaf(most) {
    size_t n = b.size();
    cx.resize(n);
    cy.resize(n);
    cz.resize(n);
    for (size_t i = 0; i < n; i++) {
      cx[i] = 0.5f * (b[i].lo[0] + b[i].hi[0]);
      cy[i] = 0.5f * (b[i].lo[1] + b[i].hi[1]);
      cz[i] = 0.5f * (b[i].lo[2] + b[i].hi[2]);
    }
  }
  float cen(uint32_t p, int ax) const { return ax == 0 ? cx[p] : (ax == 1 ? cy[p] : cz[p]); }

  int build(int begin, int end) {
    int ni = (int)nodes.size();
    nodes.emplace_back();
    Box bb = empty_box(), cb = empty_box();
    for (int k = begin; k < end; k++) {
      uint32_t p = order[k];
      bb = merge(bb, boxes[p]);
      for (int a = 0; a < 3; a++) {
        cb.lo[a] = std::min(cb.lo[a], cen(p, a));
        cb.hi[a] = std::max(cb.hi[a], cen(p, a));
      }
    }
    int n = end - begin;
    nodes[ni].box = bb;
    nodes[ni].nprims = n;
    nodes[ni].first = begin;
    if (n <= leaf) {
      nodes[ni].count = n;
      return ni;
    }
    if (n <= 3) {  // leaf 1: the pair with the smaller box
      if (n == 3) {
        uint32_t* q = &order[begin];
        const float a01 = half_area(merge(boxes[q[0]], boxes[q[1]]));
        const float a02 = half_area(merge(boxes[q[0]], boxes[q[2]]));
        const float a12 = half_area(merge(boxes[q[1]], boxes[q[2]]));
        if (a12 < a01 && a12 <= a02) std::swap(q[0], q[2]);
        else if (a02 < a01) std::swap(q[1], q[2]);
      }
      const int l = build(begin, end - 1), r = build(end - 1, end);
      nodes[ni].left = l;
      nodes[ni].right = r;
      return ni;
    }
    const int NB = 32, nb = leaf == 1 ? std::min(NB, 2 * n) : NB;  // few for few
    float best = FLT_MAX;
    int best_ax = -1, best_bin = -1;
    for (int ax = 0; ax < 3; ax++) {
      float lo = cb.lo[ax], hi = cb.hi[ax];
      if (!(hi - lo > 0.f)) continue;
      Box bins[NB];
      int cnt[NB] = {0};
      for (int k = 0; k < nb; k++) bins[k] = empty_box();
      float scale = nb / (hi - lo);
      for (int k = begin; k < end; k++) {
        uint32_t p = order[k];
        int b = std::min(nb - 1, std::max(0, (int)((cen(p, ax) - lo) * scale)));
        cnt[b]++;
        bins[b] = merge(bins[b], boxes[p]);
      }
      float la[NB];
      int lc[NB];
      Box acc = empty_box();
      int c = 0;
      for (int k = 0; k < nb; k++) {
        acc = merge(acc, bins[k]);
        c += cnt[k];
        la[k] = half_area(acc);
        lc[k] = c;
      }
      acc = empty_box();
      c = 0;
      for (int k = nb - 1; k > 0; k--) {
        acc = merge(acc, bins[k]);
        c += cnt[k];
        if (lc[k - 1] == 0 || c == 0) continue;
        float cost = la[k - 1] * lc[k - 1] + half_area(acc) * c;
        if (cost < best) {
          best = cost;
          best_ax = ax;
          best_bin = k - 1;
        }
      }
    }
    int mid = begin + n / 2;
    if (best_ax >= 0) {
      float lo = cb.lo[best_ax], hi = cb.hi[best_ax];
      float scale = nb / (hi - lo);
      auto it = std::partition(order.begin() + begin, order.begin() + end, [&](uint32_t p) {
        int b = std::min(nb - 1, std::max(0, (int)((cen(p, best_ax) - lo) * scale)));
        return b <= best_bin;
      });
      mid = (int)(it - order.begin());
      if (mid == begin || mid == end) mid = begin + n / 2;
    } else {
      // all centroids coincide: split by index
      mid = begin + n / 2;
    }
    int l = build(begin, mid);
    int r = build(mid, end);
    nodes[ni].left = l;
    nodes[ni].right = r;
    return ni;
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
// ones 1.60 -> 1.26 ms; the textures scene 2.14 -> 2.02 ms; commit of the 488
// spheres within 0.1 ms of what it was.
// A primitive test against a node step: 0.15 / 0.2 / 0.3 / 0.4 / 0.6 gave
// 110.6 / 110.7 / 109.7 / 111.5 / 112.1 ms on the spheres.
#ifndef PT_FIT_PRIM
#define PT_FIT_PRIM 0.3f
#endif
constexpr float kCostPrim = PT_FIT_PRIM;

struct Fit {
  const std::vector<BNode>& B;
  const int width;
  std::vector<float> inner;   // a node's cost below itself, as a wide node
  std::vector<uint8_t> split; // per node under the current wide node: slots of its left child by
                              // its own slots (0: it takes one)
  float p[3], step[3], inv[3];

  Fit(const std::vector<BNode>& b, int w) : B(b), width(w), inner(w ? b.size() : 0, 0.f),
                                         split(9 * inner.size(), 0) {
    for (size_t k = w ? b.size() : 0; k-- > 0;)  // children come after their parents
      if (b[k].left >= 0) inner[k] = open((int)k);
  }
  float area(int c) const {  // of its box in the current wide node's grid
    float e[3];
    for (int a = 0; a < 3; a++) {
      const float lo = std::floor((B[c].box.lo[a] - p[a]) * inv[a] - PT_BOX_SLACK);
      const float hi = std::ceil((B[c].box.hi[a] - p[a]) * inv[a] + PT_BOX_SLACK);
      e[a] = (hi - lo) * step[a];
    }
    return e[0] * e[1] + e[1] * e[2] + e[2] * e[0];
  }
  // as one child of the current wide node: a leaf, or a wide node of its own
  float slot(int c, bool* leaf = nullptr) const {
    const float a = area(c), node = a + inner[c], prims = kCostPrim * a * (float)B[c].nprims;
    const bool is_leaf = B[c].left < 0 || (B[c].nprims <= 3 && prims <= node);
    if (leaf) *leaf = is_leaf;
    return is_leaf ? prims : node;
  }
  // cost[k]: the subtree of c in at most k slots, k = 1..the result, which is
  // `most` or its primitives if they are fewer
  int share(int c, int most, float* cost) {
    uint8_t* s = &split[9 * (size_t)c];
    cost[1] = slot(c);
    s[1] = 0;
    most = std::min(most, B[c].nprims);
    if (most < 2) return 1;
    float l[9], r[9];
    const int ml = share(B[c].left, most - 1, l), mr = share(B[c].right, most - 1, r);
    for (int k = 2; k <= most; k++) {
      cost[k] = cost[k - 1];
      s[k] = s[k - 1];
      for (int i = std::max(1, k - mr); i <= std::min(k - 1, ml); i++)
        if (l[i] + r[k - i] < cost[k]) {
          cost[k] = l[i] + r[k - i];
          s[k] = (uint8_t)(i | (k << 4));
        }
    }
    return most;
  }
  // node x as a wide node: its children's cost, their shares left in `split`
  float open(int x) {
    for (int a = 0; a < 3; a++) {
      const int ex = box_grid(B[x].box.lo[a], B[x].box.hi[a], true, p[a]);
      step[a] = std::ldexp(1.0f, ex);
      inv[a] = std::ldexp(1.0f, -ex);
    }
    float l[9], r[9];
    const int most = std::min(width, B[x].nprims);
    const int ml = share(B[x].left, most - 1, l), mr = share(B[x].right, most - 1, r);
    float best = FLT_MAX;
    uint8_t& s = split[9 * (size_t)x];
    s = 1 | (2 << 4);  // where no cost is a number
    for (int k = 2; k <= most; k++)
      for (int i = std::max(1, k - mr); i <= std::min(k - 1, ml); i++)
        if (l[i] + r[k - i] < best) {
          best = l[i] + r[k - i];
          s = (uint8_t)(i | (k << 4));
        }
    return best;
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
  // the children of node x as a wide node
  void children(int x, std::vector<int>& kids) {
    open(x);
    const uint8_t s = split[9 * (size_t)x];
    take(B[x].left, s & 15, kids);
    take(B[x].right, (s >> 4) - (s & 15), kids);
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
  b2.nodes.reserve(2 * n);
  b2.build(0, (int)n);
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
      cost.children(pd.bnode, kids);
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
    Box parent = empty_box();
    for (int k = 0; k < nch; k++) {
      const BNode& c = B[kids[k]];
      wc[k].box = c.box;
      parent = merge(parent, c.box);
      bool leaf = c.nprims <= 3;
      if (fit && c.left >= 0) cost.slot(kids[k], &leaf);
      if (leaf) {
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
    encode_node(parent, wc, nch, child_base, prim_base, &out.nodes[(size_t)self * 20], fit);
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
