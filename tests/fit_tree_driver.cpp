// Host-built trees with wide nodes by cost: the structural rules at every
// width and size, and every primitive's box inside the decoded boxes of its
// leaf and of all nodes above it with slack to spare, with primitives of very
// different sizes.  One line per tree, "ALL PASS" at the end.
#include <cmath>
#include <cstdio>
#include <random>
#include "bvh_build.h"

using pt::Box;

static std::vector<Box> scene(size_t n, int kind) {
  std::mt19937 r(1 + (uint32_t)n);
  auto U = [&] { return (float)(r() >> 8) * (1.0f / 16777216.0f); };
  std::vector<Box> v;
  for (size_t i = 0; i < n; i++) {
    Box b;
    for (int a = 0; a < 3; a++) {
      const float size = kind == 1 && i == 0 ? 1000.f : 0.4f * U();  // 1: one that dwarfs the rest
      const float c = kind == 2 ? 0.25f : 20.f * U();                // 2: all at one place
      b.lo[a] = c - (kind == 3 && a == 1 ? 0.f : size);              // 3: flat ones
      b.hi[a] = c + (kind == 3 && a == 1 ? 0.f : size);
    }
    v.push_back(b);
  }
  return v;
}

// every leaf below node k lies inside the boxes on its path
static bool inside(const pt::Bvh8Out& t, const std::vector<Box>& boxes, uint32_t k, Box& all) {
  const uint32_t* w = &t.nodes[20 * (size_t)k];
  const float* p = (const float*)w;
  for (int a = 0; a < 3; a++) {
    all.lo[a] = INFINITY;
    all.hi[a] = -INFINITY;
  }
  for (int i = 0; i < 8; i++) {
    const uint32_t m = (w[6 + (i >> 2)] >> (8 * (i & 3))) & 255u;
    if (!m) continue;
    Box b;
    for (int a = 0; a < 3; a++) {
      b.lo[a] = INFINITY;
      b.hi[a] = -INFINITY;
    }
    if (m & 0x80u) {
      if (!inside(t, boxes, w[4] + (m & 7u), b)) return false;
    } else {
      for (uint32_t q = 0; q < m >> 5; q++) {
        const Box& x = boxes[t.leaf_order[w[5] + (m & 31u) + q]];
        for (int a = 0; a < 3; a++) {
          b.lo[a] = std::fmin(b.lo[a], x.lo[a]);
          b.hi[a] = std::fmax(b.hi[a], x.hi[a]);
        }
      }
    }
    for (int a = 0; a < 3; a++) {
      const double s = std::ldexp(1.0, (int)((w[3] >> (8 * a)) & 255u) - 127);
      const double lo = p[a] + s * ((w[8 + 2 * a + (i >> 2)] >> (8 * (i & 3))) & 255u);
      const double hi = p[a] + s * ((w[14 + 2 * a + (i >> 2)] >> (8 * (i & 3))) & 255u);
      // a sixteenth of a step at least, 16 times what the traversal's decode is off by
      if (lo > b.lo[a] - s / 16 || hi < b.hi[a] + s / 16) return false;
      all.lo[a] = std::fmin(all.lo[a], b.lo[a]);
      all.hi[a] = std::fmax(all.hi[a], b.hi[a]);
    }
  }
  return true;
}

int main() {
  bool all = true;
  for (int kind = 0; kind < 4; kind++)
    for (int width = 2; width <= 8; width++)
      for (size_t n : {1u, 2u, 3u, 4u, 8u, 9u, 25u, 400u}) {
        const std::vector<Box> boxes = scene(n, kind);
        pt::Bvh8Out t;
        pt::build_bvh8_host(boxes, t, width, true);
        Box b;
        const bool ok = pt::validate_bvh8(t, n) && inside(t, boxes, 0, b);
        printf("%s kind%d_w%d_n%zu\n", ok ? "PASS" : "FAIL", kind, width, n);
        all = all && ok;
      }
  if (all) printf("ALL PASS\n");
  return all ? 0 : 1;
}
