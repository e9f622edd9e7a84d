// Host-built trees: "hash K W N FIT H" for boxes of kind K at width W (a hash of
// the nodes and the leaf order), and "nonfinite ok" if boxes with infinite
// bounds still give valid trees.
#include <cmath>
#include <cstdio>
#include <random>
#include "bvh_build.h"

using pt::Box;

static std::vector<Box> scene(size_t n, int kind, uint32_t seed) {
  std::mt19937 r(seed);
  auto U = [&] { return (float)(r() >> 8) * (1.0f / 16777216.0f); };
  std::vector<Box> v;
  for (size_t i = 0; i < n; i++) {
    Box b;
    for (int a = 0; a < 3; a++) {
      float c = 20.f * U() - 10.f, s = 0.4f * U();
      if (kind == 1 && i == 0) s = 1000.f;            // one that dwarfs the rest
      if (kind == 2) c = 0.25f;                       // all at one place
      if (kind == 3) c = std::floor(c), s = 0.25f;    // many coincide
      if (kind == 4 && a == 1) c = 0.f, s = 0.f;      // flat
      if (kind == 5) c = 1e6f * c + 1e7f;             // far from the origin
      b.lo[a] = c - s;
      b.hi[a] = c + s;
    }
    v.push_back(b);
  }
  return v;
}

int main() {
  for (int kind = 0; kind < 6; kind++)
    for (int width : {2, 5, 8})
      for (size_t n : {2u, 3u, 4u, 7u, 61u, 700u})
        for (int fit = 0; fit < 2; fit++) {
          pt::Bvh8Out t;
          pt::build_bvh8_host(scene(n, kind, 1 + (uint32_t)n), t, width, fit != 0);
          uint64_t h = 1469598103934665603ull;
          for (uint32_t w : t.nodes) h = (h ^ w) * 1099511628211ull;
          for (uint32_t w : t.leaf_order) h = (h ^ w) * 1099511628211ull;
          printf("hash %d %d %zu %d %016llx\n", kind, width, n, fit, (unsigned long long)h);
        }
  bool ok = true;
  for (int it = 0; it < 100; it++) {
    std::vector<Box> v = scene(2 + 5 * it, it % 6, 77 + it);
    for (size_t i = 0; i < v.size(); i += 1 + it % 7)
      for (int a = 0; a < 3; a++) {
        if ((i + a) % 5 == 0) v[i].hi[a] = INFINITY;
        if ((i + a) % 7 == 0) v[i].lo[a] = -INFINITY;
        if ((i + a) % 11 == 0) v[i].lo[a] = v[i].hi[a] = 3e38f;
      }
    for (int fit = 0; fit < 2; fit++) {
      pt::Bvh8Out t;
      pt::build_bvh8_host(v, t, 2 + it % 7, fit != 0);
      ok = ok && pt::validate_bvh8(t, v.size());
    }
  }
  printf("nonfinite %s\n", ok ? "ok" : "FAIL");
  return 0;
}
