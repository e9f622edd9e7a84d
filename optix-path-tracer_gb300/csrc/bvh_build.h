/*
 * bvh_build.h - BVH8 builders (host: bvh_host.cpp, GPU: bvh_gpu.cu).  Both
 * emit the 80-byte compressed node format documented in pt_types.h.
 */
#ifndef PT_BVH_BUILD_H
#define PT_BVH_BUILD_H

#include <math.h>
#include <stdint.h>
#include <string.h>
#include <vector>

#if defined(__CUDACC__)
#define PT_BVH_HD __host__ __device__
#else
#define PT_BVH_HD
#endif

#ifndef PT_BOX_SLACK
#define PT_BOX_SLACK 0.25f
#endif

namespace pt {

struct Box {
  float lo[3], hi[3];
};

struct WideChild {
  Box box;
  bool internal;
  uint32_t count;     /* leaf: primitives (1..3) */
  uint32_t prim_off;  /* leaf: offset from the node's prim_base */
};

/* Device scratch of the GPU builder, kept by its owner across builds (grown
 * on demand, freed with cudaFree by the owner). */
struct BuildArena {
  void* p = nullptr;
  size_t bytes = 0;
};

struct Bvh8Out {
  std::vector<uint32_t> nodes;       /* 20 words per node */
  std::vector<uint32_t> leaf_order;  /* primitive index at each leaf position */
  int depth = 0;                     /* levels of wide nodes */
};

// 2^e, -126 <= e <= 127.
PT_BVH_HD inline float exp2i(int e) {
  const uint32_t u = (uint32_t)(e + 127) << 23;
  float f;
  memcpy(&f, &u, 4);
  return f;
}
// floorf, without a call where the host has no instruction for it.
PT_BVH_HD inline float round_down(float v) {
  if (!(v > -8388608.0f && v < 8388608.0f)) return v;  // whole already, or not a number
  const float t = (float)(int)v;
  return t > v ? t - 1.0f : t;
}
// The exponent of a node's step along one axis and the grid's origin p, for the
// node's bounds [lo, hi].
PT_BVH_HD inline int box_grid(float lo, float hi, bool guard, float& p) {
  p = lo;
  const float ext = hi - lo;
  int ex = -126;
  if (ext > 0.f) {
    const float q = ext / 255.0f;
    uint32_t u;
    memcpy(&u, &q, 4);
    ex = (int)(u >> 23) - 126;  // q < 2^ex
    if (ex > 121) ex = 121;     // 255 * 2^121 is past every float
    while (ex > -126 && 255.0f * exp2i(ex - 1) >= ext) ex--;
    while (255.0f * exp2i(ex) < ext) ex++;
  }
  if (guard) {  // the origin may round downward by more than a step
    p = lo - exp2i(ex);
    while (hi - p > 254.0f * exp2i(ex)) {
      ex++;
      p = lo - exp2i(ex);
    }
  }
  return ex;
}

// Quantises the child boxes of one wide node into the 80-byte record: per
// axis the smallest power-of-two step s with 255 s >= the parent's extent;
// child bounds rounded outward to the step grid plus one step of slack for
// the float decode in traversal.  Float-only, so host and device agree.
// Without `guard` a bound on the node's own boundary has no step of slack (its
// q is clamped to 0 or 255), and as a decoded plane is off by up to 2^-8 of a
// step, a ray that hits the geometry within that distance of the boundary can
// pass it by (on closed scenes of large walls about one path in 10^5).  With
// `guard` the origin lies a step below the lower bound and a step is spare
// above, so every bound has its slack, and PT_BOX_SLACK of a step is enough
// of it: 64 times what the decode is off by.  (Where half an ulp of the origin is
// more than a step, the origin rounds back to the bound; there the padding of
// the boxes themselves, 8 ulps, is the slack.)  (A whole step made the boxes of
// a 2.1 M-triangle terrain larger by what costs 2.7 % of a render: 78.4
// against 76.3 ms.)  Guarded are all trees of triangle meshes that the GPU
// builds, and the host's trees except those of closed rooms of rectangles and
// boxes, those of one node and the few by area (deep ones).  These, and the GPU's
// trees of scenes with other shapes, are without the guard, as their images have
// been.
PT_BVH_HD inline void encode_node_dev(const Box& parent, const WideChild* ch, int nch,
                                      uint32_t child_base, uint32_t prim_base, uint32_t out[20],
                                      bool guard = false) {
  for (int w = 0; w < 20; w++) out[w] = 0;
  uint32_t e[3];
  float p[3], step[3];
  for (int a = 0; a < 3; a++) {
    const int ex = box_grid(parent.lo[a], parent.hi[a], guard, p[a]);
    e[a] = (uint32_t)(ex + 127);
    step[a] = exp2i(ex);
  }
  memcpy(&out[0], &p[0], 4);
  memcpy(&out[1], &p[1], 4);
  memcpy(&out[2], &p[2], 4);
  uint32_t imask = 0, rank = 0;
  // empty slots keep an inverted box (lo 255, hi 0): no ray passes its slab test
  uint32_t meta[2] = {0, 0}, qhi[3][2] = {{0, 0}, {0, 0}, {0, 0}};
  uint32_t qlo[3][2] = {{0xffffffffu, 0xffffffffu}, {0xffffffffu, 0xffffffffu},
                        {0xffffffffu, 0xffffffffu}};
  // internal children take the low slots in their given order (slot ==
  // rank, the offset of the child node from child_base), leaves follow
  int ord[8], no = 0;
  for (int i = 0; i < nch; i++)
    if (ch[i].internal) ord[no++] = i;
  for (int i = 0; i < nch; i++)
    if (!ch[i].internal) ord[no++] = i;
  for (int i = 0; i < nch; i++) {
    const WideChild& c = ch[ord[i]];
    uint32_t m;
    if (c.internal) {
      m = 0x80u | rank;
      imask |= 1u << i;
      rank++;
    } else {
      m = (c.count << 5) | c.prim_off;
    }
    meta[i >> 2] |= m << (8 * (i & 3));
    for (int a = 0; a < 3; a++) {
      float lo = (c.box.lo[a] - p[a]) / step[a], hi = (c.box.hi[a] - p[a]) / step[a];
      lo = guard ? round_down(lo - PT_BOX_SLACK) : round_down(lo) - 1.0f;
      hi = guard ? -round_down(-(hi + PT_BOX_SLACK)) : 1.0f - round_down(-hi);
      lo = lo > 0.0f ? (lo < 255.0f ? lo : 255.0f) : 0.0f;
      hi = hi > 0.0f ? (hi < 255.0f ? hi : 255.0f) : 0.0f;
      qlo[a][i >> 2] = (qlo[a][i >> 2] & ~(0xffu << (8 * (i & 3)))) | ((uint32_t)lo << (8 * (i & 3)));
      qhi[a][i >> 2] |= (uint32_t)hi << (8 * (i & 3));
    }
  }
  out[3] = e[0] | (e[1] << 8) | (e[2] << 16) | (imask << 24);
  out[4] = child_base;
  out[5] = prim_base;
  out[6] = meta[0];
  out[7] = meta[1];
  out[8] = qlo[0][0];
  out[9] = qlo[0][1];
  out[10] = qlo[1][0];
  out[11] = qlo[1][1];
  out[12] = qlo[2][0];
  out[13] = qlo[2][1];
  out[14] = qhi[0][0];
  out[15] = qhi[0][1];
  out[16] = qhi[1][0];
  out[17] = qhi[1][1];
  out[18] = qhi[2][0];
  out[19] = qhi[2][1];
}

// World box of a moving sphere (f = centre at time0 (3), radius, time0,
// time1, centre at time1 (3)) over every time a ray can carry: ray times lie
// in [cam_t0, cam_t0 + (cam_t1 - cam_t0)] (or the reverse), the centre
// c0 + ((t - time0) / (time1 - time0)) * (c1 - c0) is monotonic in t in
// floating point too, so the boxes at the two end times hold it.
PT_BVH_HD inline void moving_sphere_box(const float* f, float cam_t0, float cam_t1, float lo[3],
                                        float hi[3]) {
  const float te = cam_t0 + (cam_t1 - cam_t0);
  const float ta = fminf(fminf(f[4], cam_t0), te), tb = fmaxf(fmaxf(f[5], cam_t0), te);
  for (int a = 0; a < 3; a++) {
    const float d = f[6 + a] - f[a];
    const float ca = f[a] + ((ta - f[4]) / (f[5] - f[4])) * d;
    const float cb = f[a] + ((tb - f[4]) / (f[5] - f[4])) * d;
    lo[a] = fminf(ca, cb) - f[3];
    hi[a] = fmaxf(ca, cb) + f[3];
  }
}

// Structural rules of node k of an nn-node BVH8 over n primitives: internal
// children fill slots 0..r-1 with child index base + slot, each above k and
// below nn, the internal-slot mask (bits 24-31 of word 3) is (1 << r) - 1,
// and every leaf slot holds 1..3 primitive positions below n, each passed to
// on_prim (which counts how often a position is covered).  Returns false on
// the first broken rule.  The host validator and the GPU builder's check
// both apply it.
template <typename F>
PT_BVH_HD inline bool check_node8(const uint32_t* w, uint64_t k, uint64_t nn, uint64_t n,
                                  F&& on_prim) {
  uint32_t rank = 0;
  for (int i = 0; i < 8; i++) {
    const uint32_t meta = ((i < 4 ? w[6] : w[7]) >> (8 * (i & 3))) & 0xffu;
    if (!meta) continue;
    if (meta & 0x80u) {
      const uint64_t c = (uint64_t)w[4] + (meta & 7u);
      if ((meta & 7u) != rank || (uint32_t)i != rank || c <= k || c >= nn) return false;
      rank++;
    } else {
      const uint32_t cnt = meta >> 5, off = meta & 31u;
      if (cnt < 1 || cnt > 3) return false;
      for (uint32_t q = 0; q < cnt; q++) {
        const uint64_t pi = (uint64_t)w[5] + off + q;
        if (pi >= n || !on_prim(pi)) return false;
      }
    }
  }
  return (w[3] >> 24) == (1u << rank) - 1u;
}

inline void encode_node(const Box& parent, const WideChild* ch, int nch, uint32_t child_base,
                        uint32_t prim_base, uint32_t out[20], bool guard = false) {
  encode_node_dev(parent, ch, nch, child_base, prim_base, out, guard);
}
/* width: most children per node, 2..8 (the node format holds 8).  fit: wide
 * nodes chosen by the cost of the quantised boxes, on guarded grids
 * (encode_node_dev); else by the largest area, without. */
int build_bvh8_host(const std::vector<Box>& boxes, Bvh8Out& out, int width = 8, bool fit = false);
bool validate_bvh8(const Bvh8Out& b, size_t num_prims);

}  // namespace pt

#endif
