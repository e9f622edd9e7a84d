/*
 * pt_bvh.cuh - the parts of BVH8 traversal that the trace kernels
 * (pt_trace.cu) and the tail kernel (pt_tail.cu) share: the eight child boxes
 * of a node, its hit leaves as a primitive mask, and the primitive tests.
 */
#pragma once
#include "pt_device.cuh"

namespace ptd {

// Three-input max / min (one instruction each on sm_100+) and the paired
// FP32 fused multiply-add: a node step evaluates 8 children x 3 axes of
// (near, far) slab distances, so pairs share one instruction.
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// (a.x * s + t, a.y * s + t), each rounded once.
__device__ __forceinline__ float2 fma2s(float ax, float ay, float s, float t) {
  unsigned long long a, b, c, d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(ax), "f"(ay));
  asm("mov.b64 %0, {%1, %1};" : "=l"(b) : "f"(s));
  asm("mov.b64 %0, {%1, %1};" : "=l"(c) : "f"(t));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
  return r;
}

__device__ __forceinline__ WtRay wt_unpack(float4 w) {
  WtRay r;
  uint32_t k = __float_as_uint(w.w);
  r.kx = (int)(k & 3u);
  r.ky = (int)((k >> 2) & 3u);
  r.kz = (int)((k >> 4) & 3u);
  r.Sx = w.x;
  r.Sy = w.y;
  r.Sz = w.z;
  return r;
}

// Candidate of one primitive for a world-space ray (object space inside);
// MOTION: spheres may move (at the ray's `time`), else every sphere is static.
template <bool MOTION>
__device__ __forceinline__ bool prim_test(const DevScene& S, const PrimRec& p, V3 o, V3 d,
                                          const WtRay& wt, float tmin, float tmax, float& t,
                                          float& bu, float& bv, float time) {
  bu = bv = 0.f;
  if (S.tri_only) return tri_candidate(p, o, wt, tmin, tmax, t, bu, bv);
  int type = prim_type(p);
  if (type == PT_PRIM_TRIANGLE) return tri_candidate(p, o, wt, tmin, tmax, t, bu, bv);
  V3 oo = o, dd = d;
  int xf = prim_xform(p);
  if (xf >= 0) {
    const float4* I = S.xforms + 6 * xf + 3;
    oo = xpoint(I, o);
    dd = xvector(I, d);
  }
  if (type == PT_PRIM_SPHERE)
    return sphere_candidate_at(p, MOTION ? sphere_center(p, time) : v3(p.r0.x, p.r0.y, p.r0.z), oo,
                               dd, tmin, tmax, t);
  if (type == PT_PRIM_RECT) return rect_candidate(p, oo, dd, tmin, tmax, t);
  return box_candidate(p, oo, dd, tmin, tmax, t);
}

// A ray that hits nothing by definition: with a NaN in its origin or
// direction every primitive test fails or yields a NaN distance (but fminf /
// fmaxf would let it pass every box test).
__device__ __forceinline__ bool nan_ray(V3 o, V3 d) {
  return !(o.x == o.x && o.y == o.y && o.z == o.z && d.x == d.x && d.y == d.y && d.z == d.z);
}

// What the box tests need of a ray.
struct BoxRay {
  V3 o;
  float tmin, ix, iy, iz;
  bool negx, negy, negz;
  __device__ __forceinline__ void set_direction(V3 d) {
    const float eps = 1e-18f;
    float dx = fabsf(d.x) < eps ? copysignf(eps, d.x) : d.x;
    float dy = fabsf(d.y) < eps ? copysignf(eps, d.y) : d.y;
    float dz = fabsf(d.z) < eps ? copysignf(eps, d.z) : d.z;
    ix = 1.0f / dx;
    iy = 1.0f / dy;
    iz = 1.0f / dz;
    negx = ix < 0.f;
    negy = iy < 0.f;
    negz = iz < 0.f;
  }
};

// The hit children of a node.  Internal children fill the low slots (slot ==
// offset of the child node from child_base), leaves follow.  k1, k2: the two
// nearest hit internal children, entry distance (>= 0, so its bits order like
// the value) with the slot in the low 3 bits; the caller sets ihit and
// leafmask to 0 and k1, k2 to 0xffffffff.
struct NodeHits {
  uint32_t ihit, leafmask, child_base, pbase, mlo, mhi, k1, k2;
};

// Tests the eight child boxes of the node at nptr against [r.tmin, tlim].
__device__ __forceinline__ void node_step(const uint4* nptr, const BoxRay& r, float tlim,
                                          NodeHits& h) {
  uint4 n0 = __ldg(nptr), n1 = __ldg(nptr + 1), n2 = __ldg(nptr + 2), n3 = __ldg(nptr + 3),
        n4 = __ldg(nptr + 4);
  h.child_base = n1.x;
  h.pbase = n1.y;
  h.mlo = n1.z;
  h.mhi = n1.w;
  const uint32_t im = n0.w >> 24;
  // child bound q (8 bits) is read as the float f = 1 + q * 2^-15 built by
  // one byte permute; t = q*a + b = f*A + B with A = 2^15 a, B = b - A
  float sx = __uint_as_float((n0.w & 0xffu) << 23);
  float sy = __uint_as_float(((n0.w >> 8) & 0xffu) << 23);
  float sz = __uint_as_float(((n0.w >> 16) & 0xffu) << 23);
  float Ax = 32768.0f * (sx * r.ix), Ay = 32768.0f * (sy * r.iy), Az = 32768.0f * (sz * r.iz);
  float Bx = (__uint_as_float(n0.x) - r.o.x) * r.ix - Ax;
  float By = (__uint_as_float(n0.y) - r.o.y) * r.iy - Ay;
  float Bz = (__uint_as_float(n0.z) - r.o.z) * r.iz - Az;
  uint32_t nx0 = r.negx ? n3.z : n2.x, nx1 = r.negx ? n3.w : n2.y;
  uint32_t fx0 = r.negx ? n2.x : n3.z, fx1 = r.negx ? n2.y : n3.w;
  uint32_t ny0 = r.negy ? n4.x : n2.z, ny1 = r.negy ? n4.y : n2.w;
  uint32_t fy0 = r.negy ? n2.z : n4.x, fy1 = r.negy ? n2.w : n4.y;
  uint32_t nz0 = r.negz ? n4.z : n3.x, nz1 = r.negz ? n4.w : n3.y;
  uint32_t fz0 = r.negz ? n3.x : n4.z, fz1 = r.negz ? n3.y : n4.w;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const uint32_t sel = 0x7604u | ((uint32_t)(k & 3) << 4);
    float2 tx = fma2s(__uint_as_float(__byte_perm(k < 4 ? nx0 : nx1, 0x3F800000u, sel)),
                      __uint_as_float(__byte_perm(k < 4 ? fx0 : fx1, 0x3F800000u, sel)), Ax, Bx);
    float2 ty = fma2s(__uint_as_float(__byte_perm(k < 4 ? ny0 : ny1, 0x3F800000u, sel)),
                      __uint_as_float(__byte_perm(k < 4 ? fy0 : fy1, 0x3F800000u, sel)), Ay, By);
    float2 tz = fma2s(__uint_as_float(__byte_perm(k < 4 ? nz0 : nz1, 0x3F800000u, sel)),
                      __uint_as_float(__byte_perm(k < 4 ? fz0 : fz1, 0x3F800000u, sel)), Az, Bz);
    float tn = max3f(tx.x, ty.x, fmaxf(tz.x, r.tmin));
    float tf = min3f(tx.y, ty.y, fminf(tz.y, tlim));
    // an empty slot (meta 0) has an inverted box and fails here; were it
    // to pass (infinite slab distances), it is a leaf of no primitives.
    if (tn <= tf) {
      if ((im >> k) & 1u) {
        const uint32_t key = (__float_as_uint(tn) & 0xfffffff8u) | (uint32_t)k;
        h.k2 = min(h.k2, max(h.k1, key));
        h.k1 = min(h.k1, key);
        h.ihit |= 1u << k;
      } else {
        h.leafmask |= 1u << k;
      }
    }
  }
}

// The primitives of the hit leaves as bits over the node's range: bit j =
// record pbase + j (a node's leaves hold at most 24 primitives).
__device__ __forceinline__ uint32_t leaf_prims(const NodeHits& h) {
  uint32_t pm = 0, m = h.leafmask;
  while (m) {
    const int k = __ffs(m) - 1;
    m &= m - 1;
    const uint32_t meta = (k < 4 ? h.mlo : h.mhi) >> (8 * (k & 3));
    pm |= ((1u << ((meta >> 5) & 7u)) - 1u) << (meta & 31u);
  }
  return pm;
}

}  // namespace ptd
