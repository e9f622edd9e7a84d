/*
 * pt_shade.cuh - one bounce of a path: the arithmetic that the wavefront
 * kernels (pt_kernels.cu) and the tail kernel (pt_tail.cu) share.  A bounce
 * takes and returns values in registers; the callers move path state between
 * queues (wavefront) or keep it (tail).
 */
#pragma once
#include "pt_device.cuh"
#include "pt_guide.cuh"
#include "pt_internal.h"
#include "pt_wave.cuh"

namespace ptd {
// ---------------------------------------------------------- path state ----
// st.x = seed, st.y = path id in the chunk, st.z = depth | prevSpecular<<16 |
// scene<<17 (batch), st.w = pdf of the last BSDF sample (consistent mode)

// Depth limit and Russian roulette of a path (per render, or per scene of a
// batch).
struct PathCtl {
  int max_depth, rr_enable, rr_depth;
};
__device__ __forceinline__ void finalize_path(const WaveState& W, uint32_t pid, V3 col) {
  // de_nan, programs/raygen.cu:126-134
  if (!(col.x == col.x)) col.x = 0.f;
  if (!(col.y == col.y)) col.y = 0.f;
  if (!(col.z == col.z)) col.z = 0.f;
  __stcs(&W.results[pid], make_float4(col.x, col.y, col.z, 1.f));
}

// raygen.cu:81-122 after the closest-hit program: event dispatch, next
// ray, Russian roulette, depth limit.
struct Tail {
  int event;  // 0 bounced, 1 cancelled, 2 hit light
  bool isSpecular;
  V3 origin, direction;
};

// raygen.cu:81-122 after the closest-hit program: event dispatch, Russian
// roulette, depth limit.  Returns whether the path continues (its next ray
// is tl's); else col is its colour.
__device__ __forceinline__ bool path_advance(const PathCtl& ctl, uint4& st, V3& thr, V3& rad,
                                             const Tail& tl, V3& col) {
  uint32_t depth = st.z & PT_ST_DEPTH_MASK;
  bool prevSpec = (st.z >> PT_ST_SPEC_BIT) & 1u;
  if (tl.event == 2) {
    if (depth == 0 || prevSpec) rad += thr;
    col = rad;
    return false;
  }
  if (tl.event == 1) {
    col = rad;
    return false;
  }
  prevSpec = tl.isSpecular;
  if (ctl.rr_enable) {
    float prob = max_component(thr);
    if ((int)depth > ctl.rr_depth) {
      if (rnd(st.x) >= prob) {
        col = rad + thr;
        return false;
      }
      thr *= 1.f / prob;
    }
  }
  depth++;
  if ((int)depth >= ctl.max_depth) {
    col = v3(0.f);
    return false;
  }
  st.z = (st.z & PT_ST_KEEP_MASK) | depth | ((uint32_t)prevSpec << PT_ST_SPEC_BIT);
  return true;
}

// Segment of a batch chunk that holds path `pid` (binary search over the
// segments' first paths).
__device__ __forceinline__ uint32_t find_seg(const BatchSeg* __restrict__ segs, uint32_t lo,
                                             uint32_t hi, uint32_t pid, bool by_pixel) {
  // invariant: segs[lo].off <= pid, answer in [lo, hi)
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    uint32_t off = by_pixel ? segs[mid].pix_off : segs[mid].path_off;
    if (off <= pid) lo = mid;
    else hi = mid;
  }
  return lo;
}

// A new path: its state, camera ray and time (renderPixel up to color()'s
// loop, raygen.cu:148-162, 50-69).
struct NewPath {
  uint4 st;
  Ray3 ray;
  float tm;
};

template <bool BATCH>
__device__ __forceinline__ NewPath new_path(const DevScene& S0, const WaveCtl& ctl,
                                            const BatchRefs& br, uint32_t pid) {
  uint32_t width = (uint32_t)ctl.width, height = (uint32_t)ctl.height;
  uint32_t wh_m = ctl.wh_m, wh_l = ctl.wh_l, w_m = ctl.w_m, w_l = ctl.w_l;
  uint32_t frame0 = (uint32_t)ctl.frame0, local = pid, scene = 0;
  const DevScene* Sp = &S0;
  if (BATCH) {
    const BatchSeg& sg = br.segs[find_seg(br.segs, ctl.seg_begin, ctl.seg_end, pid, false)];
    scene = sg.scene;
    const BatchScene& B = br.scenes[scene];
    Sp = &B.S;
    width = (uint32_t)B.width;
    height = (uint32_t)B.height;
    wh_m = B.wh_m;
    wh_l = B.wh_l;
    w_m = B.w_m;
    w_l = B.w_l;
    frame0 = sg.frame0;
    local = pid - sg.path_off;
  }
  const DevScene& S = *Sp;
  uint32_t WH = width * height;
  uint32_t fr = fastdiv(local, wh_m, wh_l);
  uint32_t frame = frame0 + fr;
  uint32_t pix = local - fr * WH;
  uint32_t y = fastdiv(pix, w_m, w_l);
  uint32_t x = pix - y * width;
  uint32_t seed = tea64(width * y + x, frame);
  NewPath np;
  np.ray = camera_ray(S.cam, x, y, width, height, seed);
  // color(): prd.time draw, programs/raygen.cu:69
  np.tm = S.cam.time0 + rnd(seed) * (S.cam.time1 - S.cam.time0);
  np.st = make_uint4(seed, pid, scene << PT_ST_SCENE_SHIFT, 0u);
  return np;
}

// Scene and path controls of a path: the render's, or its batch scene's.
template <bool BATCH>
__device__ __forceinline__ const DevScene& path_scene(const DevScene& S0, const BatchRefs& br,
                                                      uint32_t stz) {
  return BATCH ? br.scenes[stz >> PT_ST_SCENE_SHIFT].S : S0;
}
template <bool BATCH>
__device__ __forceinline__ PathCtl path_ctl(const WaveCtl& ctl, const BatchRefs& br,
                                            uint32_t stz) {
  PathCtl pc;
  if (BATCH) {
    const BatchScene& B = br.scenes[stz >> PT_ST_SCENE_SHIFT];
    pc.max_depth = B.max_depth;
    pc.rr_enable = B.rr_enable;
    pc.rr_depth = B.rr_depth;
  } else {
    pc.max_depth = ctl.max_depth;
    pc.rr_enable = ctl.rr_enable;
    pc.rr_depth = ctl.rr_depth;
  }
  return pc;
}

// Direct_Light (programs/materials/light_sample.cuh:36-73) up to the shadow
// ray.  Returns 0: no contribution, stop here; 1: shadow ray queued.
__device__ __forceinline__ int nee_begin(const DevScene& S, uint32_t& seed, V3 P, V3 N,
                                         bool isLight, V3& Wi, float& lightPDF, int& index) {
  int numLights = S.num_lights;
  if (numLights == 0) return 0;
  index = ((int)(rnd(seed) * numLights)) % numLights;
  if (isLight && numLights == 1) return 0;
  GpuLight L = load_light(S.lights, index);
  Wi = light_sample(L, P, seed);
  lightPDF = light_pdf(L, P, Wi);
  if (dot(Wi, N) < 0.f) return 0;
  return 1;
}

// programs/materials/light_sample.cuh:76-103: MIS after the shadow test.
__device__ __forceinline__ V3 nee_end(const DevScene& S, const GpuMaterial& m, uint32_t& seed,
                                      V3 P, V3 Wo, V3 N, V3 Wi, float lightPDF, int index,
                                      bool occluded) {
  V3 directLight = v3(0.f);
  if (occluded) return v3(0.f);
  GpuLight L = load_light(S.lights, index);
  V3 emission = v3(L.ex, L.ey, L.ez);
  if (lightPDF != 0.f && !isNull(emission)) {
    float matPDF = 0.f;
    V3 matValue = brdf_eval(m, Wo, Wi, N, matPDF);
    if (matPDF != 0.f && !isNull(matValue)) {
      float f = 1u * lightPDF, g = 1u * matPDF;
      float weight = (f * f) / (f * f + g * g);
      directLight += matValue * emission * weight / lightPDF;
    }
  }
  Wi = brdf_sample(m, Wo, N, seed);
  float matPDF = 0.f;
  V3 matValue = brdf_eval(m, Wo, Wi, N, matPDF);
  if (matPDF != 0.f && !isNull(matValue)) {
    lightPDF = light_pdf(L, P, Wi);
    if (!lightPDF || isNull(emission)) return directLight;
    float f = 1u * matPDF, g = 1u * lightPDF;
    float weight = (f * f) / (f * f + g * g);
    directLight += matValue * emission * weight / matPDF;
  }
  return directLight;
}

// Closest-hit continuation after Direct_Light for the NEE materials
// (lambertian.cu:55-72, oren_nayar.cu:56-69, diffuse_light.cu:40-47).
__device__ __forceinline__ void after_nee(const GpuMaterial& m, uint32_t& seed, V3 P, V3 Wo, V3 N,
                                          V3 direct, V3& thr, V3& rad, Tail& tl) {
  rad += thr * direct;
  if (m.type == PT_MAT_DIFFUSE_LIGHT) {
    if (dot(N, Wo) < 0.f) thr *= v3(m.c0x, m.c0y, m.c0z);
    tl.event = 2;
    return;
  }
  V3 Wi = brdf_sample(m, Wo, N, seed);
  float pdf = 0.f;
  V3 attenuation = brdf_eval(m, Wo, Wi, N, pdf);
  tl.event = 0;
  tl.origin = P;
  tl.direction = Wi;
  thr *= clamp3(attenuation / pdf, 0.f, 1.f);
  tl.isSpecular = false;
}

__device__ __forceinline__ V3 env_lookup(const GpuMiss& ms, float u, float v) {
  if (!(u == u) || !(v == v) || fabsf(u) > 1e6f || fabsf(v) > 1e6f) return v3(0.f);
  float x = u * (float)ms.w - 0.5f, y = v * (float)ms.h - 0.5f;
  float fx = floorf(x), fy = floorf(y);
  float ax = x - fx, ay = y - fy;
  int ix0 = (int)fx % ms.w; if (ix0 < 0) ix0 += ms.w;
  int iy0 = (int)fy % ms.h; if (iy0 < 0) iy0 += ms.h;
  int ix1 = ix0 + 1 == ms.w ? 0 : ix0 + 1;
  int iy1 = iy0 + 1 == ms.h ? 0 : iy0 + 1;
  float4 e00 = __ldg(ms.env + iy0 * ms.w + ix0), e10 = __ldg(ms.env + iy0 * ms.w + ix1);
  float4 e01 = __ldg(ms.env + iy1 * ms.w + ix0), e11 = __ldg(ms.env + iy1 * ms.w + ix1);
  V3 c00 = f4xyz(e00), c10 = f4xyz(e10), c01 = f4xyz(e01), c11 = f4xyz(e11);
  return (c00 * (1.f - ax) + c10 * ax) * (1.f - ay) + (c01 * (1.f - ax) + c11 * ax) * ay;
}

// The colours of a textured material at a hit (Get_Parameters of the
// closest-hit programs).  Compiled only into the shading kernels of scenes
// with textures (the TEX variants): untextured shading never computes the
// texture coordinates.
__device__ __forceinline__ void apply_textures(const DevScene& S, GpuMaterial& m, const PrimRec& p,
                                               V3 ro, V3 rd, float t, float bu, float bv,
                                               float tm) {
  HitRecord rec = hit_record(S, p, ro, rd, t, bu, bv, true, tm);
  resolve_textures(S, m, rec.u, rec.v, rec.P, rec.tindex);
}

// programs/miss.cu:30-95; returns the multiplier applied to throughput.
__device__ __forceinline__ V3 miss_color(const GpuMiss& ms, V3 d) {
  if (ms.type == 0) {
    V3 unit_direction = normalize(d);
    float t = 0.5f * (unit_direction.y + 1.f);
    V3 c = (1.f - t) * v3(ms.c1x, ms.c1y, ms.c1z);
    c += t * v3(ms.c2x, ms.c2y, ms.c2z);
    return c;
  }
  if (ms.type == 1) return v3(ms.c1x, ms.c1y, ms.c1z);
  if (ms.type == 3) {
    float theta = pt_atan2f(d.x, d.z);
    float phi = PTM_PI * 0.5f - pt_acosf(d.y);
    float u = (theta + PTM_PI) * (0.5f * (1.0f / PTM_PI));
    float v = 0.5f * (1.f + pt_sinf(phi));
    return env_lookup(ms, u, v);
  }
  float u, v;
  if (ms.spherical) {
    env_uv(d, u, v);
  } else {
    float theta = pt_atan2f(d.x, d.z);
    theta = theta < 0.f ? theta + (2.f * PI_F) : theta;
    float phi = pt_acosf(d.y);
    u = 1.f - (theta / (2.f * PI_F));
    v = phi / PI_F;
  }
  return 2.f * env_lookup(ms, u, v);
}

// ---------------------------------------------------- reference mode ------
// Direct_Light's context while its shadow ray is in flight.
struct NeeCtx {
  V3 P, N, Wo, Wi;
  float lightPDF;
  int lindex;
  uint32_t mid;
  bool textured;  // the material's colours come from textures:
  V3 tcol;        // its colour at this hit (Direct_Light needs it)
};

enum { STEP_ENDED = 0, STEP_TAIL = 1, STEP_SHADOW = 2 };

// The closest-hit program of a hit, or the miss program (leaf PT_NO_HIT; then
// col is the path's colour: STEP_ENDED).  STEP_SHADOW: Direct_Light waits for
// the shadow ray of n; STEP_TAIL: the bounce is complete (path_advance next).
template <bool TEX>
__device__ __forceinline__ int shade_step(const DevScene& S, float4 hit, V3 ro, V3 rd, float tm,
                                          uint4& st, V3& thr, V3& rad, NeeCtx& n, Tail& tl,
                                          V3& col) {
  tl.event = 1;
  tl.isSpecular = false;
  n.textured = false;
  uint32_t leaf = __float_as_uint(hit.w);
  if (leaf == PT_NO_HIT) {
    thr *= miss_color(S.miss, rd);
    col = rad + clamp3(thr, 0.f, 1.f);  // raygen.cu:81-82
    return STEP_ENDED;
  }
  PrimRec p = load_prim(S.prims, leaf);
  HitRecord rec = hit_record(S, p, ro, rd, hit.x, hit.y, hit.z, false, tm);
  n.mid = rec.index;
  GpuMaterial m = load_material(S.mats, n.mid);
  n.textured = TEX && (m.tex0 >= 0 || m.tex1 >= 0);
  if (n.textured) {
    apply_textures(S, m, p, ro, rd, hit.x, hit.y, hit.z, tm);
    n.tcol = v3(m.c0x, m.c0y, m.c0z);
  }
  n.P = rec.P;
  n.Wo = rec.Wo;
  n.N = rec.shading_normal;
  V3 P = n.P, Wo = n.Wo, N = n.N;
  switch (m.type) {
    case PT_MAT_LAMBERTIAN:
    case PT_MAT_OREN_NAYAR:
    case PT_MAT_DIFFUSE_LIGHT: {
      bool isLight = m.type == PT_MAT_DIFFUSE_LIGHT;
      if (nee_begin(S, st.x, P, N, isLight, n.Wi, n.lightPDF, n.lindex)) {
        return STEP_SHADOW;
      } else {
        after_nee(m, st.x, P, Wo, N, v3(0.f), thr, rad, tl);
      }
      break;
    }
    case PT_MAT_METAL: {  // programs/materials/metal.cu:38-56
      V3 reflected = reflect(-Wo, N);
      tl.direction = reflected + m.p0 * random_in_unit_sphere(st.x);
      tl.event = 0;
      tl.origin = P;
      thr *= v3(m.c0x, m.c0y, m.c0z);
      tl.isSpecular = true;
      break;
    }
    case PT_MAT_DIELECTRIC: {  // programs/materials/dielectric.cu:46-96
      float ref_idx = m.p0;
      V3 Wd = -rec.Wo;
      V3 Nd = N;
      V3 absorption = v3(1.f);
      float ni_over_nt;
      float cosine = dot(Wd, Nd);
      if (cosine > 0.f) {
        Nd = -Nd;
        ni_over_nt = ref_idx;
        cosine = ref_idx * cosine / length(Wd);
      } else {
        ni_over_nt = 1.f / ref_idx;
        cosine = -cosine / length(Wd);
      }
      V3 refracted = v3(0.f);
      float reflect_prob;
      if (Refract(Wd, Nd, ni_over_nt, refracted))
        reflect_prob = schlick(cosine, ref_idx);
      else
        reflect_prob = 1.f;
      if (rnd(st.x) < reflect_prob)
        tl.direction = reflect(Wd, Nd);
      else
        tl.direction = normalize(refracted);
      tl.event = 0;
      tl.origin = P;
      thr *= (v3(m.c0x, m.c0y, m.c0z) * absorption);
      tl.isSpecular = true;
      break;
    }
    case PT_MAT_TORRANCE_SPARROW:
    case PT_MAT_ASHIKHMIN_SHIRLEY: {
      V3 Wn = brdf_sample(m, Wo, N, st.x);
      float pdf = 0.f;
      V3 attenuation = brdf_eval(m, Wo, Wn, N, pdf);
      tl.event = 0;
      tl.origin = P;
      tl.direction = Wn;
      if (m.type == PT_MAT_TORRANCE_SPARROW)
        thr *= clamp3(attenuation / pdf, 0.f, 1.f);
      else
        thr *= clamp3(attenuation, 0.f, 1.f);
      tl.isSpecular = true;
      break;
    }
    default:
      tl.event = 1;
  }
  return STEP_TAIL;
}

// After the shadow test: the rest of Direct_Light and the continuation.
__device__ __forceinline__ void finish_step(const DevScene& S, uint4& st, V3& thr, V3& rad,
                                            const NeeCtx& n, bool occluded, Tail& tl) {
  tl.event = 1;
  tl.isSpecular = false;
  GpuMaterial m = load_material(S.mats, n.mid);
  if (m.tex0 >= 0) {  // NEE materials (Lambertian, Oren-Nayar, diffuse light) read only c0
    m.c0x = n.tcol.x;
    m.c0y = n.tcol.y;
    m.c0z = n.tcol.z;
  }
  V3 direct = nee_end(S, m, st.x, n.P, n.Wo, n.N, n.Wi, n.lightPDF, n.lindex, occluded);
  after_nee(m, st.x, n.P, n.Wo, n.N, direct, thr, rad, tl);
}

// Radiance and sampling density of an importance-sampled environment (then the
// miss program is the spherical HDR map) in direction d, from one set of
// coordinates.
__device__ __forceinline__ void env_eval(const DevScene& S, V3 d, V3& Le, float& pdf) {
  float u, v;
  env_uv(d, u, v);
  pdf = env_pdf_uv(S, u, v);
  Le = 2.f * env_lookup(S.miss, u, v);
}

// Sum over the lights of their sampling pdf for direction d from P (per
// light selection), the MIS partner of BSDF sampling at emitter hits.
__device__ __forceinline__ float lights_pdf_c(const DevScene& S, V3 P, V3 d, int n_sel) {
  float acc = 0.f;
  for (int k = 0; k < S.num_lights; k++) acc += light_pdf(load_light(S.lights, k), P, d);
  return acc / (float)n_sel;
}

// ---------------------------------------------------- guide training data --
// A path whose id is a multiple of W.grec_stride records its first two
// guided vertices (shading point, sampled direction, BSDF pdf) in
// W.grec[2 * (id / stride) + v], with the throughput arriving at the vertex
// (luminance, kept in .weight) and the radiance collected so far (pad[0]).
// The record word in the path's radiance w is 2 * records + (1 if the
// current vertex recorded), so the NEE term of that vertex, known after its
// shadow ray, joins the mark.  At the end of the path each record's weight
// becomes (radiance after the vertex) / (throughput at it) = F / q of its
// direction, the training signal.
__device__ __forceinline__ float lum3(V3 c) {
  return 0.2126f * c.x + 0.7152f * c.y + 0.0722f * c.z;
}

__device__ __forceinline__ void guide_end(const WaveState& W, uint32_t pid, float code,
                                          V3 rad_end) {
  int count = (int)code >> 1;
  if (count <= 0) return;
  uint32_t base = 2u * (pid / W.grec_stride);
  float le = lum3(rad_end);
  for (int v = 0; v < count; v++) {
    GuideSample& r = W.grec[base + v];
    float T = r.weight, w = (le - r.pad[0]) / T;
    r.weight = (T > 0.f && w > 0.f && w < 1e30f) ? fminf(w, 1e6f) : 0.f;
    r.pad[1] = 2.f;  // complete
  }
}

// The occlusion ray of a path's NEE term has been traced: adds the term if
// nothing was hit.  A vertex that just recorded a guide sample: its NEE light
// did not come along the recorded direction.
__device__ __forceinline__ void nee_arrived(const WaveState& W, float occluded, float4 C,
                                            uint32_t pid, int word, V3& rad) {
  if (occluded != 0.f) return;
  rad += f4xyz(C);
  if (word & 1)
    W.grec[2u * (pid / W.grec_stride) + (uint32_t)((word & 6) >> 1) - 1u].pad[0] += lum3(f4xyz(C));
}

// ------------------------------------------------- consistent mode --------
// What a bounce of the consistent integrator leaves: its shadow ray (P, Wi,
// tmax) with the NEE term C that an unoccluded ray adds to the radiance, and
// the continuation (P, dcont), unless the path ended.
struct BounceC {
  V3 P, Wi, C, dcont;
  float tmax, code;  // code: the guide-record word
  bool ended, shadow;
};

// One bounce of the consistent integrator (the oracle's color_c): emission
// with MIS at hits and misses, NEE over lights + environment, BSDF
// continuation, Russian roulette.  The NEE term waits for its shadow ray while
// the path goes on.  With
// GUIDE the continuation is drawn from alpha * guide + (1 - alpha) * BSDF
// (the guide of this position from k_guide_infer) and that mixture density is
// the MIS partner of NEE and of emitter hits at the next vertex.  i: the path's
// position in its buffer (GUIDE).
template <bool GUIDE, bool TEX>
__device__ __forceinline__ void shade_step_c(const DevScene& S, const PathCtl& pc,
                                             const WaveState& W, uint32_t guide_depth, uint32_t i,
                                             float4 hit, V3 ro, V3 d, float tm, uint4& st, V3& thr,
                                             V3& rad, BounceC& b) {
  const int n_sel = S.num_lights + (S.env_valid ? 1 : 0);
  V3 P = v3(0.f), Wi = v3(0.f), dcont = v3(0.f), C = v3(0.f);
  float tmax = 0.f, code = b.code;
  bool ended = false, shadow = false;
  uint32_t depth = st.z & PT_ST_DEPTH_MASK;
  // a camera ray counts as a specular bounce: emission it sees is not MIS-weighted
  bool prev_spec = ((st.z >> PT_ST_SPEC_BIT) & 1u) || depth == 0;
  float pdf_prev = __uint_as_float(st.w);
  uint32_t leaf = __float_as_uint(hit.w);
  if (leaf == PT_NO_HIT) {
    V3 Le;
    float w = 1.f;
    if (!prev_spec && S.env_valid) {
      float pe;
      env_eval(S, d, Le, pe);
      w = power_mis(pdf_prev, pe / (float)n_sel);
    } else {
      Le = miss_color(S.miss, d);
    }
    rad += thr * Le * w;
    ended = true;
  } else {
    PrimRec p = load_prim(S.prims, leaf);
    HitRecord rec = hit_record(S, p, ro, d, hit.x, hit.y, hit.z, false, tm);
    GpuMaterial m = load_material(S.mats, rec.index);
    if (TEX && (m.tex0 >= 0 || m.tex1 >= 0))
      apply_textures(S, m, p, ro, d, hit.x, hit.y, hit.z, tm);
    P = rec.P;
    V3 Wo = rec.Wo, N = rec.shading_normal;
    if (m.type == PT_MAT_DIFFUSE_LIGHT) {
      float w = 1.f;
      if (!prev_spec && n_sel > 0) w = power_mis(pdf_prev, lights_pdf_c(S, ro, d, n_sel));
      rad += thr * v3(m.c0x, m.c0y, m.c0z) * w;
      ended = true;
    } else if (m.type == PT_MAT_METAL) {  // programs/materials/metal.cu:38-56
      V3 reflected = reflect(-Wo, N);
      dcont = reflected + m.p0 * random_in_unit_sphere(st.x);
      thr *= v3(m.c0x, m.c0y, m.c0z);
      prev_spec = true;
    } else if (m.type == PT_MAT_DIELECTRIC) {  // programs/materials/dielectric.cu:46-96
      float ref_idx = m.p0;
      V3 Wd = -rec.Wo, Nd = N;
      float ni_over_nt;
      float cosine = dot(Wd, Nd);
      if (cosine > 0.f) {
        Nd = -Nd;
        ni_over_nt = ref_idx;
        cosine = ref_idx * cosine / length(Wd);
      } else {
        ni_over_nt = 1.f / ref_idx;
        cosine = -cosine / length(Wd);
      }
      V3 refracted = v3(0.f);
      float reflect_prob;
      if (Refract(Wd, Nd, ni_over_nt, refracted)) reflect_prob = schlick(cosine, ref_idx);
      else reflect_prob = 1.f;
      if (rnd(st.x) < reflect_prob) dcont = reflect(Wd, Nd);
      else dcont = normalize(refracted);
      thr *= (v3(m.c0x, m.c0y, m.c0z) * v3(1.f));
      prev_spec = true;
    } else {
      Frame fr(N);
      V3 wo_l = fr.to_local(Wo);
      // bounces past the guided depth use the BSDF alone (alpha = 0)
      const bool guided = GUIDE && depth < guide_depth;
      const GuidePacked* G = GUIDE ? W.guide + i : nullptr;
      const float G_alpha = guided ? __ldg(&G->alpha) : 0.f;
      if (n_sel > 0) {
        int k = (int)(rnd(st.x) * (float)n_sel);
        if (k > n_sel - 1) k = n_sel - 1;
        float pl = 0.f;
        V3 Le;
        tmax = PT_RAY_TMAX;
        if (k < S.num_lights) {
          GpuLight L = load_light(S.lights, k);
          if (L.type == PT_LIGHT_RECT) {
            Wi = light_sample(L, P, st.x);
            tmax = 1.f - 1e-4f;
          } else {
            Wi = sphere_light_sample_c(L, P, st.x);
            V3 lc = v3(L.cx, L.cy, L.cz);
            float a = dot(Wi, Wi), b = dot(P - lc, Wi);
            float cc = dot(P - lc, P - lc) - L.r * L.r;
            float disc = b * b - a * cc;
            float tn = disc >= 0.f ? (-b - ptm_sqrt(disc)) / a : 0.f;
            tmax = tn * (1.f - 1e-4f);
          }
          pl = light_pdf(L, P, Wi);
          Le = v3(L.ex, L.ey, L.ez);
        } else {
          float u1 = rnd(st.x);
          float u2 = rnd(st.x);
          Wi = env_sample_dir(S, u1, u2);
          env_eval(S, Wi, Le, pl);
        }
        V3 wi_n = normalize(Wi);
        float cs = dot(wi_n, N);
        float pls = pl / (float)n_sel;
        if (cs > 0.f && pls > 0.f && tmax > 1e-3f) {
          V3 wi_l = fr.to_local(wi_n);
          V3 f;
          float pbs;
          bsdf_eval_c(m, wo_l, wi_l, f, pbs);
          if (guided)
            pbs = G_alpha * guide_pdf_packed(G, wi_n.x, wi_n.y, wi_n.z) + (1.f - G_alpha) * pbs;
          V3 cv = f * Le * (cs * power_mis(pls, pbs) / pls);
          if (!isNull(cv)) {
            shadow = true;
            C = thr * cv;
          }
        }
      }
      V3 wi_l, wdir;
      if (guided && rnd(st.x) < G_alpha) {
        float u0 = rnd(st.x);
        float u1 = rnd(st.x);
        float u2 = rnd(st.x);
        guide_sample_packed(G, u0, u1, u2, wdir.x, wdir.y, wdir.z);
        wi_l = fr.to_local(wdir);
      } else {
        wi_l = bsdf_sample_c(m, wo_l, st.x);
        wdir = fr.to_world(wi_l);
      }
      V3 f;
      float pbs;
      bsdf_eval_c(m, wo_l, wi_l, f, pbs);
      float q = pbs;
      if (guided) q = G_alpha * guide_pdf_packed(G, wdir.x, wdir.y, wdir.z) + (1.f - G_alpha) * pbs;
      if (!(q > 0.f) || isNull(f) || !(wi_l.y > 0.f)) {
        ended = true;
      } else {
        if (guided) {
          int count = (int)code >> 1;
          code = (float)(2 * count);
          if (count < 2 && st.y % W.grec_stride == 0) {
            uint32_t slot = 2u * (st.y / W.grec_stride) + (uint32_t)count;
            if (slot < W.grec_n) {
              GuideSample r;
              r.P[0] = P.x; r.P[1] = P.y; r.P[2] = P.z;
              r.N[0] = N.x; r.N[1] = N.y; r.N[2] = N.z;
              r.Wo[0] = Wo.x; r.Wo[1] = Wo.y; r.Wo[2] = Wo.z;
              r.wi[0] = wdir.x; r.wi[1] = wdir.y; r.wi[2] = wdir.z;
              r.p_bsdf = pbs;
              r.weight = lum3(thr);
              r.pad[0] = lum3(rad);
              r.pad[1] = 1.f;
              W.grec[slot] = r;
              code = (float)(2 * (count + 1) + 1);
            }
          }
        }
        thr *= f * (wi_l.y / q);
        prev_spec = false;
        pdf_prev = q;
        dcont = wdir;
      }
    }
    if (!ended) {
      if (pc.rr_enable && (int)depth > pc.rr_depth) {
        float q = fminf(1.f, max_component(thr));
        if (rnd(st.x) >= q) ended = true;
        else thr *= 1.f / q;
      }
      if (!ended) {
        depth++;
        if ((int)depth >= pc.max_depth) ended = true;
      }
    }
    st.z = (st.z & PT_ST_KEEP_MASK) | depth | ((uint32_t)prev_spec << PT_ST_SPEC_BIT);
    st.w = __float_as_uint(pdf_prev);
  }
  b.P = P;
  b.Wi = Wi;
  b.C = C;
  b.dcont = dcont;
  b.tmax = tmax;
  b.code = code;
  b.ended = ended;
  b.shadow = shadow;
}

}  // namespace ptd
