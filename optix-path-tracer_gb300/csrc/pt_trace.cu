/*
 * pt_trace.cu - BVH8 traversal kernels for sm_103a: the closest hit of
 * extension rays (replaces rtTrace into the scene's top object), the shadow
 * ray of Direct_Light (programs/hit.cu:16-24 under the closest-hit rule), the
 * occlusion rays of the consistent mode (in one launch with the extension
 * rays) and first-hit queries.
 *
 * The BVH8 (csrc/bvh_gpu.cu, csrc/bvh_host.cpp) stores 80-byte nodes with
 * 8-bit quantised child boxes and 48-byte primitive records; rays come from
 * the wavefront's path and shadow arrays (pt_kernels.cu), results go back to
 * them.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include "pt_bvh.cuh"
#include "pt_internal.h"
#include "pt_wave.cuh"

using namespace ptd;

// ------------------------------------------------------------ BVH8 trace --
// Closest hit through the BVH8 with warp-collective leaf tests.
//
// Each lane traverses its own ray node by node: into the nearest hit
// internal child, with one stack entry per level for the group of the
// node's other hit internal children (the second nearest taken first, the
// rest in slot order: a node step hits at most two internal children in
// nearly every case, so two running minima replace a full sort).  Primitive
// tests are not run by the lane that reaches a leaf: after every node step
// the warp gathers all (ray, primitive) pairs its lanes produced into shared
// memory and the 32 lanes test them together, merging the results per ray
// with a 64-bit atomicMin on (t, primitive id) - the order-independent
// closest-hit rule of the oracle.  Per-lane leaf loops of 1..24 triangles
// would otherwise serialise the warp.  Lanes whose rays are done wait until
// enough of the warp is idle, then write their results and take new rays
// together (persistent threads), and a stack group whose nearest child lies
// beyond the closest hit is dropped without visiting it.
//
// One node step yields at most PT_MAX_PAIRS pairs per warp (the builders
// bound the primitives under one node's leaf children by 24); they are
// tested in rounds of PT_PAIR_CAP, so the pair buffer stays small and more
// blocks fit on an SM.
#define PT_MAX_PAIRS (32 * 24)
#ifndef PT_PAIR_CAP
#define PT_PAIR_CAP (32 * 8)
#endif

struct WarpShared {
  float4 ro[32];                  // origin, tmin
  float4 rd[32];                  // direction, tmax
  float4 wt[32];                  // watertight-test constants Sx, Sy, Sz, axes
  unsigned long long best[32];    // (t bits << 32) | primitive id
  float tm[32];                   // the ray's path time (scenes with moving spheres)
  uint32_t pair_prim[PT_PAIR_CAP];
  uint8_t pair_owner[PT_PAIR_CAP];
};

struct FirstHitOut {
  uint32_t* prim;
  uint32_t* mat;
  float* t;
  int width, height, frame;
  uint32_t* err;
};

#define PT_ONE_BLOCK 128  // k_trace_one: threads per block
#ifndef PT_ONE_MINBLOCKS
#define PT_ONE_MINBLOCKS 8
#endif

#ifndef PT_ANYHIT_NEAREST
#define PT_ANYHIT_NEAREST 1  // occlusion rays enter the nearest child first
#endif

// BATCH: rays of several scenes; each starts at its scene's root node (the
// scene index is in the path state word st.z).  list: extension rays are put on
// the shading lists.  MOTION: the scene has moving
// spheres, so each ray carries its path's time (other scenes do without).
template <int MODE, bool COUNT, bool BATCH, bool MOTION>
__device__ __forceinline__ void trace_rays(const DevScene& S, const WaveState& W,
                                           const WaveCtl* __restrict__ ctlp, int max_stack,
                                           const FirstHitOut& fo, const BatchRefs& br,
                                           int refetch, int list) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  WarpShared& ws = ((WarpShared*)smem)[threadIdx.x >> 5];
  unsigned char* stk_base = smem + (blockDim.x >> 5) * sizeof(WarpShared);
  uint2* stk = (uint2*)stk_base + threadIdx.x;
  float* stkt = (float*)((uint2*)stk_base + (size_t)max_stack * blockDim.x) + threadIdx.x;
  const int bd = blockDim.x;

  uint32_t n;
  WaveCounters c;
  if (MODE != TRACE_FIRST) c = *W.ctr;
  constexpr bool consistent = MODE == TRACE_OCCLUDED;
  constexpr bool SHADOWRAY = MODE == TRACE_SHADOW || MODE == TRACE_OCCLUDED;
  if (MODE == TRACE_EXT) {
    n = c.n_cur + gen_count(c, *ctlp, (uint32_t)W.slots);
  } else if (MODE == TRACE_OCCLUDED) {
    n = c.n_occ;
  } else if (MODE == TRACE_SHADOW) {
    n = c.n_shadow;
  } else {
    n = (uint32_t)fo.width * (uint32_t)fo.height;
  }
  // rays are handed out to warps in arrival order from a per-launch counter
  // (first-hit queries: a fixed grid-stride assignment)
  const uint32_t stride = gridDim.x * blockDim.x;
  uint32_t* take = MODE == TRACE_EXT ? &W.ctr->ray_next[0] : (SHADOWRAY ? &W.ctr->ray_next[1] : nullptr);
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  bool started = false;
  uint32_t nn = 0, np = 0;

  // per-lane ray state (the direction and tmax of a lane's ray live in the
  // warp's shared copy, ws.rd[lane]: the node tests need only o, tmin and
  // the reciprocal direction)
  const uint32_t parity = MODE == TRACE_EXT || MODE == TRACE_OCCLUDED ? c.parity : 0u;
  BoxRay ray;
  V3& o = ray.o;
  float& tmin = ray.tmin;
  o = v3(0.f);
  tmin = ray.ix = ray.iy = ray.iz = 0.f;
  ray.negx = ray.negy = ray.negz = false;
  float tbest = 0.f;
  uint32_t cur = 0, best_id = PT_NO_HIT;
  int sp = 0;
  bool active = false;

  // loads ray i into o, d, tmin, tmax
  auto load_ray = [&](V3& d, float& tmax) {
    if (MODE == TRACE_EXT) {
      float4 ro = W.path[parity].ray_o[i], rdv = W.path[parity].ray_d[i];
      o = f4xyz(ro);
      d = f4xyz(rdv);
      tmin = ro.w;
      tmax = rdv.w;
    } else if (MODE == TRACE_OCCLUDED) {
      // from the point where its path goes on (i: the path's position)
      o = f4xyz(W.path[parity].ray_o[i]);
      d = f4xyz(W.nee[parity].Wi[i]);
      tmin = 1e-3f;
      tmax = W.nee[parity].C[i].w;
    } else if (MODE == TRACE_SHADOW) {
      o = f4xyz(W.sh.P[i]);
      d = f4xyz(W.sh.Wi[i]);
      tmin = 1e-3f;
      tmax = PT_RAY_TMAX;
    } else {
      uint32_t x = i % (uint32_t)fo.width, y = i / (uint32_t)fo.width;
      uint32_t seed = tea64((uint32_t)fo.width * y + x, (uint32_t)fo.frame);
      Ray3 r = camera_ray(S.cam, x, y, fo.width, fo.height, seed);
      o = v3(r.o.x, r.o.y, r.o.z);
      d = v3(r.d.x, r.d.y, r.d.z);
      tmin = 1e-6f;
      tmax = PT_RAY_TMAX;
      if (MOTION)  // color()'s prd.time, programs/raygen.cu:69
        ws.tm[lane] = S.cam.time0 + rnd(seed) * (S.cam.time1 - S.cam.time0);
    }
  };

  // puts position i on the shading list of its key (the lanes that finish
  // together share an atomic per key)
  auto list_hit = [&](uint32_t key) {
    const uint32_t act = __activemask();
    const uint32_t same = __match_any_sync(act, key);
    const int leader = __ffs(same) - 1;
    uint32_t at = 0;
    if (lane == leader) at = atomicAdd(&W.listed[key * PT_LISTED_STRIDE], (uint32_t)__popc(same));
    at = __shfl_sync(same, at, leader) + (uint32_t)__popc(same & ((1u << lane) - 1u));
    W.lists[(size_t)key * (size_t)W.slots + at] = i;
  };

  auto finish = [&](V3 d, float tmax) {
    if (MODE == TRACE_EXT) {
      uint32_t key = 0;
      float4 h = make_float4(tmax, 0.f, 0.f, __uint_as_float(PT_NO_HIT));
      if (best_id != PT_NO_HIT) {
        uint32_t leaf = __ldg(S.leaf_of_id + best_id);
        PrimRec p = load_prim(S.prims, leaf);
        float t = tbest, bu = 0.f, bv = 0.f;
        if (prim_type(p) == PT_PRIM_TRIANGLE) tri_candidate(p, o, wt_setup(d), tmin, tmax, t, bu, bv);
        h = make_float4(tbest, bu, bv, __uint_as_float(leaf));
        if (list) key = 1u + (uint32_t)__ldg(&S.mats[prim_material(p)].type);
      }
      W.hit[i] = h;
      if (list) list_hit(key);
    } else if (MODE == TRACE_OCCLUDED) {
      // anything before the light
      W.nee[parity].Wi[i].w = best_id != PT_NO_HIT ? 1.f : 0.f;
    } else if (MODE == TRACE_SHADOW) {
      bool occluded = true;
      if (best_id != PT_NO_HIT) {
        PrimRec p = load_prim(S.prims, __ldg(S.leaf_of_id + best_id));
        bool is_light = S.mats[prim_material(p)].type == PT_MAT_DIFFUSE_LIGHT;
        occluded = !(is_light && dot(f4xyz(W.sh.N[i]), d) > 0.f);
      }
      W.sh.Wi[i].w = occluded ? 1.f : 0.f;
    } else {
      if (best_id == PT_NO_HIT) {
        fo.prim[i] = PT_NO_HIT;
        fo.mat[i] = PT_NO_HIT;
        fo.t[i] = 0.f;
      } else {
        PrimRec p = load_prim(S.prims, __ldg(S.leaf_of_id + best_id));
        fo.prim[i] = best_id;
        fo.mat[i] = prim_material(p);
        fo.t[i] = tbest;
      }
    }
  };

  auto finish_traced = [&]() {
    float4 rdv = ws.rd[lane];
    finish(f4xyz(rdv), rdv.w);
  };

  bool idle = true;   // wants a ray (finished one, or none taken yet)
  bool done = false;  // traced a ray whose result is not written yet
  // a traversal ends: the result is written with the warp's next batch of
  // fetches, when most lanes do the same work together
  auto end_ray = [&]() {
    active = false;
    idle = true;
    done = true;
  };
  // loads ray i (< n) and sets up its traversal
  auto fetch = [&]() {
    // Some rays end here, without a traversal: one with a NaN in its origin or
    // direction (every primitive test fails or yields a NaN distance, which never
    // wins the closest-hit minimum, but it would pass every box test), any ray of
    // an empty scene, and an extension ray whose path has ended (tmax 0: the path
    // only waits for its NEE term).
    V3 d;
    float tmax;
    load_ray(d, tmax);
    if (nan_ray(o, d) || S.num_prims == 0 || (MODE == TRACE_EXT && tmax == 0.f)) {
      best_id = PT_NO_HIT;
      tbest = tmax;
      finish(d, tmax);
      active = false;
      idle = true;
      return;
    }
    active = true;
    ray.set_direction(d);
    WtRay w = wt_setup(d);
    ws.ro[lane] = make_float4(o.x, o.y, o.z, tmin);
    ws.rd[lane] = make_float4(d.x, d.y, d.z, tmax);
    ws.wt[lane] = make_float4(w.Sx, w.Sy, w.Sz,
                              __uint_as_float((uint32_t)w.kx | ((uint32_t)w.ky << 2) |
                                              ((uint32_t)w.kz << 4)));
    tbest = tmax;
    best_id = PT_NO_HIT;
    ws.best[lane] = ((unsigned long long)__float_as_uint(tmax) << 32) | 0xffffffffull;
    if (MOTION && MODE != TRACE_FIRST)  // the path's time rides in throughput.w
      ws.tm[lane] = MODE == TRACE_SHADOW ? W.sh.thr[i].w : W.path[parity].thr[i].w;
    cur = S.root;
    if (BATCH) {
      uint32_t z = MODE == TRACE_SHADOW ? W.sh.st[i].z : W.path[parity].st[i].z;
      cur = __ldg(br.roots + (z >> PT_ST_SCENE_SHIFT));
    }
    sp = 0;
  };

  while (true) {
    // idle lanes take and load their next rays together once `refetch`
    // lanes wait (or nothing else runs), so the warp pays one load latency
    // per batch; a lane whose index is past the end has no more work (the
    // counter only grows)
    uint32_t busy = __ballot_sync(0xffffffffu, active);
    uint32_t waiting = __ballot_sync(0xffffffffu, idle);
    if (waiting && (__popc(waiting) >= refetch || busy == 0)) {
      if (done) {
        finish_traced();
        done = false;
      }
      if (MODE == TRACE_FIRST) {
        if (idle) {
          if (started) i += stride;
          started = true;
        }
      } else {
        const int leader = __ffs(waiting) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(take, (uint32_t)__popc(waiting));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (idle) i = base + (uint32_t)__popc(waiting & ((1u << lane) - 1u));
      }
      if (idle) {
        idle = false;
        if (i < n) {
          if (MODE == TRACE_OCCLUDED) i = W.nee[parity].queue[i];
          fetch();
        }
      }
      busy = __ballot_sync(0xffffffffu, active);
      if (!busy) {
        if (__ballot_sync(0xffffffffu, idle)) continue;  // only rays that ended at load
        break;
      }
    }
    if (!busy) break;
    // ---- node step: the eight child boxes of each active lane's node
    NodeHits hits;
    hits.ihit = hits.leafmask = hits.pbase = hits.mlo = hits.mhi = hits.child_base = 0;
    hits.k1 = hits.k2 = 0xffffffffu;
    if (active) {
      if (COUNT) nn++;
      node_step(S.nodes + 5 * (size_t)cur, ray, tbest * 1.0000005f, hits);
    }
    // ---- next node, chosen before the primitive tests: the nearest hit
    // internal child, the others pushed as one group (closest hit: in
    // near-to-far order with the distance of the nearest; occlusion: as a
    // mask).  With no internal child hit, a closest-hit ray pops after the
    // tests, which may shorten it and so drop groups beyond the new hit.
    const uint32_t ihit = hits.ihit, child_base = hits.child_base, pbase = hits.pbase;
    const uint32_t k1 = hits.k1, k2 = hits.k2;
    const int nint = __popc(ihit);
    bool pop = false;
    float tnext = 0.f;
    if (active) {
      if (consistent) {
        if (ihit) {
          uint32_t b = (uint32_t)(__ffs(ihit) - 1);
          if (PT_ANYHIT_NEAREST) b = k1 & 7u;
          cur = child_base + b;
          const uint32_t rest = ihit & ~(1u << b);
          if (rest) {
            if (sp >= max_stack) {
              atomicOr(&W.ctr->error, 1u);
              sp = 0;  // abandon this ray (the host reports the error)
              end_ray();
            } else {
              stk[sp * bd] = make_uint2(child_base, rest);
              sp++;
            }
          }
        } else if (sp > 0) {
          uint2 e = stk[(sp - 1) * bd];
          cur = e.x + (uint32_t)(__ffs(e.y) - 1);
          e.y &= e.y - 1;
          if (e.y == 0) sp--;
          else stk[(sp - 1) * bd].y = e.y;
        } else {
          end_ray();
        }
      } else if (nint >= 1) {
        cur = child_base + (k1 & 7u);
        tnext = __uint_as_float(k1 & 0xfffffff8u);
        if (nint > 1) {
          // pending group: the other hit children as a slot mask, the second
          // nearest marked to be taken first (the rest in slot order), and
          // the entry distance of the second nearest, below every one of them
          if (sp >= max_stack) {
            atomicOr(MODE == TRACE_FIRST ? fo.err : &W.ctr->error, 1u);
            sp = 0;  // abandon this ray (the host reports the error)
            end_ray();
          } else {
            stk[sp * bd] = make_uint2(child_base, (ihit & ~(1u << (k1 & 7u))) | ((k2 & 7u) << 8) | 0x800u);
            stkt[sp * bd] = __uint_as_float(k2 & 0xfffffff8u);
            sp++;
          }
        }
      } else {
        pop = true;
      }
    }
    // ---- warp-collective primitive tests of the hit leaves (also of a lane
    // whose ray ended above: its leaves of this node still count).  pm: the
    // lane's primitives as bits over the node's range, bit j = record
    // pbase + j (a node's leaves hold at most 24 primitives).
    const uint32_t pm = leaf_prims(hits);
    if (__any_sync(0xffffffffu, pm != 0)) {
      const uint32_t cnt = __popc(pm);
      const uint32_t total = __reduce_add_sync(0xffffffffu, cnt);
      const uint32_t mx = __reduce_max_sync(0xffffffffu, cnt);
      if (mx * 32u <= 2u * total) {
        // balanced: each lane tests its own primitives (at least half the
        // lane-slots do work)
        if (pm) {
          WtRay wt = wt_unpack(ws.wt[lane]);
          unsigned long long bk = ws.best[lane];
          const float4 rdv = ws.rd[lane];
          uint32_t m = pm;
          while (m) {
            const int j = __ffs(m) - 1;
            m &= m - 1;
            PrimRec p = load_prim(S.prims, pbase + (uint32_t)j);
            if (COUNT) np++;
            float t, bu, bv;
            if (prim_test<MOTION>(S, p, o, f4xyz(rdv), wt, tmin, rdv.w, t, bu, bv,
                                  MOTION ? ws.tm[lane] : 0.f)) {
              unsigned long long key = ((unsigned long long)__float_as_uint(t) << 32) | prim_id(p);
              bk = min(bk, key);
            }
          }
          ws.best[lane] = bk;
          tbest = __uint_as_float((uint32_t)(bk >> 32));
          best_id = (uint32_t)bk;
        }
      } else {
        // unbalanced: spread the (ray, primitive) pairs over the warp
        uint32_t incl = cnt;
#pragma unroll
        for (int dd = 1; dd < 32; dd <<= 1) {
          uint32_t t = __shfl_up_sync(0xffffffffu, incl, dd);
          if (lane >= dd) incl += t;
        }
        const uint32_t off0 = incl - cnt;
        for (uint32_t r0 = 0; r0 < total; r0 += PT_PAIR_CAP) {
          // this round's pairs: [r0, r0 + PT_PAIR_CAP) of the warp's list
          if (pm && off0 < r0 + PT_PAIR_CAP && off0 + cnt > r0) {
            uint32_t off = off0 - r0;  // wraps below the round: skipped
            uint32_t m = pm;
            while (m) {
              const int j = __ffs(m) - 1;
              m &= m - 1;
              if (off < PT_PAIR_CAP) {
                ws.pair_prim[off] = pbase + (uint32_t)j;
                ws.pair_owner[off] = (uint8_t)lane;
              }
              off++;
            }
          }
          __syncwarp();
          const uint32_t nr = min(total - r0, (uint32_t)PT_PAIR_CAP);
          for (uint32_t j = lane; j < nr; j += 32) {
            uint32_t pi = ws.pair_prim[j];
            uint32_t ow = ws.pair_owner[j];
            PrimRec p = load_prim(S.prims, pi);
            if (COUNT) np++;
            float4 ro = ws.ro[ow], rdv = ws.rd[ow];
            float t, bu, bv;
            if (prim_test<MOTION>(S, p, f4xyz(ro), f4xyz(rdv), wt_unpack(ws.wt[ow]), ro.w, rdv.w, t,
                                  bu, bv, MOTION ? ws.tm[ow] : 0.f)) {
              unsigned long long key = ((unsigned long long)__float_as_uint(t) << 32) | prim_id(p);
              atomicMin(&ws.best[ow], key);
            }
          }
          __syncwarp();
        }
        if (pm) {
          unsigned long long k = ws.best[lane];
          tbest = __uint_as_float((uint32_t)(k >> 32));
          best_id = (uint32_t)k;
        }
      }
    }
    // ---- occlusion rays end at the first confirmed hit before tmax
    if (consistent && active && best_id != PT_NO_HIT) end_ray();
    // ---- closest hit: a chosen child that now lies beyond the hit is
    // dropped; then the deepest pending group not beyond the hit
    if (!consistent && active) {
      const float tlim = tbest * 1.0000005f;
      if (!pop && tnext > tlim) pop = true;
      if (pop) {
        bool found = false;
        while (sp > 0) {
          uint2 e = stk[(sp - 1) * bd];
          if (stkt[(sp - 1) * bd] > tlim) {  // every child of the group starts beyond the hit
            sp--;
            continue;
          }
          uint32_t m = e.y & 0xffu;
          const uint32_t slot = (e.y & 0x800u) ? (e.y >> 8) & 7u : (uint32_t)(__ffs(m) - 1);
          m &= ~(1u << slot);
          cur = e.x + slot;
          if (m == 0) sp--;
          else stk[(sp - 1) * bd].y = m;
          found = true;
          break;
        }
        if (!found) end_ray();
      }
    }
  }
  if (COUNT) {
    atomicAdd(&W.ctr->node_fetches, (unsigned long long)nn);
    atomicAdd(&W.ctr->prim_tests, (unsigned long long)np);
  }
}

template <int MODE, bool COUNT, bool BATCH, bool MOTION>
__global__ void __maxnreg__(PT_TRACE_MAXREG)
    k_trace_t(DevScene S, WaveState W, const WaveCtl* __restrict__ ctlp, int max_stack,
              FirstHitOut fo, BatchRefs br, int refetch, int list) {
  if (MODE == TRACE_BOTH) {
    // a warp that finds no extension ray left goes on to the occlusion rays, so
    // the one kind fills the SMs while the longest rays of the other end.  Two
    // launches, with a finishing kernel behind the second, took 1052 us per
    // 1280x720 terrain frame and 80.0 ms per 64 frames at 1920x1080; this one,
    // with the path state passed on once instead of parked, 973 us and 76.9 ms
    // (GB300)
    trace_rays<TRACE_EXT, COUNT, BATCH, MOTION>(S, W, ctlp, max_stack, fo, br, refetch, list);
    __syncwarp();
    trace_rays<TRACE_OCCLUDED, COUNT, BATCH, MOTION>(S, W, ctlp, max_stack, fo, br, refetch, list);
  } else {
    trace_rays<MODE, COUNT, BATCH, MOTION>(S, W, ctlp, max_stack, fo, br, refetch, list);
  }
}
// ---------------------------------------------------- trees of one node ----
// Rays of a scene whose tree is a single node (up to 24 primitives: the
// reference's Cornell box and the like).  There is no traversal, so a warp
// takes 32 rays in order and all its lanes test the same primitive at a time
// (those that some lane's boxes let through): one type, one axis, broadcast
// record loads, no pair lists, no refetch.  Bound by instruction issue.  GB300,
// Cornell box 512x512, 64 frames: extension rays 4.1 -> 3.1 ms, shadow rays
// 3.3 -> 2.5 ms against the general kernel.
template <int MODE, bool MOTION>
__device__ __forceinline__ void trace_rays_one(const DevScene& S, const WaveState& W,
                                               const WaveCtl* __restrict__ ctlp,
                                               const FirstHitOut& fo, int list, int count) {
  const int lane = threadIdx.x & 31;
  uint32_t n, parity = 0;
  if (MODE == TRACE_FIRST) {
    n = (uint32_t)fo.width * (uint32_t)fo.height;
  } else {
    const WaveCounters c = *W.ctr;
    parity = c.parity;
    n = MODE == TRACE_EXT ? c.n_cur + gen_count(c, *ctlp, (uint32_t)W.slots)
                          : (MODE == TRACE_OCCLUDED ? c.n_occ : c.n_shadow);
  }
  uint32_t nn = 0, np = 0;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; base < n; base += stride) {
    uint32_t i = base + (uint32_t)lane;
    bool live = i < n;
    V3 o = v3(0.f), d = v3(0.f);
    float tmin = 1e-3f, tmax = PT_RAY_TMAX, tm = 0.f;
    if (live) {
      if (MODE == TRACE_EXT) {
        const float4 o4 = W.path[parity].ray_o[i], d4 = W.path[parity].ray_d[i];
        o = f4xyz(o4);
        d = f4xyz(d4);
        tmin = o4.w;
        tmax = d4.w;
        if (MOTION) tm = W.path[parity].thr[i].w;
      } else if (MODE == TRACE_OCCLUDED) {
        i = W.nee[parity].queue[i];
        o = f4xyz(W.path[parity].ray_o[i]);
        d = f4xyz(W.nee[parity].Wi[i]);
        tmax = W.nee[parity].C[i].w;
        if (MOTION) tm = W.path[parity].thr[i].w;
      } else if (MODE == TRACE_SHADOW) {
        o = f4xyz(W.sh.P[i]);
        d = f4xyz(W.sh.Wi[i]);
        if (MOTION) tm = W.sh.thr[i].w;
      } else {
        const uint32_t x = i % (uint32_t)fo.width, y = i / (uint32_t)fo.width;
        uint32_t seed = tea64((uint32_t)fo.width * y + x, (uint32_t)fo.frame);
        const Ray3 r = camera_ray(S.cam, x, y, fo.width, fo.height, seed);
        o = v3(r.o.x, r.o.y, r.o.z);
        d = v3(r.d.x, r.d.y, r.d.z);
        tmin = 1e-6f;
        if (MOTION)  // color()'s prd.time, programs/raygen.cu:69
          tm = S.cam.time0 + rnd(seed) * (S.cam.time1 - S.cam.time0);
      }
    }
    // rays that hit nothing by definition, as in trace_rays
    const bool trace = live && !nan_ray(o, d) && S.num_prims != 0 && !(MODE == TRACE_EXT && tmax == 0.f);
    NodeHits h;
    h.ihit = h.leafmask = h.mlo = h.mhi = 0;
    h.k1 = h.k2 = 0xffffffffu;
    if (trace) {
      BoxRay ray;
      ray.o = o;
      ray.tmin = tmin;
      ray.set_direction(d);
      node_step(S.nodes, ray, tmax * 1.0000005f, h);
      nn++;
    }
    const uint32_t pm = leaf_prims(h);
    np += (uint32_t)__popc(pm);
    const uint32_t pbase = __ldg(&S.nodes[1].y);
    unsigned long long best = ((unsigned long long)__float_as_uint(tmax) << 32) | PT_NO_HIT;
    uint32_t leaf = PT_NO_HIT, mat = 0;
    float hu = 0.f, hv = 0.f;
    bool have_wt = false;
    WtRay wt;
    for (uint32_t all = __reduce_or_sync(0xffffffffu, pm); all; all &= all - 1) {
      const int j = __ffs(all) - 1;
      const PrimRec p = load_prim(S.prims, pbase + (uint32_t)j);  // the same for all lanes
      if (prim_type(p) == PT_PRIM_TRIANGLE && !have_wt) {
        wt = wt_setup(d);
        have_wt = true;
      }
      if ((pm >> j) & 1u) {
        float t, bu, bv;
        if (prim_test<MOTION>(S, p, o, d, wt, tmin, tmax, t, bu, bv, tm)) {
          const unsigned long long key = ((unsigned long long)__float_as_uint(t) << 32) | prim_id(p);
          if (key < best) {
            best = key;
            leaf = pbase + (uint32_t)j;
            mat = prim_material(p);
            hu = bu;
            hv = bv;
          }
        }
      }
    }
    const float thit = __uint_as_float((uint32_t)(best >> 32));
    if (MODE == TRACE_EXT) {
      if (live) W.hit[i] = make_float4(thit, hu, hv, __uint_as_float(leaf));
      if (list) {
        const uint32_t key = !live ? 0xffu : (leaf == PT_NO_HIT ? 0u : 1u + (uint32_t)__ldg(&S.mats[mat].type));
        const uint32_t same = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(same) - 1;
        uint32_t at = 0;
        if (live && lane == leader) at = atomicAdd(&W.listed[key * PT_LISTED_STRIDE], (uint32_t)__popc(same));
        at = __shfl_sync(0xffffffffu, at, leader) + (uint32_t)__popc(same & ((1u << lane) - 1u));
        if (live) W.lists[(size_t)key * (size_t)W.slots + at] = i;
      }
    } else if (MODE == TRACE_OCCLUDED) {
      if (live) W.nee[parity].Wi[i].w = leaf != PT_NO_HIT ? 1.f : 0.f;
    } else if (MODE == TRACE_SHADOW) {
      if (live) {
        const bool light = leaf != PT_NO_HIT && S.mats[mat].type == PT_MAT_DIFFUSE_LIGHT &&
                           dot(f4xyz(W.sh.N[i]), d) > 0.f;
        W.sh.Wi[i].w = light ? 0.f : 1.f;
      }
    } else if (live) {
      fo.prim[i] = (uint32_t)best;
      fo.mat[i] = leaf == PT_NO_HIT ? PT_NO_HIT : mat;
      fo.t[i] = leaf == PT_NO_HIT ? 0.f : thit;
    }
  }
  if (count) {
    atomicAdd(&W.ctr->node_fetches, (unsigned long long)nn);
    atomicAdd(&W.ctr->prim_tests, (unsigned long long)np);
  }
}

template <int MODE, bool MOTION>
__global__ void __launch_bounds__(PT_ONE_BLOCK, PT_ONE_MINBLOCKS)
    k_trace_one(DevScene S, WaveState W, const WaveCtl* __restrict__ ctlp, FirstHitOut fo, int list,
                int count) {
  if (MODE == TRACE_BOTH) {
    trace_rays_one<TRACE_EXT, MOTION>(S, W, ctlp, fo, list, count);
    trace_rays_one<TRACE_OCCLUDED, MOTION>(S, W, ctlp, fo, list, count);
  } else {
    trace_rays_one<MODE, MOTION>(S, W, ctlp, fo, list, count);
  }
}


// ------------------------------------------------------- host launchers ---
namespace pt {

size_t trace_smem(int max_stack, int block) {
  return (size_t)(block / 32) * sizeof(WarpShared) +
         (size_t)block * max_stack * (sizeof(uint2) + sizeof(float));
}

int one_blocks_per_sm() {
  int blocks = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_trace_one<TRACE_EXT, false>,
                                                    PT_ONE_BLOCK, 0) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return blocks < 1 ? 1 : blocks;
}

int trace_blocks_per_sm(int block, size_t smem) {
  int blocks = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &blocks, k_trace_t<TRACE_EXT, false, false, false>, block, smem);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return blocks;
}

// Dynamic shared memory limit of kernel k: the per-block opt-in maximum
// minus its static shared memory.
template <typename K>
static cudaError_t smem_attr(K k, int optin) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, k);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              optin - (int)fa.sharedSizeBytes);
}

template <int MODE, bool MOTION>
static cudaError_t smem_attr_mode(int optin) {
  cudaError_t e;
  if ((e = smem_attr(k_trace_t<MODE, false, false, MOTION>, optin)) != cudaSuccess) return e;
  if ((e = smem_attr(k_trace_t<MODE, true, false, MOTION>, optin)) != cudaSuccess) return e;
  if ((e = smem_attr(k_trace_t<MODE, false, true, MOTION>, optin)) != cudaSuccess) return e;
  return smem_attr(k_trace_t<MODE, true, true, MOTION>, optin);
}

static const int kMaxDev = 64;
static bool g_smem_set[kMaxDev];

cudaError_t set_trace_smem() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < kMaxDev && g_smem_set[dev]) return cudaSuccess;
  int optin = 0;
  if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) !=
      cudaSuccess)
    return e;
  if ((e = smem_attr_mode<TRACE_EXT, false>(optin)) != cudaSuccess) return e;
  if ((e = smem_attr_mode<TRACE_SHADOW, false>(optin)) != cudaSuccess) return e;
  if ((e = smem_attr_mode<TRACE_BOTH, false>(optin)) != cudaSuccess) return e;
  if ((e = smem_attr_mode<TRACE_EXT, true>(optin)) != cudaSuccess) return e;
  if ((e = smem_attr_mode<TRACE_SHADOW, true>(optin)) != cudaSuccess) return e;
  if ((e = smem_attr_mode<TRACE_BOTH, true>(optin)) != cudaSuccess) return e;
  if ((e = smem_attr(k_trace_t<TRACE_FIRST, false, false, false>, optin)) != cudaSuccess) return e;
  if ((e = smem_attr(k_trace_t<TRACE_FIRST, false, false, true>, optin)) != cudaSuccess) return e;
  if (dev >= 0 && dev < kMaxDev) g_smem_set[dev] = true;
  return cudaSuccess;
}

template <int MODE, bool BATCH, bool MOTION>
static void launch_mode(bool counters, const DevScene& S, const WaveState& W, const WaveCtl* ctl,
                        int max_stack, const BatchRefs& br, const LaunchCfg& lc, size_t smem,
                        cudaStream_t st) {
  FirstHitOut none{};
  if (counters)
    k_trace_t<MODE, true, BATCH, MOTION><<<lc.trace_grid, lc.trace_block, smem, st>>>(
        S, W, ctl, max_stack, none, br, lc.refetch, lc.sort);
  else
    k_trace_t<MODE, false, BATCH, MOTION><<<lc.trace_grid, lc.trace_block, smem, st>>>(
        S, W, ctl, max_stack, none, br, lc.refetch, lc.sort);
}

template <bool BATCH, bool MOTION>
static void launch_kind(int mode, bool counters, const DevScene& S, const WaveState& W,
                        const WaveCtl* ctl, int max_stack, const BatchRefs& br,
                        const LaunchCfg& lc, size_t smem, cudaStream_t st) {
  if (mode == TRACE_EXT)
    launch_mode<TRACE_EXT, BATCH, MOTION>(counters, S, W, ctl, max_stack, br, lc, smem, st);
  else if (mode == TRACE_SHADOW)
    launch_mode<TRACE_SHADOW, BATCH, MOTION>(counters, S, W, ctl, max_stack, br, lc, smem, st);
  else
    launch_mode<TRACE_BOTH, BATCH, MOTION>(counters, S, W, ctl, max_stack, br, lc, smem, st);
}

template <bool MOTION>
static void launch_one(int mode, bool counters, const DevScene& S, const WaveState& W,
                       const WaveCtl* ctl, const LaunchCfg& lc, cudaStream_t st) {
  FirstHitOut none{};
  const int c = counters ? 1 : 0;
  if (mode == TRACE_EXT)
    k_trace_one<TRACE_EXT, MOTION><<<lc.one_grid, PT_ONE_BLOCK, 0, st>>>(S, W, ctl, none, lc.sort, c);
  else if (mode == TRACE_SHADOW)
    k_trace_one<TRACE_SHADOW, MOTION><<<lc.one_grid, PT_ONE_BLOCK, 0, st>>>(S, W, ctl, none, 0, c);
  else
    k_trace_one<TRACE_BOTH, MOTION><<<lc.one_grid, PT_ONE_BLOCK, 0, st>>>(S, W, ctl, none, lc.sort, c);
}

void launch_trace(int mode, bool counters, const DevScene& S, const WaveState& W,
                  const WaveCtl* ctl, int max_stack, const BatchRefs* br, const LaunchCfg& lc,
                  cudaStream_t st) {
  if (!br && lc.one_grid) {
    if (lc.motion)
      launch_one<true>(mode, counters, S, W, ctl, lc, st);
    else
      launch_one<false>(mode, counters, S, W, ctl, lc, st);
    return;
  }
  const size_t smem = trace_smem(max_stack, lc.trace_block);
  if (br && lc.motion)
    launch_kind<true, true>(mode, counters, S, W, ctl, max_stack, *br, lc, smem, st);
  else if (br)
    launch_kind<true, false>(mode, counters, S, W, ctl, max_stack, *br, lc, smem, st);
  else if (lc.motion)
    launch_kind<false, true>(mode, counters, S, W, ctl, max_stack, BatchRefs{}, lc, smem, st);
  else
    launch_kind<false, false>(mode, counters, S, W, ctl, max_stack, BatchRefs{}, lc, smem, st);
}

void launch_first_hits(const DevScene& S, int w, int h, int frame, uint32_t* prim, uint32_t* mat,
                       float* t, int max_stack, uint32_t* err, const LaunchCfg& lc,
                       cudaStream_t st) {
  FirstHitOut fo{prim, mat, t, w, h, frame, err};
  WaveState none{};
  const int grid = lc.trace_grid;
  if (lc.one_grid && S.has_motion)
    k_trace_one<TRACE_FIRST, true><<<lc.one_grid, PT_ONE_BLOCK, 0, st>>>(S, none, nullptr, fo, 0, 0);
  else if (lc.one_grid)
    k_trace_one<TRACE_FIRST, false><<<lc.one_grid, PT_ONE_BLOCK, 0, st>>>(S, none, nullptr, fo, 0, 0);
  else if (S.has_motion)
    k_trace_t<TRACE_FIRST, false, false, true>
        <<<grid, PT_TRACE_BLOCK, trace_smem(max_stack, PT_TRACE_BLOCK), st>>>(
            S, none, nullptr, max_stack, fo, BatchRefs{}, 32, 0);
  else
    k_trace_t<TRACE_FIRST, false, false, false>
        <<<grid, PT_TRACE_BLOCK, trace_smem(max_stack, PT_TRACE_BLOCK), st>>>(
            S, none, nullptr, max_stack, fo, BatchRefs{}, 32, 0);
}

}  // namespace pt
