/*
 * pt_tail.cu - the last paths of a chunk, each traced to its end by one
 * thread (one launch), in place of wavefront iterations over ever fewer
 * paths.
 *
 * A wavefront iteration costs four to six dependent launches whatever its
 * size, and Russian roulette and glass leave a long, thin tail: a few hundred
 * paths live for dozens of bounces more.  Once the paths left (live ones and
 * ones not generated yet) are at most WaveCtl.tail_max, this kernel takes
 * them all.  It is bound by the latency of one path's bounces, so the paths
 * are spread over all warps that fit on the GPU, as few lanes of each as
 * that takes: a lone path waits for no other path's traversal or BRDF.
 * The bounce arithmetic is the wavefront's (pt_shade.cuh), and a traversal's
 * result does not depend on its order (the closest hit, then the lowest id),
 * so every path's colour is the wavefront's bit for bit.
 * GB300, one frame, before and after (with the device-side iteration loop):
 * Cornell box 500x500 1233 -> 653 us, spheres 1920x1080 3438 -> 2069 us.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include "pt_bvh.cuh"
#include "../../include/pt.h"
#include "pt_internal.h"
#include "pt_shade.cuh"
#include "pt_wave.cuh"

using namespace ptd;

namespace {

// A lane's traversal stack (shared memory, one column per thread) and counts.
struct LaneTrace {
  uint2* stk;   // (child base, slot mask | second nearest << 8 | 0x800)
  float* stkt;  // entry distance of the group's nearest child
  int max_stack;
  uint32_t* err;
  uint32_t nodes, prims;
};

// Closest hit (ANY: some hit) of one ray in [tmin, tmax): (t bits << 32) | id,
// id PT_NO_HIT without a hit.
template <bool ANY>
__device__ __forceinline__ unsigned long long lane_trace(const DevScene& S, V3 o, V3 d, float tmin,
                                                         float tmax, float tm, LaneTrace& lt) {
  unsigned long long best =
      ((unsigned long long)__float_as_uint(tmax) << 32) | (unsigned long long)PT_NO_HIT;
  if (nan_ray(o, d) || S.num_prims == 0) return best;
  BoxRay ray;
  ray.o = o;
  ray.tmin = tmin;
  ray.set_direction(d);
  const WtRay wt = wt_setup(d);
  const int bd = blockDim.x;
  uint32_t cur = S.root;
  int sp = 0;
  while (true) {
    NodeHits h;
    h.ihit = h.leafmask = 0;
    h.k1 = h.k2 = 0xffffffffu;
    float tlim = __uint_as_float((uint32_t)(best >> 32)) * 1.0000005f;
    node_step(S.nodes + 5 * (size_t)cur, ray, tlim, h);
    lt.nodes++;
    uint32_t pm = leaf_prims(h);
    while (pm) {
      const int j = __ffs(pm) - 1;
      pm &= pm - 1;
      const PrimRec p = load_prim(S.prims, h.pbase + (uint32_t)j);
      lt.prims++;
      float t, bu, bv;
      if (prim_test<true>(S, p, o, d, wt, tmin, tmax, t, bu, bv, tm))
        best = min(best, ((unsigned long long)__float_as_uint(t) << 32) | prim_id(p));
    }
    if (ANY && (uint32_t)best != PT_NO_HIT) return best;
    tlim = __uint_as_float((uint32_t)(best >> 32)) * 1.0000005f;
    const uint32_t rest = h.ihit & ~(1u << (h.k1 & 7u));
    if (h.ihit && rest) {
      if (sp >= lt.max_stack) {
        atomicOr(lt.err, 1u);  // abandon this ray (the host reports the error)
        return best;
      }
      lt.stk[sp * bd] = make_uint2(h.child_base, rest | ((h.k2 & 7u) << 8) | 0x800u);
      lt.stkt[sp * bd] = __uint_as_float(h.k2 & 0xfffffff8u);
      sp++;
    }
    if (h.ihit && !(__uint_as_float(h.k1 & 0xfffffff8u) > tlim)) {
      cur = h.child_base + (h.k1 & 7u);
      continue;
    }
    // the deepest pending group that does not begin beyond the hit
    bool found = false;
    while (sp > 0) {
      const uint2 e = lt.stk[(sp - 1) * bd];
      if (lt.stkt[(sp - 1) * bd] > tlim) {
        sp--;
        continue;
      }
      uint32_t m = e.y & 0xffu;
      const uint32_t slot = (e.y & 0x800u) ? (e.y >> 8) & 7u : (uint32_t)(__ffs(m) - 1);
      m &= ~(1u << slot);
      cur = e.x + slot;
      if (m == 0) sp--;
      else lt.stk[(sp - 1) * bd].y = m;
      found = true;
      break;
    }
    if (!found) return best;
  }
}

// The hit record of an extension ray (as k_trace_t<TRACE_EXT> writes it).
__device__ __forceinline__ float4 lane_hit(const DevScene& S, V3 o, V3 d, float tmin, float tmax,
                                           float tm, LaneTrace& lt) {
  const unsigned long long best = lane_trace<false>(S, o, d, tmin, tmax, tm, lt);
  const uint32_t id = (uint32_t)best;
  if (id == PT_NO_HIT) return make_float4(tmax, 0.f, 0.f, __uint_as_float(PT_NO_HIT));
  const uint32_t leaf = __ldg(S.leaf_of_id + id);
  const PrimRec p = load_prim(S.prims, leaf);
  float t = 0.f, bu = 0.f, bv = 0.f;
  if (prim_type(p) == PT_PRIM_TRIANGLE) tri_candidate(p, o, wt_setup(d), tmin, tmax, t, bu, bv);
  return make_float4(__uint_as_float((uint32_t)(best >> 32)), bu, bv, __uint_as_float(leaf));
}

// Reference mode: the bounces of one path (color()'s loop) to its end.
template <bool BATCH>
__device__ __forceinline__ void run_path(const DevScene& S0, const WaveState& W,
                                         const WaveCtl& ctl, const BatchRefs& br, V3 o, V3 d,
                                         float tmin, float tmax, V3 thr, V3 rad, float tm, uint4 st,
                                         LaneTrace& lt, uint32_t& ext, uint32_t& shadow) {
  const DevScene& S = path_scene<BATCH>(S0, br, st.z);
  const PathCtl pc = path_ctl<BATCH>(ctl, br, st.z);
  V3 col;
  while (true) {
    ext++;
    const float4 hit = lane_hit(S, o, d, tmin, tmax, tm, lt);
    NeeCtx n;
    Tail tl;
    const int step = shade_step<true>(S, hit, o, d, tm, st, thr, rad, n, tl, col);
    if (step == STEP_ENDED) break;
    if (step == STEP_SHADOW) {
      shadow++;
      // programs/hit.cu:16-24 under the closest-hit rule: the light must be
      // the first thing the shadow ray hits
      const uint32_t id =
          (uint32_t)lane_trace<false>(S, n.P, n.Wi, 1e-3f, PT_RAY_TMAX, tm, lt);
      bool occluded = true;
      if (id != PT_NO_HIT) {
        const PrimRec p = load_prim(S.prims, __ldg(S.leaf_of_id + id));
        const bool is_light = S.mats[prim_material(p)].type == PT_MAT_DIFFUSE_LIGHT;
        occluded = !(is_light && dot(n.N, n.Wi) > 0.f);
      }
      finish_step(S, st, thr, rad, n, occluded, tl);
    }
    if (!path_advance(pc, st, thr, rad, tl, col)) break;
    o = tl.origin;
    d = tl.direction;
    tmin = 1e-3f;
    tmax = PT_RAY_TMAX;
  }
  finalize_path(W, st.y, col);
}

// Consistent mode: the same; word holds the guide-record word (the bounces left
// are past the guided depth) and whether the NEE term nee_c of the previous
// bounce still waits for its occlusion ray (nee_wi).  tmax 0: it is all that
// the path waits for.
template <bool BATCH>
__device__ __forceinline__ void run_path_c(const DevScene& S0, const WaveState& W,
                                           const WaveCtl& ctl, const BatchRefs& br, V3 o, V3 d,
                                           float tmin, float tmax, V3 thr, V3 rad, int word,
                                           float4 nee_wi, float4 nee_c, float tm, uint4 st,
                                           LaneTrace& lt, uint32_t& ext, uint32_t& shadow) {
  const DevScene& S = path_scene<BATCH>(S0, br, st.z);
  const PathCtl pc = path_ctl<BATCH>(ctl, br, st.z);
  if (word & PT_CODE_PENDING) {
    const bool hit =
        (uint32_t)lane_trace<true>(S, o, f4xyz(nee_wi), 1e-3f, nee_c.w, tm, lt) != PT_NO_HIT;
    nee_arrived(W, hit ? 1.f : 0.f, nee_c, st.y, word, rad);
  }
  while (tmax != 0.f) {
    ext++;
    const float4 hit = lane_hit(S, o, d, tmin, tmax, tm, lt);
    BounceC b;
    b.code = 0.f;
    shade_step_c<false, true>(S, pc, W, 0u, 0u, hit, o, d, tm, st, thr, rad, b);
    if (b.shadow) {
      shadow++;
      if ((uint32_t)lane_trace<true>(S, b.P, b.Wi, 1e-3f, b.tmax, tm, lt) == PT_NO_HIT)
        rad += b.C;
    }
    if (b.ended) break;
    o = b.P;
    d = b.dcont;
    tmin = 1e-3f;
    tmax = PT_RAY_TMAX;
  }
  finalize_path(W, st.y, rad);
  guide_end(W, st.y, (float)(word & 6), rad);
}

template <int MODE, bool BATCH>
__global__ void __launch_bounds__(PT_TAIL_BLOCK)
    k_tail(DevScene S0, WaveState W, const WaveCtl* __restrict__ ctlp, int max_stack, BatchRefs br,
           int count) {
  extern __shared__ __align__(16) unsigned char smem[];
  const WaveCounters c = *W.ctr;
  const WaveCtl ctl = *ctlp;
  if (!tail_ready(c, ctl)) return;
  const uint32_t total = c.n_cur + (uint32_t)(ctl.chunk_paths - c.next_path);
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (PT_TAIL_BLOCK / 32);
  const uint32_t warp = blockIdx.x * (PT_TAIL_BLOCK / 32) + (threadIdx.x >> 5);
  const uint32_t lanes = min(32u, max(1u, (total + warps - 1) / warps));
  LaneTrace lt;
  lt.stk = (uint2*)smem + threadIdx.x;
  lt.stkt = (float*)((uint2*)smem + (size_t)max_stack * PT_TAIL_BLOCK) + threadIdx.x;
  lt.max_stack = max_stack;
  lt.err = &W.ctr->error;
  lt.nodes = lt.prims = 0;
  uint32_t ext = 0, shadow = 0;
  const PathBuf& pb = W.path[c.parity];
  for (uint32_t base = warp * lanes; base < total; base += warps * lanes) {
    const uint32_t j = base + (uint32_t)lane;
    if ((uint32_t)lane < lanes && j < total) {
      V3 o, d, thr = v3(1.f), rad = v3(0.f);
      float tmin = 1e-6f, tmax = PT_RAY_TMAX, tm;
      int word = 0;
      float4 nee_wi = make_float4(0.f, 0.f, 0.f, 0.f), nee_c = nee_wi;
      uint4 st;
      if (j < c.n_cur) {
        const float4 o4 = pb.ray_o[j], d4 = pb.ray_d[j], t4 = pb.thr[j], r4 = pb.rad[j];
        o = f4xyz(o4);
        tmin = o4.w;
        d = f4xyz(d4);
        tmax = d4.w;
        thr = f4xyz(t4);
        tm = t4.w;
        rad = f4xyz(r4);
        word = (int)r4.w;
        if (MODE == 1 && (word & PT_CODE_PENDING)) {
          nee_wi = W.nee[c.parity].Wi[j];
          nee_c = W.nee[c.parity].C[j];
        }
        st = pb.st[j];
      } else {
        const NewPath np =
            new_path<BATCH>(S0, ctl, br, (uint32_t)c.next_path + (j - c.n_cur));
        o = v3(np.ray.o.x, np.ray.o.y, np.ray.o.z);
        d = v3(np.ray.d.x, np.ray.d.y, np.ray.d.z);
        tm = np.tm;
        st = np.st;
      }
      if (MODE == 1)
        run_path_c<BATCH>(S0, W, ctl, br, o, d, tmin, tmax, thr, rad, word, nee_wi, nee_c, tm, st,
                          lt, ext, shadow);
      else
        run_path<BATCH>(S0, W, ctl, br, o, d, tmin, tmax, thr, rad, tm, st, lt, ext, shadow);
    }
    __syncwarp();
  }
  ext = __reduce_add_sync(0xffffffffu, ext);
  shadow = __reduce_add_sync(0xffffffffu, shadow);
  if (lane == 0 && ext) {
    atomicAdd(&W.ctr->ext_rays, (unsigned long long)ext);
    if (shadow) atomicAdd(&W.ctr->shadow_rays, (unsigned long long)shadow);
  }
  if (count) {
    atomicAdd(&W.ctr->node_fetches, (unsigned long long)lt.nodes);
    atomicAdd(&W.ctr->prim_tests, (unsigned long long)lt.prims);
  }
}

// Marks the chunk drained once k_tail took its last paths (host loops read
// the counters; a device loop's next chunk resets them).
__global__ void k_tail_end(WaveState W, const WaveCtl* __restrict__ ctlp) {
  WaveCounters& c = *W.ctr;
  if (!tail_ready(c, *ctlp)) return;
  c.next_path = ctlp->chunk_paths;
  c.n_cur = c.n_wait = c.n_occ = 0;
}

constexpr int kMaxSmem = 200 * 1024;  // the same for every context: a function attribute is shared

size_t tail_smem(int max_stack) {
  return (size_t)PT_TAIL_BLOCK * max_stack * (sizeof(uint2) + sizeof(float));
}

template <typename K>
int tail_occupancy(K k, int max_stack) {
  int blocks = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, PT_TAIL_BLOCK,
                                                    tail_smem(max_stack)) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return blocks < 1 ? 1 : blocks;
}

// Once per device, with that device current.
constexpr int kMaxDev = 64;
std::atomic<bool> g_smem_set[kMaxDev];

}  // namespace

namespace pt {

uint32_t tail_paths(int max_stack, const LaunchCfg& lc, uint32_t limit) {
  if (tail_smem(max_stack) > kMaxSmem) return 0u;
  if (limit != PT_TAIL_AUTO) return limit;
  return lc.tex ? PT_TAIL_PATHS_TEX : PT_TAIL_PATHS;
}

cudaError_t set_tail_smem() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < kMaxDev && g_smem_set[dev]) return cudaSuccess;
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if ((e = cudaFuncSetAttribute(k_tail<0, false>, attr, kMaxSmem)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_tail<1, false>, attr, kMaxSmem)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_tail<0, true>, attr, kMaxSmem)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_tail<1, true>, attr, kMaxSmem)) != cudaSuccess) return e;
  if (dev >= 0 && dev < kMaxDev) g_smem_set[dev] = true;
  return cudaSuccess;
}

int tail_blocks_per_sm(int max_stack, bool batch) {
  if (tail_smem(max_stack) > kMaxSmem) return 1;
  const int a = batch ? tail_occupancy(k_tail<0, true>, max_stack)
                      : tail_occupancy(k_tail<0, false>, max_stack);
  const int b = batch ? tail_occupancy(k_tail<1, true>, max_stack)
                      : tail_occupancy(k_tail<1, false>, max_stack);
  return a < b ? a : b;
}

void launch_tail(const DevScene& S, const WaveState& W, const WaveCtl* ctl, int max_stack,
                 bool counters, const LaunchCfg& lc, int mode, const BatchRefs* br, bool mark,
                 cudaStream_t st) {
  if (tail_smem(max_stack) > kMaxSmem) return;  // the wavefront drains to the last path
  const size_t smem = tail_smem(max_stack);
  const BatchRefs b = br ? *br : BatchRefs{};
  const int cnt = counters ? 1 : 0;
  if (br && mode == 1)
    k_tail<1, true><<<lc.tail_grid, PT_TAIL_BLOCK, smem, st>>>(S, W, ctl, max_stack, b, cnt);
  else if (br)
    k_tail<0, true><<<lc.tail_grid, PT_TAIL_BLOCK, smem, st>>>(S, W, ctl, max_stack, b, cnt);
  else if (mode == 1)
    k_tail<1, false><<<lc.tail_grid, PT_TAIL_BLOCK, smem, st>>>(S, W, ctl, max_stack, b, cnt);
  else
    k_tail<0, false><<<lc.tail_grid, PT_TAIL_BLOCK, smem, st>>>(S, W, ctl, max_stack, b, cnt);
  if (mark) k_tail_end<<<1, 1, 0, st>>>(W, ctl);
}

}  // namespace pt
