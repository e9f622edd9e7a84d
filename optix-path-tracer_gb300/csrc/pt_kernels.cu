/*
 * pt_kernels.cu - wavefront path tracing kernels for sm_103a.
 *
 * One path = one (pixel, frame) sample of programs/raygen.cu:148-167.  The
 * reference runs each path in one OptiX megakernel thread; here the live
 * paths stream through stage kernels, and new paths top the buffer up to its
 * capacity every iteration (regeneration), so the GPU stays full:
 *
 *   k_generate      renderPixel up to color()'s loop: TEA seed, jitter,
 *                   thin-lens camera ray, time draw (raygen.cu:148-162,50-69)
 *   k_trace_t<EXT>  closest hit through the BVH8 (replaces rtTrace)
 *   k_shade         miss programs, Get_HitRecord, closest-hit programs; the
 *                   NEE of Direct_Light stops at the shadow ray
 *   k_trace_t<SHADOW> shadow rays (programs/hit.cu:16-24, closest-hit rule)
 *   k_finish        rest of Direct_Light (MIS), BSDF continuation
 *   k_advance       counter bookkeeping (one thread)
 * The consistent mode (NEE over lights and the environment with MIS) samples
 * the continuation before the occlusion test is known, so k_shade_c passes
 * the path on with its NEE term pending, and the next iteration traces both
 * rays in one launch (k_trace_t<BOTH>: extension rays, then occlusion rays,
 * which any hit before the light ends) and adds the term.  Trace warps take
 * rays from a per-launch counter (ray_next), so no warp sits idle while others
 * still have rays.
 * Without lights (or a sampled environment) the shadow stages are not
 * launched.  The iterations of a chunk run in a conditional graph node that
 * k_advance ends; the last few paths go to the tail kernel (pt_tail.cu).
 * Path state is kept in queue order: paths that continue are appended,
 * compacted with warp-aggregated atomics (ballot + popc prefix), to the other
 * buffer of a ping-pong pair, so every kernel streams its arrays
 * contiguously.  Ended paths write their colour to a per-path result slot,
 * and k_accumulate adds results to the accumulator in frame order, so the
 * image does not depend on scheduling.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <algorithm>
#include "pt_device.cuh"
#include "pt_internal.h"
#include "pt_shade.cuh"
#include "pt_wave.cuh"

using namespace ptd;

// -------------------------------------------------- warp-aggregated push --
__device__ __forceinline__ uint32_t warp_push(uint32_t* counter, bool active) {
  uint32_t mask = __ballot_sync(0xffffffffu, active);
  if (!active) return 0;
  int lane = threadIdx.x & 31;
  int leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
  base = __shfl_sync(mask, base, leader);
  return base + __popc(mask & ((1u << lane) - 1u));
}


// Appends to the next buffer and to the shadow queue with one atomic for both
// (n_next, n_shadow as one 64-bit word): all warps of a launch append to the
// same counters, which serialises them (Cornell box, 64 frames of 512x512 on a
// GB300: shading 5.3 -> 4.5 ms).  Each lane gets its place in either.
__device__ __forceinline__ void push_both(WaveCounters* ctr, bool next, bool shadow,
                                          uint32_t& next_pos, uint32_t& shadow_pos) {
  const uint32_t mn = __ballot_sync(0xffffffffu, next), ms = __ballot_sync(0xffffffffu, shadow);
  const int lane = threadIdx.x & 31;
  unsigned long long base = 0;
  if (lane == 0 && (mn | ms))
    base = atomicAdd((unsigned long long*)&ctr->n_next,
                     (unsigned long long)__popc(mn) | ((unsigned long long)__popc(ms) << 32));
  base = __shfl_sync(0xffffffffu, base, 0);
  next_pos = (uint32_t)base + __popc(mn & ((1u << lane) - 1u));
  shadow_pos = (uint32_t)(base >> 32) + __popc(ms & ((1u << lane) - 1u));
}

// Writes a path that goes on to place pos of the next buffer.  tm: the path's
// time (color()'s prd.time), carried in the throughput's w.
__device__ __forceinline__ void path_store(const WaveState& W, const WaveCounters& c, uint32_t pos,
                                           uint4 st, V3 thr, V3 rad, const Tail& tl, float tm) {
  const PathBuf& nb = W.path[c.parity ^ 1u];
  nb.ray_o[pos] = make_float4(tl.origin.x, tl.origin.y, tl.origin.z, 1e-3f);
  nb.ray_d[pos] = make_float4(tl.direction.x, tl.direction.y, tl.direction.z, PT_RAY_TMAX);
  nb.thr[pos] = make_float4(thr.x, thr.y, thr.z, tm);
  nb.rad[pos] = make_float4(rad.x, rad.y, rad.z, 0.f);
  nb.st[pos] = st;
}

// ------------------------------------------------------------- kernels ----

template <bool BATCH>
__global__ void k_generate(DevScene S0, WaveState W, const WaveCtl* __restrict__ ctlp,
                           BatchRefs br) {
  WaveCounters c = *W.ctr;
  WaveCtl ctl = *ctlp;
  uint32_t n = gen_count(c, ctl, (uint32_t)W.slots);
  const PathBuf& pb = W.path[c.parity];
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    uint32_t pos = c.n_cur + j;
    uint32_t pid = (uint32_t)(c.next_path + j);
    NewPath np = new_path<BATCH>(S0, ctl, br, pid);
    pb.ray_o[pos] = make_float4(np.ray.o.x, np.ray.o.y, np.ray.o.z, 1e-6f);
    pb.ray_d[pos] = make_float4(np.ray.d.x, np.ray.d.y, np.ray.d.z, PT_RAY_TMAX);
    pb.thr[pos] = make_float4(1.f, 1.f, 1.f, np.tm);
    pb.rad[pos] = make_float4(0.f, 0.f, 0.f, 0.f);
    pb.st[pos] = np.st;
  }
}

// -------------------------------------------------- material-ordered shading --
// The trace kernel puts every extension ray on the list of its shading key
// (miss or material type), and a warp of the sorted shade kernels takes 32
// entries of one list: it runs one material's code, and neighbouring warps the
// same code, which is what bounds these kernels (lanes in use, instruction
// fetch and the latency behind both).  The order does not change any path's
// result.  Costly materials come first, so the launch ends on cheap ones.
// GB300, before (tiles of 1024 paths sorted in shared memory, with barriers
// around; 7 blocks per SM) -> after: 64 frames of the 2.1 M-triangle terrain
// 76.3 -> 64.9 ms, one 1280x720 frame 973 -> 853 us, textures 3113 -> 2284 us,
// guided frames 22.1 -> 19.6 ms.  Scenes of cheap materials alone are faster in
// path order: random spheres 155.8 against 167.7 ms with lists, Cornell box
// 15.5 against 16.8 (the lists' writes and the scattered reads cost more).
__device__ __forceinline__ uint32_t list_key(int rank) {
  constexpr uint32_t order = 0x04123567u;  // AS, TS, ON, dielectric, metal, Lambertian, light, miss
  return (order >> (4 * rank)) & 15u;
}

// Position of this lane's path in chunk w (32 entries) of the lists, or
// 0xffffffff past a list's end; false past the last chunk.
__device__ __forceinline__ bool list_entry(const WaveState& W, uint32_t w, uint32_t& i) {
  i = 0xffffffffu;
#pragma unroll
  for (int rank = 0; rank < PT_SHADE_KEYS; rank++) {
    const uint32_t key = list_key(rank), n = W.listed[key * PT_LISTED_STRIDE], chunks = (n + 31) / 32;
    if (w < chunks) {
      const uint32_t e = 32 * w + (threadIdx.x & 31);
      if (e < n) i = __ldcs(&W.lists[(size_t)key * (size_t)W.slots + e]);
      return true;
    }
    w -= chunks;
  }
  return false;
}

// Loop of a shade kernel over its paths: by the lists (SORT) or a plain
// grid-stride loop.  Every lane of a warp runs every step (the queue appends
// inside are warp-aggregated).
#define SHADE_LOOP(CALL)                                                           \
  if (SORT) {                                                                      \
    uint32_t i;                                                                    \
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;                \
         list_entry(W, w, i);    w += (gridDim.x * blockDim.x) >> 5) {             \
      CALL;                                                                        \
    }                                                                              \
  } else {                                                                         \
    uint32_t stride = gridDim.x * blockDim.x;                                      \
    uint32_t iters = (n + stride - 1) / stride;                                    \
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;                            \
    for (uint32_t it = 0; it < iters; it++, i += stride) {                         \
      CALL;                                                                        \
    }                                                                              \
  }

// One path of k_shade (position i of the current buffer; all lanes of the
// warp call it together: the queue appends are warp-aggregated).
template <bool BATCH, bool TEX, bool LIGHTS>
__device__ __forceinline__ void shade_path(const DevScene& S0, const WaveState& W,
                                         const WaveCounters& c, const WaveCtl& ctl,
                                         const BatchRefs& br, uint32_t i, bool active) {
  const PathBuf& pb = W.path[c.parity];
  uint4 st = make_uint4(0, 0, 0, 0);
  V3 thr = v3(0.f), rad = v3(0.f), col = v3(0.f);
  float tm = 0.f;
  Tail tl;
  NeeCtx n;
  int step = -1;
  if (active) st = pb.st[i];
  const DevScene& S = path_scene<BATCH>(S0, br, st.z);
  if (active) {
    float4 t4 = pb.thr[i], r4 = pb.rad[i];
    thr = f4xyz(t4);
    tm = t4.w;
    rad = f4xyz(r4);
    step = shade_step<TEX>(S, W.hit[i], f4xyz(pb.ray_o[i]), f4xyz(pb.ray_d[i]), tm, st, thr, rad,
                           n, tl, col);
  }
  const bool shadow = step == STEP_SHADOW;
  bool cont = false;
  uint32_t pos, spos;
  if (LIGHTS) {
    if (step == STEP_TAIL) cont = path_advance(path_ctl<BATCH>(ctl, br, st.z), st, thr, rad, tl, col);
    if (__any_sync(0xffffffffu, shadow)) push_both(W.ctr, cont, shadow, pos, spos);
    else pos = warp_push(&W.ctr->n_next, cont);
  } else {
    spos = warp_push(&W.ctr->n_shadow, shadow);
  }
  // shadow rays: park the Direct_Light context and the path state
  if (shadow) {
    W.sh.P[spos] = make_float4(n.P.x, n.P.y, n.P.z, n.lightPDF);
    W.sh.N[spos] = make_float4(n.N.x, n.N.y, n.N.z, __int_as_float(n.lindex));
    W.sh.Wo[spos] = make_float4(n.Wo.x, n.Wo.y, n.Wo.z, __uint_as_float(n.mid));
    W.sh.Wi[spos] = make_float4(n.Wi.x, n.Wi.y, n.Wi.z, 0.f);
    if (n.textured) W.sh.C[spos] = make_float4(n.tcol.x, n.tcol.y, n.tcol.z, 0.f);
    W.sh.st[spos] = st;
    W.sh.thr[spos] = make_float4(thr.x, thr.y, thr.z, tm);
    W.sh.rad[spos] = make_float4(rad.x, rad.y, rad.z, 0.f);
  }
  if (!LIGHTS) {
    if (step == STEP_ENDED) finalize_path(W, st.y, col);
    if (step == STEP_TAIL) {
      cont = path_advance(path_ctl<BATCH>(ctl, br, st.z), st, thr, rad, tl, col);
      if (!cont) finalize_path(W, st.y, col);
    }
    pos = warp_push(&W.ctr->n_next, cont);
  } else if (step == STEP_ENDED || (step == STEP_TAIL && !cont)) {
    finalize_path(W, st.y, col);
  }
  if (cont) path_store(W, c, pos, st, thr, rad, tl, tm);
}

// TEX: the scene has textured materials (their colours are evaluated at
// the hit); the other variant carries no texture code at all.
// LIGHTS: some scene has lights.  Then most warps queue shadow rays beside
// paths, with one atomic for both; without any, the two appends stay apart
// (random spheres, 128 frames at 1920x1080: 157.3 against 158.3 ms).  The code of
// the shadow rays stays in that variant, although no path takes it: without it
// the compiler's schedule is the slower one (the same render 107.7 -> 120.1 ms,
// one frame 1505 -> 1525 us, at 80 bytes of spill stores in place of 72).
template <bool BATCH, bool SORT, bool TEX, bool LIGHTS>
__global__ void __launch_bounds__(PT_SHADE_BLOCK, PT_SHADE_MINBLOCKS) k_shade(DevScene S0, WaveState W,
                                                          const WaveCtl* __restrict__ ctlp,
                                                          BatchRefs br) {
  WaveCounters c = *W.ctr;
  WaveCtl ctl = *ctlp;
  uint32_t n = c.n_cur + gen_count(c, ctl, (uint32_t)W.slots);
  SHADE_LOOP((shade_path<BATCH, TEX, LIGHTS>(S0, W, c, ctl, br, i, i < n)))
}

template <bool BATCH>
__global__ void __launch_bounds__(PT_SHADE_BLOCK) k_finish(DevScene S0, WaveState W,
                                                           const WaveCtl* __restrict__ ctlp,
                                                           BatchRefs br) {
  WaveCounters c = *W.ctr;
  WaveCtl ctl = *ctlp;
  uint32_t n = c.n_shadow;
  uint32_t stride = gridDim.x * blockDim.x;
  uint32_t iters = (n + stride - 1) / stride;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  for (uint32_t it = 0; it < iters; it++, i += stride) {
    bool active = i < n;
    uint4 st = make_uint4(0, 0, 0, 0);
    V3 thr = v3(0.f), rad = v3(0.f);
    float tm = 0.f;
    Tail tl;
    if (active) st = W.sh.st[i];
    const DevScene& S = path_scene<BATCH>(S0, br, st.z);
    if (active) {
      const float4 t4 = W.sh.thr[i];
      thr = f4xyz(t4);
      tm = t4.w;
      rad = f4xyz(W.sh.rad[i]);
      float4 P4 = W.sh.P[i], N4 = W.sh.N[i], Wo4 = W.sh.Wo[i], Wi4 = W.sh.Wi[i];
      NeeCtx n;
      n.P = f4xyz(P4);
      n.N = f4xyz(N4);
      n.Wo = f4xyz(Wo4);
      n.Wi = f4xyz(Wi4);
      n.lightPDF = P4.w;
      n.lindex = __float_as_int(N4.w);
      n.mid = __float_as_uint(Wo4.w);
      if (S.mats[n.mid].tex0 >= 0) n.tcol = f4xyz(W.sh.C[i]);
      finish_step(S, st, thr, rad, n, Wi4.w != 0.f, tl);
    }
    bool cont = false;
    V3 col;
    if (active) cont = path_advance(path_ctl<BATCH>(ctl, br, st.z), st, thr, rad, tl, col);
    const uint32_t pos = warp_push(&W.ctr->n_next, cont);
    if (active && !cont) finalize_path(W, st.y, col);
    if (cont) path_store(W, c, pos, st, thr, rad, tl, tm);
  }
}

// ------------------------------------------------- consistent-mode stages --

// One path of k_shade_c (see shade_path): adds the NEE term of the previous
// bounce, then shades this one.
template <bool BATCH, bool GUIDE, bool TEX>
__device__ __forceinline__ void shade_c_path(const DevScene& S0, const WaveState& W,
                                           const WaveCounters& c, const WaveCtl& ctl,
                                           const BatchRefs& br, uint32_t i, bool active) {
  const PathBuf& pb = W.path[c.parity];
  uint4 st = make_uint4(0, 0, 0, 0);
  V3 thr = v3(0.f), rad = v3(0.f);
  float tm = 0.f;
  BounceC b;
  b.code = 0.f;
  b.ended = b.shadow = false;
  if (active) st = pb.st[i];
  const DevScene& S = path_scene<BATCH>(S0, br, st.z);
  if (active) {
    const float4 t4 = pb.thr[i], r4 = pb.rad[i], d4 = pb.ray_d[i];
    thr = f4xyz(t4);
    tm = t4.w;
    rad = f4xyz(r4);
    const int word = (int)r4.w;
    if (word & PT_CODE_PENDING) nee_arrived(W, W.nee[c.parity].Wi[i].w, W.nee[c.parity].C[i], st.y, word, rad);
    b.code = GUIDE ? (float)(word & 6) : 0.f;
    if (d4.w == 0.f)
      b.ended = true;
    else
      shade_step_c<GUIDE, TEX>(S, path_ctl<BATCH>(ctl, br, st.z), W, ctl.guide_depth, i, W.hit[i],
                               f4xyz(pb.ray_o[i]), f4xyz(d4), tm, st, thr, rad, b);
  }
  if (active && !b.shadow && b.ended) {
    finalize_path(W, st.y, rad);
    if (GUIDE) guide_end(W, st.y, b.code, rad);
  }
  // a path with an occlusion ray goes on (or, ended, waits) with its NEE term
  // pending; else the next vertex starts without a pending record of its own
  const bool push = active && (b.shadow || !b.ended);
  uint32_t pos, q;
  push_both(W.ctr, push, b.shadow, pos, q);
  if (push) {
    const PathBuf& nb = W.path[c.parity ^ 1u];
    const int word = GUIDE ? (int)b.code : 0;
    nb.ray_o[pos] = make_float4(b.P.x, b.P.y, b.P.z, 1e-3f);
    nb.ray_d[pos] = make_float4(b.dcont.x, b.dcont.y, b.dcont.z, b.ended ? 0.f : PT_RAY_TMAX);
    nb.thr[pos] = make_float4(thr.x, thr.y, thr.z, tm);
    nb.rad[pos] = make_float4(rad.x, rad.y, rad.z,
                              (float)(b.shadow ? word + PT_CODE_PENDING : word & 6));
    nb.st[pos] = st;
  }
  if (b.shadow) {
    const NeeBuf& ne = W.nee[c.parity ^ 1u];
    ne.queue[q] = pos;
    ne.Wi[pos] = make_float4(b.Wi.x, b.Wi.y, b.Wi.z, 0.f);
    ne.C[pos] = make_float4(b.C.x, b.C.y, b.C.z, b.tmax);
  }
  const uint32_t waits = __ballot_sync(0xffffffffu, b.shadow && b.ended);
  if (waits && (threadIdx.x & 31) == 0) atomicAdd(&W.ctr->n_wait_next, (uint32_t)__popc(waits));
}

template <bool BATCH, bool SORT, bool GUIDE, bool TEX>
__global__ void __launch_bounds__(PT_SHADE_BLOCK, PT_SHADE_MINBLOCKS) k_shade_c(DevScene S0, WaveState W,
                                                            const WaveCtl* __restrict__ ctlp,
                                                            BatchRefs br) {
  WaveCounters c = *W.ctr;
  WaveCtl ctl = *ctlp;
  uint32_t n = c.n_cur + gen_count(c, ctl, (uint32_t)W.slots);
  SHADE_LOOP((shade_c_path<BATCH, GUIDE, TEX>(S0, W, c, ctl, br, i, i < n)))
}

// Queue bookkeeping after an iteration.  With use_cond (the iteration loop
// is a graph conditional node) it also decides whether the loop goes on:
// not once the chunk has drained, an error was flagged, or the chunk's
// iteration bound is reached (then error bit 1 is set, so the loop always
// ends), or few enough paths are left for the tail kernel.
__global__ void k_advance(WaveState W, const WaveCtl* __restrict__ ctlp, int use_cond,
                          cudaGraphConditionalHandle cond) {
  WaveCounters& c = *W.ctr;
  const WaveCtl& ctl = *ctlp;
  uint32_t n_gen = gen_count(c, ctl, (uint32_t)W.slots);
  c.ext_rays += c.n_cur + n_gen - c.n_wait;
  c.shadow_rays += c.n_shadow;
  c.next_path += n_gen;
  c.drained = n_gen ? 1u : c.drained + 1u;
  c.n_cur = c.n_next;
  c.n_next = 0;
  c.n_wait = c.n_wait_next;
  c.n_wait_next = 0;
  c.n_occ = c.n_shadow;
  c.n_shadow = 0;
  c.ray_next[0] = 0;
  c.ray_next[1] = 0;
  for (int k = 0; k < PT_SHADE_KEYS; k++) W.listed[k * PT_LISTED_STRIDE] = 0;
  c.guide_rows = 0;
  c.parity ^= 1u;
  c.iter++;
  c.iters_total++;
  if (use_cond) {
    bool more = c.n_cur != 0 || c.next_path < ctl.chunk_paths;
    if (more && (unsigned long long)c.iter >= ctl.max_iter) c.error |= 2u;
    if (c.error || tail_ready(c, ctl)) more = false;
    cudaGraphSetConditional(cond, more ? 1u : 0u);
  }
}

// Starts a chunk: its controls, empty queues; first: zero totals and flags.
__global__ void k_chunk_begin(WaveState W, WaveCtl* ctl, WaveCtl v, int first) {
  *ctl = v;
  WaveCounters c{};
  if (!first) {
    const WaveCounters o = *W.ctr;
    c.error = o.error;
    c.ext_rays = o.ext_rays;
    c.shadow_rays = o.shadow_rays;
    c.node_fetches = o.node_fetches;
    c.prim_tests = o.prim_tests;
    c.iters_total = o.iters_total;
    c.chunks_done = o.chunks_done + (o.error ? 0u : 1u);
  }
  *W.ctr = c;
  for (int k = 0; k < PT_SHADE_KEYS; k++) W.listed[k * PT_LISTED_STRIDE] = 0;
}

// ------------------------------------------------------ batch chunk steps --
__global__ void k_batch_begin(WaveState W, WaveCtl* ctl, const BatchChunk* __restrict__ chunks,
                              int use_cond, cudaGraphConditionalHandle inner) {
  WaveCounters& c = *W.ctr;
  BatchChunk ch{};
  if (c.chunk < c.n_chunks) ch = chunks[c.chunk];
  else c.error |= 2u;  // no chunk left: run nothing
  ctl->chunk_paths = ch.paths;
  ctl->max_iter = ch.max_iter;
  ctl->seg_begin = ch.seg_begin;
  ctl->seg_end = ch.seg_end;
  ctl->pixels = ch.pixels;
  c.n_cur = 0;
  c.n_next = 0;
  c.n_shadow = c.n_occ = 0;
  c.n_wait = c.n_wait_next = 0;
  for (int k = 0; k < PT_SHADE_KEYS; k++) W.listed[k * PT_LISTED_STRIDE] = 0;
  c.parity = 0;
  c.iter = 0;
  c.next_path = 0;
  c.drained = 0;
  if (use_cond) cudaGraphSetConditional(inner, c.error || tail_ready(c, *ctl) ? 0u : 1u);
}

// acc[x, H-1-y] += (col, 1) in frame order for every pixel of every segment
// of the chunk (the batch form of k_accumulate).
__global__ void k_accumulate_batch(WaveState W, const WaveCtl* __restrict__ ctlp, BatchRefs br) {
  const WaveCtl ctl = *ctlp;
  const float4* __restrict__ results = W.results;
  if (ctl.seg_end <= ctl.seg_begin || W.ctr->error) return;
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ctl.pixels;
       g += gridDim.x * blockDim.x) {
    const BatchSeg& sg = br.segs[find_seg(br.segs, ctl.seg_begin, ctl.seg_end, g, true)];
    const BatchScene& B = br.scenes[sg.scene];
    uint32_t w = (uint32_t)B.width, h = (uint32_t)B.height, WH = w * h;
    uint32_t p = g - sg.pix_off;
    uint32_t y = fastdiv(p, B.w_m, B.w_l), x = p - y * w;
    size_t o = (size_t)(h - 1 - y) * w + x;
    float4 a = sg.acc[o];
    for (uint32_t f = 0; f < sg.frames; f++) {
      float4 r = results[(size_t)sg.path_off + (size_t)f * WH + p];
      a.x += r.x;
      a.y += r.y;
      a.z += r.z;
      a.w += 1.f;
    }
    sg.acc[o] = a;
  }
}

__global__ void k_batch_end(WaveState W, int use_cond, cudaGraphConditionalHandle outer) {
  WaveCounters& c = *W.ctr;
  c.chunk++;
  if (use_cond) cudaGraphSetConditional(outer, (c.chunk < c.n_chunks && !c.error) ? 1u : 0u);
}

// ------------------------------------------------ batch scene relocation --
__global__ void k_relocate_nodes(uint4* nodes, size_t n, uint32_t node_off, uint32_t prim_off) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    uint4 w = nodes[5 * i + 1];
    w.x += node_off;
    w.y += prim_off;
    nodes[5 * i + 1] = w;
  }
}

__global__ void k_relocate_prims(float4* prims, size_t n, uint32_t xform_off, uint32_t id_off,
                                 uint32_t mat_off) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    float4 r0 = prims[3 * i], r1 = prims[3 * i + 1], r2 = prims[3 * i + 2];
    uint32_t tag = __float_as_uint(r0.w);
    if (tag >> 8) tag += xform_off << 8;  // transform index + 1 (0: world space)
    r0.w = __uint_as_float(tag);
    r1.w = __uint_as_float(__float_as_uint(r1.w) + id_off);
    r2.w = __uint_as_float(__float_as_uint(r2.w) + mat_off);
    prims[3 * i] = r0;
    prims[3 * i + 1] = r1;
    prims[3 * i + 2] = r2;
  }
}

__global__ void k_relocate_ids(uint32_t* leaf_of_id, uint4* tri_attr, size_t n, uint32_t prim_off,
                               uint32_t attr_off) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    leaf_of_id[i] += prim_off;
    uint4 a = tri_attr[i];
    a.x += attr_off;
    a.y += attr_off;
    a.z += attr_off;
    tri_attr[i] = a;
  }
}

// acc[x, H-1-y] += (col, 1) in frame order (programs/raygen.cu:153-166)
__global__ void k_accumulate(const float4* __restrict__ results, const uint32_t* error, float4* acc,
                             int width, int height, int frames) {
  if (*error) return;
  uint32_t WH = (uint32_t)width * (uint32_t)height;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < WH; p += gridDim.x * blockDim.x) {
    uint32_t x = p % (uint32_t)width, y = p / (uint32_t)width;
    size_t o = (size_t)(height - 1 - y) * width + x;
    float4 a = acc[o];
    for (int f = 0; f < frames; f++) {
      float4 r = results[(size_t)f * WH + p];
      a.x += r.x;
      a.y += r.y;
      a.z += r.z;
      a.w += 1.f;
    }
    acc[o] = a;
  }
}

// The same accumulation into double sums (acc holds 4 doubles per pixel):
// for renders beyond a few thousand frames, where float sums of per-frame
// values lose the low bits of each new frame.
__global__ void k_accumulate64(const float4* __restrict__ results, const uint32_t* error,
                               double2* acc, int width, int height, int frames) {
  if (*error) return;
  uint32_t WH = (uint32_t)width * (uint32_t)height;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < WH; p += gridDim.x * blockDim.x) {
    uint32_t x = p % (uint32_t)width, y = p / (uint32_t)width;
    size_t o = (size_t)(height - 1 - y) * width + x;
    double2 a0 = acc[2 * o], a1 = acc[2 * o + 1];
    for (int f = 0; f < frames; f++) {
      float4 r = results[(size_t)f * WH + p];
      a0.x += (double)r.x;
      a0.y += (double)r.y;
      a1.x += (double)r.z;
      a1.y += 1.0;
    }
    acc[2 * o] = a0;
    acc[2 * o + 1] = a1;
  }
}

__global__ void k_paths_out(const float4* __restrict__ results, const uint32_t* error, float* out,
                            uint32_t n) {
  if (*error) return;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    float4 r = results[p];
    out[3 * p] = r.x;
    out[3 * p + 1] = r.y;
    out[3 * p + 2] = r.z;
  }
}

// programs/raygen.cu:136-146
__global__ void k_resolve(const float4* __restrict__ acc, uchar4* out, int n, int frame) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    float4 a = acc[p];
    float d = (float)(frame + 1);
    float r = fmaxf(0.f, fminf(ptm_sqrt(a.x / d), 1.f));
    float g = fmaxf(0.f, fminf(ptm_sqrt(a.y / d), 1.f));
    float b = fmaxf(0.f, fminf(ptm_sqrt(a.z / d), 1.f));
    out[p] = make_uchar4((unsigned char)(int)(255.99 * r), (unsigned char)(int)(255.99 * g),
                         (unsigned char)(int)(255.99 * b), (unsigned char)(int)(255.99 * 1.f));
  }
}

__global__ void k_pack_normals(const float* __restrict__ n3, size_t n, float4* n4) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    n4[i] = make_float4(n3[3 * i], n3[3 * i + 1], n3[3 * i + 2], 0.f);
}

// ------------------------------------------- environment sampling tables --
// Weight of texel (r, c) = luminance x sin(theta_r).  Each row's prefix is
// summed in double, sequentially, in the oracle's order, so the float CDFs
// come out identical on both sides.  FP64 arithmetic is scarce on this GPU,
// so the per-texel work (weights, then the normalising divisions) runs on
// every SM, and only the dependent additions of a row stay in one thread:
//   k_env_weights  pre[r][c] = weight (all texels)
//   k_env_prefix   pre[r][c] = running sum of row r, rows[r] = its total
//   k_env_cond     conditional CDFs (all entries)
__global__ void k_env_weights(const float4* __restrict__ env, int w, int h, double* pre) {
  const size_t n = (size_t)w * h;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / (size_t)w);
    float theta = PI_F * (((float)r + 0.5f) / (float)h);
    double sn = (double)pt_sinf(theta);
    float4 t = env[i];
    double lum = 0.2126 * (double)t.x + 0.7152 * (double)t.y + 0.0722 * (double)t.z;
    if (!(lum > 0.0)) lum = 0.0;
    pre[i] = lum * sn;
  }
}

__global__ void k_env_prefix(double* pre, int w, int h, double* rows) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= h) return;
  double* p = pre + (size_t)r * w;
  double acc = 0.0;
  for (int c = 0; c < w; c++) {
    acc = acc + p[c];
    p[c] = acc;
  }
  rows[r] = acc;
}

__global__ void k_env_cond(const double* __restrict__ pre, const double* __restrict__ rows, int w,
                           int h, float* cond) {
  const size_t n = (size_t)(w + 1) * h;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / (size_t)(w + 1));
    const int k = (int)(i - (size_t)r * (w + 1));
    const double a = rows[r];
    float v;
    if (k == 0) v = 0.f;
    else if (k == w) v = 1.f;
    else v = a > 0.0 ? (float)(pre[(size_t)r * w + k - 1] / a) : (float)((double)k / (double)w);
    cond[i] = v;
  }
}

// Marginal CDF over the row totals: the sums by one thread in the oracle's
// order (rows[] becomes the running sums), the divisions by the block.
// *valid: bit 0 the environment can be sampled, bit 1 its total is finite.
__global__ void k_env_marg(double* rows, int h, float* marg, float2* row, int* valid) {
  __shared__ double tot_s;
  if (blockIdx.x != 0) return;
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int r = 0; r < h; r++) tot = tot + rows[r];
    double mp = 0.0;
    for (int r = 0; r < h; r++) {
      mp = mp + rows[r];
      rows[r] = mp;
    }
    tot_s = tot;
    *valid = tot > 0.0 ? (isfinite(tot) ? 3 : 1) : 0;
  }
  __syncthreads();
  const double tot = tot_s;
  if (!(tot > 0.0)) return;
  for (int r = threadIdx.x; r < h; r += blockDim.x) marg[r + 1] = (float)(rows[r] / tot);
  if (threadIdx.x == 0) marg[0] = 0.f;
  __syncthreads();
  if (threadIdx.x == 0) marg[h] = 1.f;
  __syncthreads();
  for (int r = threadIdx.x; r < h; r += blockDim.x)
    row[r] = make_float2(marg[r + 1] - marg[r], pt_sinf(PI_F * (((float)r + 0.5f) / (float)h)));
}

// Where the searches of cdf_find_from start: row -1 the marginal CDF, rows
// 0..h-1 the conditional ones (a 2048 x 1024 sky: 2 M searches, 4 MB).
__global__ void k_env_index(const float* __restrict__ marg, const float* __restrict__ cond, int w,
                            int h, int marg_bits, int cond_bits, uint16_t* marg_idx,
                            uint16_t* cond_idx) {
  const size_t nm = ((size_t)1 << marg_bits) + 1, nc = ((size_t)1 << cond_bits) + 1;
  const size_t n = nm + nc * h;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    if (i < nm) {
      marg_idx[i] = (uint16_t)cdf_find(marg, h, (float)i / (float)(1 << marg_bits));
    } else {
      const size_t r = (i - nm) / nc, k = (i - nm) - r * nc;
      cond_idx[i - nm] =
          (uint16_t)cdf_find(cond + r * (w + 1), w, (float)k / (float)(1 << cond_bits));
    }
  }
}

// ------------------------------------------------------- host launchers ---
namespace pt {

static int g_num_sms = 0;

static int num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 1;
  }
  return g_num_sms;
}

int wave_grid(int kind, int max_stack, int block) {
  int blocks = 0;
  cudaError_t e = cudaSuccess;
  if (kind == 0)
    blocks = trace_blocks_per_sm(block, trace_smem(max_stack, block));
  else if (kind == 2 || kind == 4)
    blocks = tail_blocks_per_sm(max_stack, kind == 4);
  else if (kind == 3)
    blocks = one_blocks_per_sm();
  else
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_shade<false, false, false, true>, block, 0);
  if (e != cudaSuccess || blocks < 1) {
    cudaGetLastError();
    blocks = 1;
  }
  return blocks * num_sms();
}

LaunchCfg default_launch(int max_stack) {
  LaunchCfg lc;
  lc.trace_block = PT_TRACE_BLOCK;
  lc.shade_block = PT_SHADE_BLOCK;
  lc.sort = 1;
  lc.refetch = 32;
  lc.tex = 0;
  lc.motion = 0;
  lc.lights = lc.env = lc.one_grid = 0;
  lc.tail_grid = wave_grid(2, max_stack, PT_TAIL_BLOCK);
  lc.trace_grid = wave_grid(0, max_stack, lc.trace_block);
  lc.shade_grid = wave_grid(1, max_stack, lc.shade_block);
  return lc;
}

// The shading kernel of the integrator mode, guide, tile order and texture
// variant.
template <bool BATCH, bool TEX>
static void launch_shade(const DevScene& S, const WaveState& W, const WaveCtl* ctl, BatchRefs br,
                         int mode, bool guide, bool lights, int sort, int tgs, int sg, int sb,
                         cudaStream_t st) {
  if (mode == 1 && guide) {
    if (sort) k_shade_c<BATCH, true, true, TEX><<<tgs, sb, 0, st>>>(S, W, ctl, br);
    else k_shade_c<BATCH, false, true, TEX><<<sg, sb, 0, st>>>(S, W, ctl, br);
  } else if (mode == 1) {
    if (sort) k_shade_c<BATCH, true, false, TEX><<<tgs, sb, 0, st>>>(S, W, ctl, br);
    else k_shade_c<BATCH, false, false, TEX><<<sg, sb, 0, st>>>(S, W, ctl, br);
  } else if (lights) {
    if (sort) k_shade<BATCH, true, TEX, true><<<tgs, sb, 0, st>>>(S, W, ctl, br);
    else k_shade<BATCH, false, TEX, true><<<sg, sb, 0, st>>>(S, W, ctl, br);
  } else {
    if (sort) k_shade<BATCH, true, TEX, false><<<tgs, sb, 0, st>>>(S, W, ctl, br);
    else k_shade<BATCH, false, TEX, false><<<sg, sb, 0, st>>>(S, W, ctl, br);
  }
}

// Whether shading can queue shadow rays: Direct_Light samples lights only; the
// consistent mode samples the environment too.
static bool shadow_rays(const LaunchCfg& lc, int mode) {
  return lc.lights != 0 || (mode == 1 && lc.env != 0);
}

int iteration_kernels(const LaunchCfg& lc, int mode, bool guide) {
  return 4 + (mode != 1 && shadow_rays(lc, mode) ? 2 : 0) + (mode == 1 && guide ? 2 : 0);
}

void launch_chunk_begin(const WaveState& W, WaveCtl* ctl, const WaveCtl& v, bool first,
                        cudaStream_t st) {
  k_chunk_begin<<<1, 1, 0, st>>>(W, ctl, v, first ? 1 : 0);
}

// Blocks of a sorted shading launch: a warp per 32 paths of a full buffer (each
// list may end in a part of a chunk), at most PT_SORT_BLOCKS.
#ifndef PT_SORT_BLOCKS
#define PT_SORT_BLOCKS 8192
#endif
static int sort_grid(int slots, int block) {
  const long long warps = ((long long)slots + 31) / 32 + PT_SHADE_KEYS;
  const long long blocks = (warps * 32 + block - 1) / block;
  return (int)std::min<long long>(blocks, PT_SORT_BLOCKS);
}

template <bool BATCH>
static void launch_iteration_t(const DevScene& S, const WaveState& W, const WaveCtl* ctl,
                               int max_stack, bool counters, const LaunchCfg& lc, cudaStream_t st,
                               cudaEvent_t* ev, int mode, const BatchRefs& br, bool use_cond,
                               unsigned long long cond, const GuideInferArgs* gi) {
  const int sb = lc.shade_block, sg = lc.shade_grid;
  const BatchRefs* brp = BATCH ? &br : nullptr;
  const int tgs = sort_grid(W.slots, sb);
  if (ev) cudaEventRecordWithFlags(ev[0], st, cudaEventRecordExternal);
  k_generate<BATCH><<<sg, sb, 0, st>>>(S, W, ctl, br);
  if (ev) cudaEventRecordWithFlags(ev[1], st, cudaEventRecordExternal);
  const bool nee = shadow_rays(lc, mode);
  launch_trace(mode == 1 && nee ? TRACE_BOTH : TRACE_EXT, counters, S, W, ctl, max_stack, brp, lc,
               st);
  if (ev) cudaEventRecordWithFlags(ev[2], st, cudaEventRecordExternal);
  if (mode == 1 && gi) launch_guide_infer(S, W, ctl, *gi, 2 * num_sms(), st);
  if (lc.tex)
    launch_shade<BATCH, true>(S, W, ctl, br, mode, gi != nullptr, lc.lights != 0, lc.sort, tgs, sg, sb, st);
  else
    launch_shade<BATCH, false>(S, W, ctl, br, mode, gi != nullptr, lc.lights != 0, lc.sort, tgs, sg, sb, st);
  if (ev) cudaEventRecordWithFlags(ev[3], st, cudaEventRecordExternal);
  if (nee && mode != 1) launch_trace(TRACE_SHADOW, counters, S, W, ctl, max_stack, brp, lc, st);
  if (ev) cudaEventRecordWithFlags(ev[4], st, cudaEventRecordExternal);
  if (nee && mode != 1) k_finish<BATCH><<<sg, sb, 0, st>>>(S, W, ctl, br);
  k_advance<<<1, 1, 0, st>>>(W, ctl, use_cond ? 1 : 0, (cudaGraphConditionalHandle)cond);
  if (ev) cudaEventRecordWithFlags(ev[5], st, cudaEventRecordExternal);
}

// One wavefront iteration.
void launch_iteration(const DevScene& S, const WaveState& W, const WaveCtl* ctl, int max_stack,
                      bool counters, const LaunchCfg& lc, cudaStream_t st, cudaEvent_t* ev,
                      int mode, const BatchRefs* br, bool use_cond, unsigned long long cond,
                      const GuideInferArgs* gi) {
  if (br)
    launch_iteration_t<true>(S, W, ctl, max_stack, counters, lc, st, ev, mode, *br, use_cond, cond,
                             nullptr);
  else
    launch_iteration_t<false>(S, W, ctl, max_stack, counters, lc, st, ev, mode, BatchRefs{},
                              use_cond, cond, gi);
}

void launch_batch_begin(const WaveState& W, WaveCtl* ctl, const BatchChunk* chunks,
                        bool use_cond, unsigned long long inner, cudaStream_t st) {
  k_batch_begin<<<1, 1, 0, st>>>(W, ctl, chunks, use_cond ? 1 : 0,
                                 (cudaGraphConditionalHandle)inner);
}

void launch_batch_end(const WaveState& W, const WaveCtl* ctl, const BatchRefs& br,
                      bool use_cond, unsigned long long outer, cudaStream_t st) {
  k_accumulate_batch<<<num_sms() * 8, 256, 0, st>>>(W, ctl, br);
  k_batch_end<<<1, 1, 0, st>>>(W, use_cond ? 1 : 0, (cudaGraphConditionalHandle)outer);
}

void launch_relocate(uint4* nodes, size_t n_nodes, uint32_t node_off, uint32_t prim_off,
                     float4* prims, size_t n_prims, uint32_t xform_off, uint32_t id_off,
                     uint32_t mat_off, uint32_t* leaf_of_id, uint4* tri_attr, uint32_t attr_off,
                     cudaStream_t st) {
  int g = num_sms() * 4;
  if (n_nodes) k_relocate_nodes<<<g, 256, 0, st>>>(nodes, n_nodes, node_off, prim_off);
  if (n_prims) {
    k_relocate_prims<<<g, 256, 0, st>>>(prims, n_prims, xform_off, id_off, mat_off);
    k_relocate_ids<<<g, 256, 0, st>>>(leaf_of_id, tri_attr, n_prims, prim_off, attr_off);
  }
}

void launch_pack_normals(const float* n3, size_t n, float4* n4, cudaStream_t st) {
  k_pack_normals<<<num_sms() * 4, 256, 0, st>>>(n3, n, n4);
}

void launch_accumulate(const WaveState& W, float4* acc, int w, int h, int frames, cudaStream_t st) {
  k_accumulate<<<num_sms() * 8, 256, 0, st>>>(W.results, &W.ctr->error, acc, w, h, frames);
}

void launch_accumulate64(const WaveState& W, double* acc, int w, int h, int frames,
                         cudaStream_t st) {
  k_accumulate64<<<num_sms() * 8, 256, 0, st>>>(W.results, &W.ctr->error, (double2*)acc, w, h,
                                               frames);
}

void launch_paths_out(const WaveState& W, float* out, uint32_t n, cudaStream_t st) {
  k_paths_out<<<num_sms() * 8, 256, 0, st>>>(W.results, &W.ctr->error, out, n);
}

void launch_env_cdf(const float4* env, int w, int h, float* marg, float* cond, double* rows,
                    double* pre, int* valid, float2* row, uint16_t* marg_idx, int marg_bits,
                    uint16_t* cond_idx, int cond_bits, cudaStream_t st) {
  const int g = num_sms() * 8;
  k_env_weights<<<g, 256, 0, st>>>(env, w, h, pre);
  k_env_prefix<<<(h + 31) / 32, 32, 0, st>>>(pre, w, h, rows);
  k_env_cond<<<g, 256, 0, st>>>(pre, rows, w, h, cond);
  k_env_marg<<<1, 256, 0, st>>>(rows, h, marg, row, valid);
  if (marg_idx)
    k_env_index<<<g, 256, 0, st>>>(marg, cond, w, h, marg_bits, cond_bits, marg_idx, cond_idx);
}

void launch_resolve(const float4* acc, uchar4* out, int n, int frame, cudaStream_t st) {
  k_resolve<<<num_sms() * 8, 256, 0, st>>>(acc, out, n, frame);
}

}  // namespace pt
