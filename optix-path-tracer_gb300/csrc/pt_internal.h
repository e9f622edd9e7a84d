/*
 * pt_internal.h - library-internal structures shared by the host API
 * (pt_api.cu, bvh_build.cu) and the wavefront kernels (pt_kernels.cu).
 */
#ifndef PT_INTERNAL_H
#define PT_INTERNAL_H

#include <cuda_runtime.h>
#include <stdint.h>
#include "pt_types.h"

#ifndef PT_TRACE_BLOCK
#define PT_TRACE_BLOCK 128       /* default threads per trace block */
#endif
#ifndef PT_TRACE_MAXREG
#define PT_TRACE_MAXREG 72       /* registers per trace thread: 7 blocks of 128 per SM */
#endif
#define PT_SHADE_BLOCK 256       /* default and largest shade block */
/* Shading: 4 resident blocks of 256 threads (64 registers).  Consistent mode on
 * the 2.1 M-triangle terrain, 64 frames, with 2 / 3 / 4 / 5 / 6 / 7: 71.4 / 66.8 /
 * 64.9 / 65.6 / 66.0 / 67.6 ms (fewer registers spill, fewer blocks hide less
 * latency); guided 20.3 / 19.9 / 19.6 / 19.6 / 19.6 / 19.6 ms; reference mode is
 * 10 % slower at 5 on random spheres. */
#ifndef PT_SHADE_MINBLOCKS
#define PT_SHADE_MINBLOCKS 4
#endif
#define PT_TAIL_BLOCK 128        /* threads per block of the tail kernel */
/* Paths left in a chunk (live and not generated) that the tail kernel takes
 * over from the wavefront.  GB300, us per render with 0 (wavefront only) /
 * 8192 / 16384 / 32768 / 131072: Cornell box 500x500 1121 / 657 / 646 / 665 /
 * 805, 2.1 M camera paths on the spheres 2941 / 2025 / 2026 / 2014 / 2062,
 * terrain 1280x720 1481 / 1214 / 1124 / 1126 / 1129, textures (33 frames of
 * 321x243) 3510 / 3474 / 3524 / 3731 / 4519. */
#ifndef PT_TAIL_PATHS
#define PT_TAIL_PATHS 16384
#endif
/* The same where a material has a texture of any kind: a textured bounce can be
 * several times as long a chain of dependent loads, which a warp of one path
 * cannot hide.  GB300, us per render with 2048 / 4096 / 8192 / 16384: every
 * texture callable in one scene, 61x82, 3 frames 799 / 822 / 910 / 1157
 * (consistent mode 416 / 431 / 468 / 580), 321x243 one frame 1035 / 1053 / 1176 /
 * 1356 and 33 frames 2112 / 2121 / 2191 / 2287; 60x40 one frame 342 / 243 / 242 /
 * 245.  Where spheres have one simple texture the higher limit is the better one
 * for a frame or a few: 148 spheres, 61x82, 3 frames, constant 371 / 363 / 323 /
 * 271, checker 363 / 372 / 322 / 269, gradient 371 / 367 / 323 / 270, noise 389 /
 * 389 / 329 / 274, image 369 / 367 / 324 / 272; 33 frames of 321x243 within 2 %. */
#ifndef PT_TAIL_PATHS_TEX
#define PT_TAIL_PATHS_TEX 4096
#endif

/* Path state word st.z: depth (bits 0-15), previous bounce specular (bit 16),
 * scene of a batch (bits 17-31). */
#define PT_ST_DEPTH_MASK 0xffffu
#define PT_ST_SPEC_BIT 16
#define PT_ST_SCENE_SHIFT 17
#define PT_ST_KEEP_MASK 0xfffe0000u
#define PT_MAX_BATCH_SCENES 32767

/* Launch shape of the stage kernels. */
struct LaunchCfg {
  int trace_block, trace_grid;
  int shade_block, shade_grid;
  int sort;            /* shade in material order (by lists that the trace fills) */
  int refetch;         /* idle lanes of a trace warp that take new rays together (1..32) */
  int tex;             /* some material takes a texture: the texture variants of shading */
  int motion;          /* some sphere moves: the trace variants that carry ray times */
  int tail_grid;       /* blocks of the tail kernel: those resident at once */
  int one_grid;        /* the scene's tree is one node: blocks of its trace kernel, else 0 */
  int lights;          /* some scene has lights */
  int env;             /* some scene has an importance-sampled environment */
};

struct Ray3 {
  float3 o, d;
};

/* Counters of the streaming wavefront, in device memory. */
struct WaveCounters {
  uint32_t n_next;       /* paths written to the next buffer; with n_shadow one 64-bit word
                            for the appends that make both (push_both) */
  uint32_t n_shadow;     /* shadow rays queued this iteration */
  uint32_t n_cur;        /* live paths at the start of the current buffer (before generation) */
  uint32_t n_occ;        /* consistent mode: occlusion rays of the current buffer's paths */
  uint32_t n_wait, n_wait_next; /* paths of the current / next buffer that have ended but
                            for their NEE term */
  uint32_t parity;       /* which path buffer is current */
  uint32_t error;        /* bit 0: traversal stack overflow, bit 1: iteration bound reached */
  uint32_t iter;         /* iterations of the current chunk */
  unsigned long long next_path;   /* next path id of the chunk to generate */
  unsigned long long ext_rays, shadow_rays;
  unsigned long long node_fetches, prim_tests;
  unsigned long long iters_total; /* iterations over all chunks (batch) */
  uint32_t chunk;        /* current chunk of a batch */
  uint32_t n_chunks;     /* chunks of the batch (set by the host) */
  uint32_t ray_next[2];  /* rays taken by trace warps this iteration (extension, shadow) */
  uint32_t guide_rows;   /* positions listed for guide inference this iteration */
  uint32_t chunks_done;  /* chunks of this render that ended without an error */
  uint32_t drained;      /* iterations since the chunk's last path was generated, that one
                            included: every live path has bounced this often */
};

/* Per-chunk render controls, in device memory (kernels read them, so one
 * captured CUDA graph serves every chunk). */
struct WaveCtl {
  int width, height;
  int frame0;                     /* frame of path id 0 of this chunk */
  int max_depth, rr_enable, rr_depth, mode, guide;
  unsigned long long chunk_paths; /* paths in this chunk */
  uint32_t wh_m, wh_l, w_m, w_l;  /* invariant-divisor constants for W*H and W */
  /* batch: segments [seg_begin, seg_end) make up this chunk, `pixels` pixels */
  uint32_t seg_begin, seg_end, pixels;
  uint32_t guide_depth;           /* guided bounces: depth < guide_depth */
  uint32_t tail_max;              /* most paths left that the tail kernel takes over */
  unsigned long long max_iter;    /* device-side iteration bound of this chunk */
};

/* ---- batched multi-scene rendering ---------------------------------------
 * Every scene of a batch is copied into one set of geometry arrays (nodes,
 * records, transforms, materials, attributes) with its indices shifted, so
 * traversal needs only a per-ray root node.  Camera, miss program, lights
 * and environment tables stay per scene. */
struct BatchScene {
  DevScene S;          /* geometry pointers: the batch arrays; the rest: this scene's */
  int width, height, max_depth, rr_enable, rr_depth, pad;
  uint32_t wh_m, wh_l, w_m, w_l;
};

/* Consecutive frames of one scene inside a chunk. */
struct BatchSeg {
  uint32_t path_off;   /* first path of the segment, chunk-relative */
  uint32_t pix_off;    /* first pixel of the segment among the chunk's pixels */
  uint32_t scene;      /* index into the BatchScene table */
  uint32_t frame0, frames, pad;
  float4* acc;         /* device accumulator of the scene */
};

struct BatchChunk {
  unsigned long long paths, max_iter;
  uint32_t seg_begin, seg_end, pixels, pad;
};

/* Kernel-parameter view of a batch (null pointers for a single scene). */
struct BatchRefs {
  const BatchScene* scenes;
  const BatchSeg* segs;
  const uint32_t* roots;     /* root node per scene */
};

/* Unsigned division by an invariant 32-bit divisor d >= 1 (Granlund &
 * Montgomery 1994, "Division by invariant integers using multiplication",
 * fig. 4.1): l = ceil(log2 d), m = floor(2^32 (2^l - d) / d) + 1, then
 * n / d = (t + ((n - t) >> min(l,1))) >> max(l-1,0) with t = mulhi(m, n). */
static inline void fastdiv_magic(uint32_t d, uint32_t* m, uint32_t* l) {
  uint32_t ll = 0;
  while (ll < 32 && (1ull << ll) < d) ll++;
  *l = ll;
  *m = (uint32_t)((((1ull << 32) * ((1ull << ll) - d)) / d) + 1);
}
#ifdef __CUDACC__
__device__ __forceinline__ uint32_t fastdiv(uint32_t n, uint32_t m, uint32_t l) {
  uint32_t t = __umulhi(m, n);
  return (t + ((n - t) >> (l > 0 ? 1u : 0u))) >> (l > 0 ? l - 1 : 0u);
}
#endif

/* Path state, structure of arrays, stored in queue order: entry i of the
 * current buffer is the i-th live path of this iteration.  Paths that
 * continue are written compacted into the other buffer of the pair, so
 * every kernel reads and writes its arrays contiguously. */
struct PathBuf {
  float4 *ray_o, *ray_d;      /* origin+tmin, direction+tmax */
  float4 *thr, *rad;          /* throughput, radiance */
  uint4* st;                  /* seed, path id, depth|prevSpecular<<16 */
};

/* Reference mode: paths parked at a shadow ray (Direct_Light context: the
 * random stream after it depends on it), in shadow-queue order. */
struct ShadowBuf {
  float4 *P, *N, *Wo, *Wi;    /* P+light pdf, N+light index, Wo+material, Wi+occluded */
  float4* C;                  /* texture colour */
  float4 *thr, *rad;
  uint4* st;
};

/* Consistent mode: NEE terms of the paths of a buffer, by position.  The
 * continuation does not depend on the occlusion ray, so a path goes on at
 * once and adds its term when it is next shaded, after both its rays were
 * traced in one launch; a path that has ended waits one iteration for it
 * (ray_d.w = 0: no extension ray). */
struct NeeBuf {
  float4* Wi;                 /* direction + occluded */
  float4* C;                  /* term + tmax */
  uint32_t* queue;            /* positions of the paths with an occlusion ray */
};
#define PT_CODE_PENDING 8     /* rad.w of such a path: this + its guide-record word */

struct GuidePacked;
struct GuideSample;
struct GuideInferArgs;

struct WaveState {
  PathBuf path[2];            /* ping-pong: path[parity] is current */
  float4* hit;                /* t, u, v, leaf index: by position in the current buffer */
  uint32_t* lists;            /* sorted shading: `slots` positions for each shading key; else null */
  uint32_t* listed;           /* positions on list k: listed[k * PT_LISTED_STRIDE] */
  ShadowBuf sh;               /* reference mode */
  NeeBuf nee[2];              /* consistent mode, beside path[]; shares sh's memory */
  WaveCounters* ctr;
  float4* results;            /* per path of the chunk: colour */
  int slots;                  /* capacity of each buffer */
  /* learned guide (consistent mode, guide = 1): decoded guide by position;
   * training records, 2 per recording path (path id % grec_stride == 0) */
  GuidePacked* guide;
  GuideSample* grec;
  uint32_t grec_stride, grec_n;
};

/* float4 arrays per slot: 2 x 4 (path buffers) + 1 (hit) + 7 (shadow), and
 * uint4 arrays: 3 states. */
#define PT_SLOT_F4 16
#define PT_SLOT_U4 3
/* Shading key of a hit: 0 none, 1 + material type.  Each list's counter has a
 * cache line of its own, at the end of the uint4 block: the trace warps append
 * to all of them all the time.  The lists are memory of their own (32 bytes a
 * slot), which scenes shaded in path order do without. */
#define PT_SHADE_KEYS (PT_NUM_MAT_TYPES + 1)
#define PT_LISTED_STRIDE 32
#define PT_SLOTS_U4(s) ((size_t)(s) * PT_SLOT_U4 + PT_SHADE_KEYS * PT_LISTED_STRIDE / 4)
#define PT_SLOTS_LISTS(s) ((size_t)(s) * PT_SHADE_KEYS)

/* Ray kinds of the trace kernels: closest hit of extension rays; closest
 * hit of a shadow ray (reference mode: the light must be the first thing
 * hit); first-hit queries; any hit before tmax (consistent-mode occlusion);
 * extension rays, then occlusion rays. */
enum { TRACE_EXT = 0, TRACE_SHADOW = 1, TRACE_FIRST = 2, TRACE_OCCLUDED = 3, TRACE_BOTH = 4 };

namespace pt {
/* Dynamic shared memory of a trace block (pt_trace.cu). */
size_t trace_smem(int max_stack, int block);
/* Resident blocks per SM of the trace kernel for trees of one node. */
int one_blocks_per_sm();
/* Resident trace blocks per SM (0 if the shape does not fit). */
int trace_blocks_per_sm(int block, size_t smem);
/* One trace launch of `mode` (TRACE_EXT, TRACE_SHADOW or TRACE_BOTH)
 * over the wavefront's rays, with the launch shape of lc. */
void launch_trace(int mode, bool counters, const DevScene& S, const WaveState& W,
                  const WaveCtl* ctl, int max_stack, const BatchRefs* br, const LaunchCfg& lc,
                  cudaStream_t st);
/* WaveCtl.tail_max for a BVH of this stack depth and launch shape: the limit
 * (PT_TAIL_AUTO: PT_TAIL_PATHS, or PT_TAIL_PATHS_TEX where lc.tex), or 0 where
 * the tail kernel's stacks would not fit in shared memory. */
uint32_t tail_paths(int max_stack, const LaunchCfg& lc, uint32_t limit);
/* Resident tail blocks per SM (pt_tail.cu); batch: of its batch form. */
int tail_blocks_per_sm(int max_stack, bool batch);
/* Dynamic shared memory limit of the tail kernels (once per device). */
cudaError_t set_tail_smem();
/* The chunk's last paths, each to its end, when at most tail_max are left
 * (pt_tail.cu); mark: the counters then say that the chunk has drained. */
void launch_tail(const DevScene& S, const WaveState& W, const WaveCtl* ctl, int max_stack,
                 bool counters, const LaunchCfg& lc, int mode, const BatchRefs* br, bool mark,
                 cudaStream_t st);
/* Starts a chunk: *ctl = v, empty queues; first: the totals start at zero
 * too (else they go on, with the error flags). */
void launch_chunk_begin(const WaveState& W, WaveCtl* ctl, const WaveCtl& v, bool first,
                        cudaStream_t st);
/* Kernels of one iteration in `mode` (without a light or environment to
 * sample there are no shadow rays to trace or finish). */
int iteration_kernels(const LaunchCfg& lc, int mode, bool guide);
/* Resident blocks per SM x SMs for a trace (kind 0), shade (kind 1) or tail
 * (kind 2, of a batch 4, blocks of PT_TAIL_BLOCK) kernel of `block` threads, or
 * for the trace kernel of one-node trees (kind 3). */
int wave_grid(int kind, int max_stack, int block);
/* Raises the dynamic shared memory limit of the trace kernels to the
 * device maximum (once per device). */
cudaError_t set_trace_smem();
/* Default launch shape for a BVH of the given stack depth. */
LaunchCfg default_launch(int max_stack);
/* One wavefront iteration (iteration_kernels launches).  ev, if not null, holds 6 events
 * recorded between the stages.  br: batch tables, or null for one scene.
 * use_cond: the queue-advance kernel sets graph conditional `cond` to
 * whether the chunk has work left (device-side iteration loop).  gi: the
 * learned guide (consistent mode only): its inference kernel runs between
 * trace and shade (counted in the shade stage) and shading samples from it. */
void launch_iteration(const DevScene& S, const WaveState& W, const WaveCtl* ctl, int max_stack,
                      bool counters, const LaunchCfg& lc, cudaStream_t st, cudaEvent_t* ev,
                      int mode, const BatchRefs* br, bool use_cond,
                      unsigned long long cond, const GuideInferArgs* gi = nullptr);
/* Batch chunk boundaries: begin loads chunk c.chunk into *ctl and resets the
 * queues (and sets conditional `inner` to 1); end accumulates the chunk's
 * results into the scenes' accumulators, moves to the next chunk and sets
 * conditional `outer` to whether one is left. */
void launch_batch_begin(const WaveState& W, WaveCtl* ctl, const BatchChunk* chunks,
                        bool use_cond, unsigned long long inner, cudaStream_t st);
void launch_batch_end(const WaveState& W, const WaveCtl* ctl, const BatchRefs& br,
                      bool use_cond, unsigned long long outer, cudaStream_t st);
/* Adds offsets to the indices of one scene copied into the batch arrays. */
void launch_relocate(uint4* nodes, size_t n_nodes, uint32_t node_off, uint32_t prim_off,
                     float4* prims, size_t n_prims, uint32_t xform_off, uint32_t id_off,
                     uint32_t mat_off, uint32_t* leaf_of_id, uint4* tri_attr, uint32_t attr_off,
                     cudaStream_t st);
/* The importance-sampling tables of an environment (DevScene.env_*);
 * marg_idx null: without the search tables. */
void launch_env_cdf(const float4* env, int w, int h, float* marg, float* cond, double* rows,
                    double* pre, int* valid, float2* row, uint16_t* marg_idx, int marg_bits,
                    uint16_t* cond_idx, int cond_bits, cudaStream_t st);
/* Normals of 3 floats to 16-byte vectors. */
void launch_pack_normals(const float* n3, size_t n, float4* n4, cudaStream_t st);
/* The three below write nothing once W's error flags are set: the results of a
 * chunk that failed are not complete. */
void launch_accumulate(const WaveState& W, float4* acc, int w, int h, int frames, cudaStream_t st);
/* acc: 4 doubles per pixel (16-byte aligned) */
void launch_accumulate64(const WaveState& W, double* acc, int w, int h, int frames,
                         cudaStream_t st);
void launch_paths_out(const WaveState& W, float* out, uint32_t n, cudaStream_t st);
/* First hits of the camera rays of one frame. */
void launch_first_hits(const DevScene& S, int w, int h, int frame, uint32_t* prim, uint32_t* mat,
                       float* t, int max_stack, uint32_t* err, const LaunchCfg& lc,
                       cudaStream_t st);
void launch_resolve(const float4* acc, uchar4* out, int n, int frame, cudaStream_t st);
}  // namespace pt

#endif
