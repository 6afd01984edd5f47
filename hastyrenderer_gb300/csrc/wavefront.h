// Wavefront path state and kernel launch interface (host + device).
//
// One path slot per camera sample of a batch: slot = k * (W*H) + pixel for
// pass pass_base + k. State lives in HBM as arrays of 32-byte records, the
// fields that a kernel reads together; each bounce runs `trace` (closest hit of
// every queued ray) and `shade` (resolve the previous vertex's NEE and BSDF
// samples, shade the new vertex, emit its rays). Queues are compacted with warp
// ballots.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "hasty_types.h"

namespace hasty {

// flags word (w of the first half of a path's PathsDev::state record)
enum : uint32_t {
  PF_DEPTH_MASK = 0xFFu,          // depth of the vertex the pending BRDF ray leaves from
  PF_WL_SHIFT = 8,                // wavelength + 1 (0: not chosen yet)
  PF_WL_MASK = 0x3u << 8,
  PF_PEND_B = 1u << 14,           // BSDF-sampled ray queued in ray slot 2s
  PF_PEND_L = 1u << 15,           // light-sampled ray queued in ray slot 2s+1
  PF_CAMERA = 1u << 16,           // pending ray is the camera ray
  PF_NMED_SHIFT = 17,             // media on the stack (0..kMediaMax)
  PF_NMED_MASK = 0x1Fu << 17,
  PF_CHUNK_SHIFT = 24,            // packed batches: chunk of the path's job (0 otherwise); also
  PF_CHUNK_MASK = 0xFFu << 24,    // the bits of w of the path's ray origins
};
// Medium stack of a path (LightRayInfo's media, core/include/Hasty/LightRayInfo.h:51):
// the first kMaxMedia entries in the path's own slots; a path nested deeper
// takes one overflow block of kMediaBlock entries from the batch's pool
// (P.med_pool, P.counts[kMediaPoolCounter]), for kMediaMax entries in all.
// A push beyond that, or with the pool exhausted, is dropped and counted
// (ST_MEDIA_OVERFLOW).
constexpr int kMaxMedia = 4;
constexpr int kMediaBlock = 16;
constexpr int kMediaMax = kMaxMedia + kMediaBlock;
static_assert(kMediaMax < 32, "the stack depth has 5 bits in the flags");

// Fields that a kernel reads together share 32 bytes, one load or store of
// the GPU: a queue of surviving paths is sparse in slot order, so a 16-byte
// field alone would use half of each 32-byte sector it moves.
struct PathsDev {
  float4* state;        // 2 per path: xyz radiance gathered so far, w flags; x, y PCG32 state,
                        // z the path's overflow block in med_pool (-1: none), w unused
  float4* thr;          // 2 per path: xyz path throughput up to the pending BSDF sample, w its pdf;
                        // xyz BSDF-sample weight (f|cos|/pdf * RR/Beer of its vertex), w vertex triangle;
                        // between the resolve and the sample kernel the latter is the vertex's Beer/roulette factor
  float4* nee;          // 2 per path: xyz throughput * f * |cos| of the light sample, w BSDF pdf of its
                        // direction; xyz medium transmittance along the light ray, w sampled light triangle (-1: env)
  float4* med;          // 4 per path: medium transmittance xyz, IOR
  int32_t* med_geom;    // 4 per path: OBJ shape id of the medium
  float4* med_pool;     // overflow blocks: kMediaBlock entries each (transmittance, IOR)
  int32_t* med_pool_geom;
  int32_t med_pool_blocks;
  float4* ray;          // 2 per ray (2 rays per path): origin, w the path's chunk (bits); direction
  float4* hit;          // 1 per ray: t, u, v, triangle (-1 miss)
  int32_t* pq[2];       // path queues
  int32_t* rq[2];       // ray queues (ray ids 2s, 2s+1); once traced, queue q is the sample queue of its
                        // bounce (paths that continue past resolve)
  uint32_t* counts;     // [pq0, rq0, pq1, rq1, then kFetchCounter.. below]
  float4* out_color;    // per slot: final radiance of the sample
  float4* out_normal;
  float4* out_albedo;
  unsigned long long* stats;   // see StatIndex
  int32_t capacity;
};

#ifdef __CUDACC__
// Both halves of a 32-byte record (32-byte aligned), one load or store.
__device__ __forceinline__ float4 pair_half(unsigned long long x, unsigned long long y) {
  return make_float4(__uint_as_float(uint32_t(x)), __uint_as_float(uint32_t(x >> 32)), __uint_as_float(uint32_t(y)),
                     __uint_as_float(uint32_t(y >> 32)));
}
__device__ __forceinline__ unsigned long long pair_word(float lo, float hi) {
  return (unsigned long long)__float_as_uint(lo) | (unsigned long long)__float_as_uint(hi) << 32;
}
__device__ __forceinline__ void ld_pair(const float4* p, float4& a, float4& b) {
  const ulonglong4_32a v = *reinterpret_cast<const ulonglong4_32a*>(p);
  a = pair_half(v.x, v.y);
  b = pair_half(v.z, v.w);
}
__device__ __forceinline__ void st_pair(float4* p, float4 a, float4 b) {
  ulonglong4_32a v;
  v.x = pair_word(a.x, a.y); v.y = pair_word(a.z, a.w);
  v.z = pair_word(b.x, b.y); v.w = pair_word(b.z, b.w);
  *reinterpret_cast<ulonglong4_32a*>(p) = v;
}
#endif

// ST_STACK_OVERFLOW: rays whose traversal stack was full when a subtree had
// to be pushed (the subtree is skipped; the hit may then not be the closest).
enum StatIndex { ST_RAYS = 0, ST_SHADED, ST_PATHS, ST_NAN, ST_MEDIA_OVERFLOW, ST_TRIAL_CAP, ST_STACK_OVERFLOW, ST_COUNT };
constexpr int kCountSlots = 8;
// Lengths of path and ray queue q: neighbours, so that one 64-bit atomic
// reserves room in both.
constexpr __host__ __device__ int path_count(int q) { return 2 * q; }
constexpr __host__ __device__ int ray_count(int q) { return 2 * q + 1; }
constexpr int kFetchCounter = 4;   // counts[4]: rays handed out by the persistent trace kernels
constexpr int kSampleCount = 5;    // counts[5]: length of the sample queue
constexpr int kFinishTicket = 7;   // counts[7]: blocks of the finishing kernel that are done
constexpr int kMediaPoolCounter = 6;   // counts[6]: medium overflow blocks handed out in this batch

struct BatchDesc {
  uint64_t seed;
  uint32_t pass_base;
  int32_t n_passes;
  int32_t n_paths;      // n_passes * W * H
};

// Kernel launchers (integrator.cu / trace.cu). All launches go to `stream`.
void launch_raygen(const SceneDev& sc, const PathsDev& p, const BatchDesc& b, cudaStream_t stream);
// blocks_per_sm > 0 caps the persistent wide-BVH grid at that many resident
// blocks per SM (room for another stream's kernels); 0: all that fit.
void launch_trace(const SceneDev& sc, const PathsDev& p, int q, int max_rays, cudaStream_t stream, int blocks_per_sm = 0);
// True when sc's closest hits run one ray per thread instead of the
// persistent kernel: a wide BVH of at most simple_trace_nodes() nodes.
int simple_trace_nodes();
bool simple_trace_bvh(const SceneDev& sc);
void launch_shade(const SceneDev& sc, const PathsDev& p, const BatchDesc& b, int bounce, int max_paths, cudaStream_t stream);
void launch_accumulate(const SceneDev& sc, const PathsDev& p, const BatchDesc& b, double* acc_color, double* acc_normal,
                       double* acc_albedo, cudaStream_t stream);
// The shading records of a mesh (out: kTriRecord float4 per triangle).
void launch_tri_records(const MeshDev& mesh, float4* out, cudaStream_t stream);
// Replaces n cumulative probabilities (doubles) by their draw thresholds
// (cdf_threshold), in place.
void launch_cdf_thresholds(double* cdf, int64_t n, cudaStream_t stream);
void launch_estimate(const double* acc, int n, float den, float scale, float* out, cudaStream_t stream);

// Packed multi-job batches (batching and serving). A batch lays out chunks
// of consecutive passes of several jobs one after another in slot space:
// chunk c covers slots [first_slot, first_slot + n_passes * npix), slot
// first_slot + k * npix + px being pass pass_base + k of pixel px of its
// job. Every path carries its chunk index in its flags (PF_CHUNK_*) and its
// rays in the origin's w, so the kernels find the job's scene, seed and accumulators
// without a per-slot table. The tables travel as kernel parameters.
constexpr int kMaxChunks = 64;
struct ChunkDev {
  SceneDev sc;
  uint64_t seed;
  int32_t first_slot;
  uint32_t pass_base;
  int32_t npix;
  int32_t n_passes;
};
struct ChunkTable {
  int32_t n;            // chunks
  int32_t n_paths;      // slots of all chunks
  ChunkDev c[kMaxChunks];
};
// The closest-hit kernel's part of a chunk.
struct TraceChunk {
  const float4* nodes;
  const float4* tris;
  int32_t nee_first_hit;   // light rays stop at their first hit (environment-only lighting)
  int32_t n_nodes, n_tris; // sizes of nodes and tris (the bounds-checked build checks them)
  int32_t pad;
};
struct TraceTable {
  int32_t n;
  int32_t bvh_kind;     // of every chunk (a context's jobs share one BVH layout)
  TraceChunk c[kMaxChunks];
};
#ifdef __CUDACC__
// Kernels of a batch follow each other on their lane's stream, a few
// microseconds each near the batch's end. launch_dependent lets a kernel's
// blocks be placed while the one before flushes and ends; the kernel calls
// after_previous() before it touches memory, which waits for all of that one's
// work. (Letting the next kernel start once all blocks of this one run, with
// launch_dependents at the top, holds the other lane's places: 1080p field
// 28.4 -> 30.5 ms.) Plain launches / these, ms: 64k-triangle field 1.59 / 1.54,
// 256k-triangle field with 0.6M samples 0.601 / 0.554, stress scene 16.79 /
// 16.58, 1080p field 28.42 / 28.31, textured room 7.81 / 7.78, Cornell box
// 4.87 / 4.87.
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... P, class... A>
void launch_dependent(void (*kernel)(P...), int grid, int block, cudaStream_t st, const A&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(unsigned(block));
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}
#endif

static_assert(sizeof(ChunkTable) < 32000, "kernel parameters are limited to 32764 bytes");

void launch_raygen_packed(const ChunkTable& t, const PathsDev& p, cudaStream_t stream);
void launch_trace_packed(const TraceTable& t, const PathsDev& p, int q, int max_rays, cudaStream_t stream,
                         int blocks_per_sm = 0);
// resolve_threads 128 or 256, sample_threads 256 or 512 (block shapes; any
// other value takes 256 / 512).
void launch_shade_packed(const ChunkTable& t, const PathsDev& p, int bounce, int max_paths, cudaStream_t stream,
                         int resolve_threads = 256, int sample_threads = 512);
// Adds slots [first_slot, first_slot + n_passes * npix) (passes in order) into
// FP64 accumulators of npix pixels.
void launch_accumulate_range(const PathsDev& p, int first_slot, int npix, int n_passes, double* acc_color,
                             double* acc_normal, double* acc_albedo, cudaStream_t stream);

// Path kernel (scenes that stay in L1/L2): persistent threads, each carrying
// one camera sample through all its bounces in a slot of `slots` (path_slots()
// slots at least), finished samples written to `out`'s per-sample arrays
// (out_color/out_normal/out_albedo, indexed like a wavefront batch). Same
// samples as the wavefront kernels, bit for bit.
int64_t path_slots();
void launch_paths(const SceneDev& sc, const BatchDesc& b, const PathsDev& slots, const PathsDev& out, cudaStream_t stream);
void launch_paths_packed(const ChunkTable& t, int bvh_kind, const PathsDev& slots, const PathsDev& out,
                         cudaStream_t stream);

// Finishing small queues: the path kernel on a batch's own state. Carries the
// paths of queue q (before their closest hits of this bounce) to their ends
// if there are at most `limit`, leaving the queue empty; otherwise does nothing.
// Same samples, bit for bit.
// FinishLimits: the largest batch finished at bounce 0, with no other launch, and
// the most paths of a larger one that are; finish_check: whether to offer it at
// bounce `bounce`.
struct FinishLimits { int64_t at_once = 0, later = 0; };
FinishLimits finish_limits(const SceneDev& sc);
bool finish_check(int bounce, int max_depth, int64_t n_paths, const FinishLimits& l);
void launch_finish(const SceneDev& sc, const BatchDesc& b, const PathsDev& p, int q, int64_t limit, cudaStream_t stream);
void launch_finish_packed(const ChunkTable& t, int bvh_kind, const PathsDev& p, int q, int64_t limit, cudaStream_t stream);

// Closest hits of a caller's rays (6 floats each) and where they go, all in
// device memory.
struct RayLists { float* rays; int32_t* tri; float *t, *u, *v; };
void launch_trace_rays(const SceneDev& sc, const RayLists& q, int n, cudaStream_t stream);

// ---------------------------------------------------------------------------
// Multi-job engine (batching and serving). Many resident jobs share one pool
// of path slots. Work is a sequence of segments, each one pass of one job
// (W*H camera samples); camera samples are issued in global order through the
// segments into whatever slots are free, so the pool stays full until the
// last sample (path regeneration). The host appends segments between engine
// waves (serving interleaves the passes of the resident jobs this way).
// Finished samples are added to per-job int64 fixed-point accumulators
// (2^-32 units): integer addition is order-independent, so a job's image is
// bit-identical however it is mixed with other jobs.
constexpr double kFixedScale = 4294967296.0;   // 2^32

struct JobDev {
  SceneDev sc;
  unsigned long long* acc;     // [lane][9][npix] int64: colour, normal, albedo components (two's complement)
  unsigned long long* done;    // finished camera samples
  uint64_t seed;
  uint32_t npix;
  uint32_t lanes;              // a sample of pass p goes to lane p % lanes (spreads the atomics of small frames)
};

// One pass of one job: global samples [begin, begin + npix) of the job table
// entry `job`, pixel = global sample - begin.
struct SegDev {
  unsigned long long begin;
  int32_t job;
  uint32_t pass;
};

struct MultiDev {
  const JobDev* jobs;          // job table (entries are reused once a job has finished)
  const SegDev* segs;          // ring of segments, power-of-two capacity
  uint32_t seg_mask;
  const uint32_t* seg_window;  // [lo, hi): logical indices of the live segments (device-resident)
  uint4* slot_meta;            // per slot: job, pixel and pass of the path's camera sample, accumulator
                               // lane (one 16-byte load in the shading kernels)
  int32_t* free_slots;         // first slot of each free group (kGroup slots, no live path), ascending
                               // (rebuilt every iteration)
  uint8_t* flags;              // per slot: path lives on / BSDF ray queued / light ray queued
  uint32_t* block_sums;        // 3 per compaction block: counts, then exclusive offsets
  uint32_t* free_count;
  unsigned long long* next_sample;
  unsigned long long* total_samples;
  unsigned long long* regen_base;   // first global sample of the current regeneration
  uint32_t* ctl;               // kCtlWords: [0] queue parity, [1] regen count, [2] unused,
                               // [3] path-queue base, [4] ray-queue base, [5] iterations, [6] bound hit,
                               // [7] iteration at which the current wave ends, [8], [9] first and last
                               // segment (logical index) of the current regeneration
  uint32_t regen_below;        // regenerate only when fewer live paths than this
  uint32_t max_iter;           // iteration bound of one run (device-side loop guard)
};

constexpr int kCtlWords = 16;
constexpr int kGroup = 32;     // slots regenerated together (one warp); the engine's capacity is a multiple
static_assert(kGroup == 32, "a group is one warp of the compaction kernels");

enum MultiStat { MS_RAYS = ST_RAYS, MS_SHADED = ST_SHADED, MS_PATHS = ST_PATHS, MS_NAN = ST_NAN,
                 MS_MEDIA_OVERFLOW = ST_MEDIA_OVERFLOW, MS_TRIAL_CAP = ST_TRIAL_CAP, MS_SATURATED = ST_COUNT,
                 MS_COUNT };

// One engine iteration (regenerate, trace, shade, loop condition) launched
// into `stream`; `cond` is the CUDA-graph conditional handle of the enclosing
// while node (0 when launched without a graph).
void launch_multi_iteration(const PathsDev& p, const MultiDev& m, int capacity, int bvh_kind,
                            unsigned long long cond_handle, int use_cond, cudaStream_t stream, int trace_blocks_per_sm = 0);
void launch_multi_init(const PathsDev& p, const MultiDev& m, int capacity, cudaStream_t stream);
// Compaction blocks of an engine with `capacity` slots (3 block_sums entries each).
int compact_blocks(int capacity);
// Sums lanes 1.. of a job's fixed-point sums into lane 0 (integer adds:
// exact, so the result does not depend on the lane count).
void launch_fold_lanes(unsigned long long* acc, int npix, int lanes, cudaStream_t stream);
// Adds a finished job's fixed-point sums (lane 0) into FP64 accumulators (sum * 2^-32).
void launch_fixed_to_double(const unsigned long long* acc, int npix, double* c, double* n, double* a, cudaStream_t stream);
// trace.cu: closest hit of the queued rays of the multi-job engine.
void launch_trace_multi(const PathsDev& p, const MultiDev& m, int bvh_kind, int max_rays, cudaStream_t stream,
                        int blocks_per_sm = 0);

}  // namespace hasty
