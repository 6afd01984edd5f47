// C ABI of the GB300 path tracer (include/hasty_gpu.h): job lifecycle, device
// upload, batch orchestration and outputs. The pass loop replaces the
// reference's renderThread (core/src/PathTracing.cpp:98-160): instead of one
// CPU thread rendering whole 1-spp frames, a batch of passes is rendered as
// one wavefront of W*H*passes camera samples on the job's CUDA stream, and the
// per-sample results are folded into FP64 accumulators in pass order.
#include "hasty_gpu.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <string>
#include <sys/mman.h>
#include <sys/stat.h>
#include <system_error>
#include <thread>
#include <unistd.h>
#include <vector>

#include "bvh_build.h"
#include "job.h"
#include "image_out.h"
#include "scene_load.h"
#include "wavefront.h"

namespace hasty {
// integrator.cu
uint32_t bounds_status_integrator();
uint32_t bounds_status_trace();
uint32_t bounds_status_photon();
void launch_debug_bsdf(int which, const float* in, int n, const uint32_t* replay, int n_replay, float* out, cudaStream_t st);
// trace.cu
void host_trace_rays(int kind, const float4* nodes, const float4* tris, const float* rays, int64_t n, float4* hits);
}

using namespace hasty;

namespace hasty {
thread_local std::string g_error;
}

namespace {

}  // namespace

void hasty::carve_paths(PathsDev& p, int64_t cap, int n_stats, const std::function<void*(size_t)>& alloc,
                        unsigned long long* stats, int64_t media_blocks) {
  auto A = [&](size_t bytes) { return alloc(bytes); };
  p.capacity = int32_t(cap);
  size_t c = size_t(cap);
  p.state = static_cast<float4*>(A(2 * c * sizeof(float4)));
  p.thr = static_cast<float4*>(A(2 * c * sizeof(float4)));
  p.nee = static_cast<float4*>(A(2 * c * sizeof(float4)));
  p.med = static_cast<float4*>(A(c * kMaxMedia * sizeof(float4)));
  p.med_geom = static_cast<int32_t*>(A(c * kMaxMedia * sizeof(int32_t)));
  p.med_pool_blocks = int32_t(media_blocks > 0 ? media_blocks : std::max<int64_t>(64, cap / 4));
  p.med_pool = static_cast<float4*>(A(size_t(p.med_pool_blocks) * kMediaBlock * sizeof(float4)));
  p.med_pool_geom = static_cast<int32_t*>(A(size_t(p.med_pool_blocks) * kMediaBlock * sizeof(int32_t)));
  p.ray = static_cast<float4*>(A(4 * c * sizeof(float4)));
  p.hit = static_cast<float4*>(A(2 * c * sizeof(float4)));
  p.pq[0] = static_cast<int32_t*>(A(c * sizeof(int32_t)));
  p.pq[1] = static_cast<int32_t*>(A(c * sizeof(int32_t)));
  p.rq[0] = static_cast<int32_t*>(A(2 * c * sizeof(int32_t)));
  p.rq[1] = static_cast<int32_t*>(A(2 * c * sizeof(int32_t)));
  p.counts = static_cast<uint32_t*>(A(kCountSlots * sizeof(uint32_t)));
  p.out_color = static_cast<float4*>(A(c * sizeof(float4)));
  p.out_normal = static_cast<float4*>(A(c * sizeof(float4)));
  p.out_albedo = static_cast<float4*>(A(c * sizeof(float4)));
  p.stats = stats ? stats : static_cast<unsigned long long*>(A(size_t(n_stats) * sizeof(unsigned long long)));
}

void hasty::alloc_paths_into(PathsDev& p, int64_t cap, int n_stats, const std::function<void*(size_t)>& alloc, cudaStream_t st,
                             unsigned long long* stats) {
  carve_paths(p, cap, n_stats, alloc, stats);
  if (!stats) ck(cudaMemsetAsync(p.stats, 0, sizeof(unsigned long long) * size_t(n_stats), st), "memset stats");
  ck(cudaMemsetAsync(p.counts, 0, sizeof(uint32_t) * kCountSlots, st), "memset counts");
}

int64_t hasty::carved_bytes(int64_t cap, int n_stats, size_t align, size_t extra_blocks, size_t extra_bytes) {
  size_t used = 0;
  auto count = [&](size_t bytes) -> void* {
    used = ((used + align - 1) / align) * align + bytes;
    return reinterpret_cast<void*>(uintptr_t(align));   // never dereferenced
  };
  PathsDev p{};
  carve_paths(p, cap, n_stats, count, nullptr);
  for (size_t k = 0; k < extra_blocks; ++k) count(extra_bytes);
  return int64_t(used);
}

// Path-state buffers of the single-job path are allocated at the first
// render (jobs that only feed the multi-job engine never need them) and
// re-allocated when the paths-in-flight setting changes.
namespace {
// One block for all of p's buffers (an allocation each, for two lanes, took
// 1 ms of a job's first call).
void alloc_path_buffers(hasty_job& j, PathsDev& p, int64_t cap, unsigned long long* stats) {
  constexpr size_t kAlign = 256;
  uint8_t* next = j.alloc<uint8_t>(size_t(carved_bytes(cap, ST_COUNT, kAlign, 0, 0)));
  alloc_paths_into(p, cap, ST_COUNT, [&](size_t b) {
    void* at = next;
    next += (b + kAlign - 1) / kAlign * kAlign;
    return at;
  }, j.stream, stats);
}

// Frees the path buffers of p (not the statistics it points to).
void release_path_buffers(hasty_job& j, PathsDev& p) {
  j.release(p.state);                   // the block's first buffer
  unsigned long long* stats = p.stats;
  p = PathsDev{};
  p.stats = stats;
}
}  // namespace

void hasty::ensure_paths(hasty_job& j, int64_t need) {
  for (int k = 0; k < 2; ++k) {
    if (!j.lane_stream[k]) ck(cudaStreamCreateWithFlags(&j.lane_stream[k], cudaStreamNonBlocking), "lane stream");
    if (!j.lane_done[k]) ck(cudaEventCreateWithFlags(&j.lane_done[k], cudaEventDisableTiming), "lane event");
    if (!j.lane_free[k]) ck(cudaEventCreateWithFlags(&j.lane_free[k], cudaEventDisableTiming), "lane event");
  }
  if (!j.main_ready) ck(cudaEventCreateWithFlags(&j.main_ready, cudaEventDisableTiming), "lane event");
  // buffers grow to what a call needs, up to the paths-in-flight setting
  need = std::max<int64_t>(1, std::min(need, j.capacity));
  if (j.pd.state && j.pd.capacity >= need && j.pd.capacity <= j.capacity) return;
  ck(cudaStreamSynchronize(j.stream), "sync");
  for (cudaStream_t s : j.lane_stream) ck(cudaStreamSynchronize(s), "sync");
  release_path_buffers(j, j.pd);
  release_path_buffers(j, j.pd2);       // lane 1 is allocated again when next used
  unsigned long long* stats = j.pd.stats;
  alloc_path_buffers(j, j.pd, need, stats);
  j.lane_free_valid[0] = j.lane_free_valid[1] = false;
  j.lanes_wait_main = true;             // counters were cleared on `stream`
}

// Lane 1's path buffers, sharing lane 0's statistics.
void ensure_lane2(hasty_job& j) {
  if (j.pd2.state && j.pd2.capacity == j.pd.capacity) return;
  release_path_buffers(j, j.pd2);
  alloc_path_buffers(j, j.pd2, j.pd.capacity, j.pd.stats);
  j.lane_free_valid[1] = false;
  j.lanes_wait_main = true;
}

namespace {

// Host half of the upload: BVH and CDF guide tables (no device work).
void prepare_scene(hasty_job& j) {
  if (j.prep) return;
  HostScene& h = j.host;
  std::unique_ptr<hasty_job::Prepared> p(new hasty_job::Prepared());
  bool binary = (j.ctx->flags & HASTY_CTX_BINARY_BVH) != 0;
  bool on_host = (j.ctx->flags & HASTY_CTX_HOST_BVH) != 0;
  if (!on_host) ck(cudaSetDevice(j.ctx->device), "cudaSetDevice");
  if (binary) {
    if (on_host) build_bvh_binary(h.tri_pos.data(), h.n_tris(), 4, p->bvh);
    else build_bvh_binary_gpu(h.tri_pos.data(), h.n_tris(), 4, p->bvh);
    if (p->bvh.depth > 60) throw ApiError{HASTY_ERR_LOAD, "BVH deeper than the traversal stack (64)"};
  } else {
    if (on_host) build_bvh_wide(h.tri_pos.data(), h.n_tris(), p->bvh);
    else build_bvh_wide_gpu(h.tri_pos.data(), h.n_tris(), p->bvh);
    if (p->bvh.depth > 30) throw ApiError{HASTY_ERR_LOAD, "wide BVH deeper than the traversal stack (32)"};
  }
  p->binary = binary;
  p->light_guide = build_cdf_guide(h.light_cdf, p->light_guide_log2);
  p->env_guide = build_cdf_guide(h.env_cdf, p->env_guide_log2);
  j.prep = std::move(p);
}

// A job's scene arrays share one device block, carved in the order of use. The
// mesh arrays, which only live until the shading records are made of them, use
// the place of the arrays that come after the records, so that a load needs no
// more device memory than the scene keeps. They go there in slices where they
// are larger than those arrays (spheres: 98 bytes per triangle, in 101).
constexpr size_t kArenaAlign = 256;
struct Arena {
  uint8_t* base = nullptr;     // null: only counts
  size_t used = 0;
  template <class T>
  T* take(size_t n) {
    if (n == 0) return nullptr;
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += (n * sizeof(T) + kArenaAlign - 1) / kArenaAlign * kArenaAlign;
    return p;
  }
  // A host array's place in the block, and its copy there.
  template <class T>
  T* put(const std::vector<T>& v, cudaStream_t st) {
    T* p = take<T>(v.size());
    if (p) ck(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st), "upload");
    return p;
  }
};

constexpr int64_t kMeshSlice = 4096;     // triangles at a time, at least

// What all slices of the triangles refer to, and slice [first, first + n).
MeshDev put_mesh(const HostScene& h, Arena& a, cudaStream_t st) {
  MeshDev m{};
  m.normals = a.put(h.normals, st);
  m.texcoords = a.put(h.texcoords, st);
  m.n_texcoords = int64_t(h.texcoords.size());
  return m;
}
void put_slice(const HostScene& h, int64_t first, int64_t n, MeshDev& m, Arena& a, cudaStream_t st) {
  m.n_tris = int32_t(n);
  float* pos = a.take<float>(9 * size_t(n));
  TriAttr* attr = a.take<TriAttr>(size_t(n));
  m.tri_pos = pos;
  m.tri_attr = attr;
  if (!a.base || n == 0) return;
  ck(cudaMemcpyAsync(pos, &h.tri_pos[9 * size_t(first)], 9 * size_t(n) * sizeof(float), cudaMemcpyHostToDevice, st), "upload");
  ck(cudaMemcpyAsync(attr, &h.tri_attr[size_t(first)], size_t(n) * sizeof(TriAttr), cudaMemcpyHostToDevice, st), "upload");
}

// The shading records of all triangles, by slices through `room` bytes at `at`.
void put_records(const HostScene& h, float4* rec, uint8_t* at, size_t room, cudaStream_t st) {
  Arena a;
  a.base = at;
  MeshDev mesh = put_mesh(h, a, st);
  const size_t used = a.used;
  const int64_t n = int64_t(h.n_tris());
  constexpr size_t kTriBytes = 9 * sizeof(float) + sizeof(TriAttr);
  const int64_t fit = room > used + 2 * kArenaAlign ? int64_t((room - used - 2 * kArenaAlign) / kTriBytes) : 0;
  const int64_t slice = std::max(kMeshSlice, fit);
  for (int64_t first = 0; first < n; first += slice) {
    a.used = used;
    put_slice(h, first, std::min(slice, n - first), mesh, a, st);
    launch_tri_records(mesh, rec + kTriRecord * first, st);
  }
}
// Room that put_records needs at least.
size_t records_room(const HostScene& h) {
  Arena a;
  MeshDev m = put_mesh(h, a, nullptr);
  put_slice(h, 0, std::min<int64_t>(kMeshSlice, int64_t(h.n_tris())), m, a, nullptr);
  return a.used;
}

// The scene's arrays and tables; total: the block's bytes, 0 when only counting.
void put_scene(const HostScene& h, const hasty_job::Prepared& p, size_t total, Arena& a, SceneDev& s, cudaStream_t st) {
  float4* rec = a.take<float4>(size_t(kTriRecord) * h.n_tris());
  s.tri_rec = rec;
  if (a.base) put_records(h, rec, a.base + a.used, total - a.used, st);
  s.nodes = reinterpret_cast<const float4*>(a.put(p.bvh.nodes, st));
  s.isect_tris = reinterpret_cast<const float4*>(a.put(p.bvh.tris, st));
  s.mats = a.put(h.mats, st);
  s.textures = a.put(h.textures, st);
  s.tex_pool = a.put(h.tex_pool, st);
  s.tex_pool8 = a.put(h.tex_pool8, st);
  s.light_tris = a.put(h.light_tris, st);
  s.light_guide = a.put(p.light_guide, st);
  EnvDev& e = s.env;
  e.texels = a.put(h.env_texels, st);
  e.weights = a.put(h.env_weights, st);
  e.guide = a.put(p.env_guide, st);
  // the cumulative tables, as the thresholds the kernels draw with
  double* light_cdf = a.put(h.light_cdf, st);
  double* env_cdf = a.put(h.env_cdf, st);
  if (light_cdf) launch_cdf_thresholds(light_cdf, int64_t(h.light_cdf.size()), st);
  if (env_cdf) launch_cdf_thresholds(env_cdf, int64_t(h.env_cdf.size()), st);
  s.light_cdf = reinterpret_cast<const uint64_t*>(light_cdf);
  e.cdf = reinterpret_cast<const uint64_t*>(env_cdf);
}

// Device bytes of a prepared scene: what upload_scene allocates and keeps.
size_t scene_bytes(const HostScene& h, const hasty_job::Prepared& p) {
  Arena rec, all;
  rec.take<float4>(size_t(kTriRecord) * h.n_tris());
  SceneDev s{};
  put_scene(h, p, 0, all, s, nullptr);
  return std::max(all.used, rec.used + records_room(h));
}

void upload_scene(hasty_job& j) {
  prepare_scene(j);
  const auto u0 = std::chrono::steady_clock::now();
  HostScene& h = j.host;
  SceneDev& s = j.sd;
  hasty_job::Prepared& p = *j.prep;
  j.bvh_depth = p.bvh.depth; j.bvh_ms = p.bvh.build_ms; j.bvh_tree_ms = p.bvh.tree_ms;
  Arena scene;
  const size_t total = scene_bytes(h, p);
  scene.base = j.alloc<uint8_t>(total);
  put_scene(h, p, total, scene, s, j.stream);
  s.n_tris = int32_t(h.n_tris());
  s.bvh_kind = p.binary ? 0 : 1;
  s.n_nodes = int32_t(p.bvh.nodes.size() / (p.binary ? 16 : kWideNodeWords));
  s.n_mats = int32_t(h.mats.size());
  s.n_textures = int32_t(h.textures.size());
  s.n_light_tris = int32_t(h.light_tris.size());
  s.light_guide_log2 = p.light_guide_log2;
  s.light_pdf_area = h.light_tris.empty() ? 0.0f : 1.0f / h.total_light_area;
  EnvDev& e = s.env;
  e.is_texture = h.env_texture ? 1 : 0;
  for (int c = 0; c < 3; ++c) e.color[c] = h.bg[c];
  e.w = h.env_w; e.h = h.env_h;
  e.guide_log2 = p.env_guide_log2;
  e.value_sum = h.env_value_sum;
  s.cam = h.cam;
  const RenderSettingsH& st = h.settings;
  s.width = int32_t(st.width); s.height = int32_t(st.height);
  s.max_depth = st.max_depth; s.rr_start = st.roulette_start; s.rr_q = st.roulette_q;
  s.two_strategies = (h.has_light() && st.use_mis) ? 1 : 0;
  s.env_is_sampled = h.env_texture ? 1 : 0;
  s.p_surface = !h.env_texture ? 1.0f : (!h.light_tris.empty() ? 0.5f : 0.0f);   // Scene.cpp:545
  ck(cudaGetLastError(), "scene tables");
  ck(cudaStreamSynchronize(j.stream), "sync upload");   // the host arrays may be freed after this
  j.upload_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - u0).count();
  j.prep.reset();
}

void clear_accumulators(hasty_job& j) {
  size_t n = size_t(j.sd.width) * size_t(j.sd.height) * 3;
  for (double* a : j.acc) ck(cudaMemsetAsync(a, 0, n * sizeof(double), j.stream), "memset acc");
  ck(cudaMemsetAsync(j.pd.stats, 0, sizeof(unsigned long long) * ST_COUNT, j.stream), "memset stats");
  j.lanes_wait_main = true;
  j.samples_done = 0;
  j.kernel_ms = j.trace_ms = j.shade_ms = j.path_ms = 0.0;
  j.trace_launches = j.kernel_launches = j.path_launches = 0;
}

// Up to 16M camera samples in flight per render lane (about 7 GB of path
// state each, allocated as far as a call needs it): fewer, larger batches
// per call. 1080p, 8 passes per call, two lanes (M samples/s): 2M paths 777,
// 4M 848, 8M 884, 16.6M (all 8 passes in one batch) 896.
int64_t default_capacity(int64_t npix) {
  int64_t cap = int64_t(1) << 24;
  if (npix > cap) cap = npix;
  return (cap / npix) * npix;
}

// Whether a call that fits one batch is rendered as two, one per render lane:
// tracing, which is bound by instruction issue, then runs beside shading, which
// is bound by latency, for a second set of launches and of last bounces with
// few paths. One batch / two, ms: Cornell box (tiny BVH), depth 8, 0.26M
// samples 0.54 / 0.64, 0.5M 0.83 / 0.72, 1M 1.40 / 1.26, 4.2M 5.06 / 4.78, depth
// 2, 1M 0.60 / 0.57, 16.8M 8.78 / 8.68, depth 32, 1M 2.00 / 2.00, 4.2M 5.88 /
// 5.63. Up to depth 9, 2.1M and 4.2M samples: textured room 1.98 / 1.96 and 3.53
// / 3.38, 64k-triangle field 1.00 / 0.99 and 1.64 / 1.61, 128k-triangle field at
// depth 6 1.08 / 1.06 and 1.79 / 1.73, 52k-triangle stress scene at depth 8 4.23 /
// 4.17 and 7.91 / 7.71. At depths 10 to 12, 3.1M and 6.3M: room 2.82 / 2.93 and
// 5.17 / 5.06, stress scene 6.51 / 6.68 and 12.15 / 11.83, but lit by the sky
// alone, 64k-triangle field 1.37 / 1.34 and 2.30 / 2.30, 128k 1.49 / 1.44. Deeper,
// room at 16, 4.9M 4.78 / 4.93, and of larger trees, 1.02M-triangle field 2M 2.47 /
// 2.72, 5.2M 5.19 / 5.29 (the two lanes' tracing shares the L2), stress scene at
// depth 32, 2M 4.75 / 5.08.
bool worth_two_batches(const hasty_job& j, int64_t samples) {
  if (simple_trace_bvh(j.sd)) return samples >= int64_t(1) << 20;
  const int64_t least = int64_t(j.sd.max_depth <= 9 || j.sd.n_light_tris == 0 ? 2 : 6) << 20;
  return samples >= least && j.sd.max_depth <= 12 && j.sd.n_tris <= 1 << 17;
}

// Passes per batch of a call: at most the paths in flight, the batches of one
// size and, where there are several, as many on one lane as on the other.
int passes_per_batch(const hasty_job& j, int n_passes) {
  const int64_t npix = int64_t(j.sd.width) * j.sd.height;
  const int64_t most = std::max<int64_t>(1, j.capacity / npix), n = n_passes;
  if (j.stage_timing || j.path_kernel) return int(std::min(most, n));
  int64_t batches = (n + most - 1) / most;
  if (batches == 1 ? n > 1 && worth_two_batches(j, n * npix) : batches % 2 == 1) ++batches;
  return int((n + batches - 1) / batches);
}

// Resident blocks per SM of the persistent closest-hit kernel while two
// render lanes run: fewer than fit (8 on GB300) leaves room for the other
// lane's shading blocks. ms at 3 / 4 / 5 / 6 / 7 / all: 1080p field of 1.02M
// triangles 30.39 / 28.31 / 28.08 / 28.24 / 28.34 / 28.17, textured room 8.22 /
// 7.90 / 7.90 / 7.92 / 7.94 / 7.93; the stress scene and the Cornell box (whose
// closest hits run one ray per thread) are level.
constexpr int kLaneTraceBlocksPerSM = 5;
}  // namespace

// Largest scene the path kernel takes by default: none. Measured on GB300
// (ms, path kernel / default): Cornell box 256x256, 16 passes 1.84 / 1.28;
// 64k-triangle field 512x512, 8 passes 1.44 / 1.03; textured room 640x480, 8
// passes 4.04 / 2.28; a 100x80 field, 4 passes, which the same kernel finishes
// on the batch's state, 0.15 both. Its path state stays in L2, but the
// wavefront's shading kernels are bound by load latency, not by their traffic,
// and the path kernel loses more to idle lanes, block barriers and undivided
// traversal than it saves. HASTY_PATH_KERNEL_TRIS (or HASTY_CTX_PATH_KERNEL)
// selects it.
constexpr int64_t kPathKernelMaxTris = 0;

int64_t hasty::path_kernel_max_triangles() {
  static const int64_t v = [] {
    const char* e = std::getenv("HASTY_PATH_KERNEL_TRIS");
    return e ? std::max<int64_t>(0, std::atoll(e)) : kPathKernelMaxTris;
  }();
  return v;
}

bool hasty::may_use_path_kernel(const hasty_ctx* ctx) {
  return !(ctx->flags & HASTY_CTX_WAVEFRONT) && ((ctx->flags & HASTY_CTX_PATH_KERNEL) || path_kernel_max_triangles() > 0);
}

bool hasty::use_path_kernel(const hasty_ctx* ctx, const SceneDev& sc) {
  if (sc.max_depth <= 0 || !may_use_path_kernel(ctx)) return false;
  return (ctx->flags & HASTY_CTX_PATH_KERNEL) || int64_t(sc.n_tris) <= path_kernel_max_triangles();
}

void hasty::alloc_path_slots(PathsDev& p, const std::function<void*(size_t)>& alloc, unsigned long long* stats) {
  // a slot keeps its overflow block for all the paths it carries in a launch
  const int64_t n = path_slots();
  carve_paths(p, n, ST_COUNT, alloc, stats, std::max<int64_t>(64, n / 2));
}

// HASTY_LANE_TRACE_BLOCKS overrides it (0: no cap).
int hasty::lane_trace_blocks() {
  static const int v = [] {
    const char* e = std::getenv("HASTY_LANE_TRACE_BLOCKS");
    return e ? std::max(0, std::atoi(e)) : kLaneTraceBlocksPerSM;
  }();
  return v;
}

namespace {

// One batch of passes on render lane `lane` (the two lanes alternate; see
// hasty_job): ray generation and the bounces on the lane's stream, then the
// accumulation on the job's stream.
void render_batch(hasty_job& j, int n_passes, int lane, bool more_batches) {
  BatchDesc b;
  b.seed = j.seed;
  b.pass_base = uint32_t(j.samples_done);
  b.n_passes = n_passes;
  b.n_paths = n_passes * j.sd.width * j.sd.height;
  PathsDev& pd = lane ? j.pd2 : j.pd;
  cudaStream_t ls = j.lane_stream[lane];
  // cap the trace grid only while the other lane has work to overlap
  bool other_busy = more_batches;
  if (!other_busy && j.lane_free_valid[lane ^ 1]) {
    const cudaError_t qs = cudaEventQuery(j.lane_done[lane ^ 1]);
    if (qs == cudaErrorNotReady) {
      other_busy = true;
      (void)cudaGetLastError();        // "not ready" is an answer, not an error to report later
    }
  }
  const int trace_cap = (j.stage_timing || !other_busy) ? 0 : lane_trace_blocks();
  if (j.lane_free_valid[lane]) ck(cudaStreamWaitEvent(ls, j.lane_free[lane], 0), "lane wait");
  auto timed = [&](int stage, auto&& fn) {
    if (!j.stage_timing) { fn(); return; }
    cudaEvent_t a, c;
    ck(cudaEventCreate(&a), "event"); ck(cudaEventCreate(&c), "event");
    ck(cudaEventRecord(a, ls), "event record");
    fn();
    ck(cudaEventRecord(c, ls), "event record");
    j.pending_events.push_back({a, c, stage});
  };
  uint64_t launches = 2;              // path kernel: it and the accumulation
  if (j.path_kernel) {
    PathsDev& slots = j.slots[lane];
    if (!slots.state) {
      alloc_path_slots(slots, [&](size_t bytes) { return static_cast<void*>(j.alloc<uint8_t>(bytes)); }, j.pd.stats);
      ck(cudaMemsetAsync(slots.counts, 0, sizeof(uint32_t) * kCountSlots, ls), "memset counts");
    }
    timed(3, [&] { launch_paths(j.sd, b, slots, pd, ls); });
    j.path_launches += 1;
  } else {
    // Stage timing measures the wavefront's stages, so it leaves the
    // finishing of small queues out.
    const bool finish = !(j.ctx->flags & HASTY_CTX_WAVEFRONT) && !j.stage_timing && j.sd.max_depth > 0;
    const FinishLimits limits = finish ? finish_limits(j.sd) : FinishLimits{};
    launch_raygen(j.sd, pd, b, ls);
    launches = 2;                     // with the accumulation
    const int max_paths = b.n_paths;
    if (max_paths <= limits.at_once) {
      launch_finish(j.sd, b, pd, 0, limits.at_once, ls);
      ++launches;
    } else {
      for (int bounce = 0; bounce < j.sd.max_depth; ++bounce) {
        int q = bounce & 1;
        if (finish && finish_check(bounce, j.sd.max_depth, max_paths, limits)) {
          launch_finish(j.sd, b, pd, q, limits.later, ls);
          ++launches;
        }
        timed(1, [&] { launch_trace(j.sd, pd, q, 2 * max_paths, ls, trace_cap); });
        timed(2, [&] { launch_shade(j.sd, pd, b, bounce, max_paths, ls); });
        launches += 3;
      }
      j.trace_launches += uint64_t(j.sd.max_depth);
    }
  }
  ck(cudaEventRecord(j.lane_done[lane], ls), "lane event");
  ck(cudaStreamWaitEvent(j.stream, j.lane_done[lane], 0), "lane wait");
  launch_accumulate(j.sd, pd, b, j.acc[0], j.acc[1], j.acc[2], j.stream);
  ck(cudaGetLastError(), "kernel launch");
  ck(cudaEventRecord(j.lane_free[lane], j.stream), "lane event");
  j.lane_free_valid[lane] = true;
  j.kernel_launches += launches;
  j.samples_done += n_passes;
}

hasty_job* as_job(hasty_job* j) {
  if (!j) throw ApiError{HASTY_ERR_ARG, "null job handle"};
  return j;
}

constexpr size_t kShortRays = size_t(1) << 14;

// Has the system provide the pages of a caller's buffer that were never touched.
// Where the copy to a partly touched buffer is left to fault for them, the device
// waits some 65 us for each (64 KB pages): a new job's first full-HD image, in
// heap memory that its load had half used, took 5 to 19 ms to read in a third of
// the calls; the host's faults take 0.4 to 1 ms, a buffer with all its pages 0.02
// to 0.1. The contents stay as they are, and where the system declines, the copy
// goes on as before.
void provide_pages(void* buffer, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
  if (bytes < size_t(1) << 20) return;
  const uintptr_t page = uintptr_t(sysconf(_SC_PAGESIZE)), first = uintptr_t(buffer) & ~(page - 1);
  madvise(reinterpret_cast<void*>(first), uintptr_t(buffer) + bytes - first, MADV_POPULATE_WRITE);
#else
  (void)buffer; (void)bytes;
#endif
}

// Room for `rays` rays in list k (and, for the second one, its stream).
void ray_list(hasty_job& j, int k, size_t rays) {
  if (k == 1 && !j.ray_stream) {
    ck(cudaStreamCreateWithFlags(&j.ray_stream, cudaStreamNonBlocking), "ray stream");
    ck(cudaEventCreateWithFlags(&j.ray_ready, cudaEventDisableTiming), "ray event");
  }
  if (rays <= j.ray_cap[k]) return;
  const size_t cap = (rays + 63) / 64 * 64;
  hasty::RayLists& l = j.ray_lists[k];
  constexpr size_t kRayBytes = 10 * sizeof(float);
  if (l.rays) cudaFree(l.rays);
  l = {};
  j.ray_bytes -= int64_t(j.ray_cap[k] * kRayBytes);
  j.ray_cap[k] = 0;
  float* p = nullptr;
  ck(cudaMalloc(&p, cap * kRayBytes), "cudaMalloc rays");
  j.ray_bytes += int64_t(cap * kRayBytes);
  l = {p, reinterpret_cast<int32_t*>(p + 6 * cap), p + 7 * cap, p + 8 * cap, p + 9 * cap};
  j.ray_cap[k] = cap;
}

}  // namespace

std::unique_ptr<hasty_job> hasty::load_job_host(hasty_ctx* ctx, const std::string& path) {
  std::unique_ptr<hasty_job> j(new hasty_job());
  j->ctx = ctx;
  const auto t0 = std::chrono::steady_clock::now();
  load_render_job(path, j->host);
  j->parse_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  j->seed = j->host.settings.seed;
  return j;
}

void hasty::finish_job_load(hasty_job& job, bool plain) {
  hasty_job* j = &job;
  ck(cudaSetDevice(j->ctx->device), "cudaSetDevice");
  ck(cudaStreamCreateWithFlags(&j->stream, cudaStreamNonBlocking), "stream");
  upload_scene(*j);
  j->path_kernel = use_path_kernel(j->ctx, j->sd);
  int64_t npix = int64_t(j->sd.width) * j->sd.height;
  j->capacity = default_capacity(npix);
  if (plain) {
    j->pd.stats = j->alloc<unsigned long long>(ST_COUNT);
    for (double*& a : j->acc) a = j->alloc<double>(size_t(npix) * 3);
    j->est = j->alloc<float>(size_t(npix) * 3);
    clear_accumulators(*j);
  }
  ck(cudaStreamSynchronize(j->stream), "sync");
  // the host copies of the large arrays are not needed after upload
  std::vector<float>().swap(j->host.tri_pos);
  std::vector<float>().swap(j->host.env_texels);
  std::vector<float>().swap(j->host.tex_pool);
  std::vector<uint8_t>().swap(j->host.tex_pool8);
}

std::unique_ptr<hasty_job> hasty::load_job(hasty_ctx* ctx, const std::string& path, bool plain) {
  std::unique_ptr<hasty_job> j = load_job_host(ctx, path);
  finish_job_load(*j, plain);
  return j;
}

int64_t hasty::prepare_job_upload(hasty_job& j) {
  prepare_scene(j);
  return int64_t(scene_bytes(j.host, *j.prep));
}

extern "C" {

int hasty_last_error(char* buf, size_t len) {
  if (!buf || len == 0) return HASTY_ERR_ARG;
  std::strncpy(buf, g_error.c_str(), len - 1);
  buf[len - 1] = 0;
  return HASTY_OK;
}

int hasty_version(int* major, int* minor) {
  if (major) *major = 0;
  if (minor) *minor = 1;
  return HASTY_OK;
}

int hasty_ctx_create(int device, uint32_t flags, hasty_ctx** out) {
  return guarded([&] {
    if (!out) throw ApiError{HASTY_ERR_ARG, "null output pointer"};
    int n = 0;
    ck(cudaGetDeviceCount(&n), "cudaGetDeviceCount");
    if (device < 0 || device >= n) throw ApiError{HASTY_ERR_ARG, "no CUDA device " + std::to_string(device)};
    ck(cudaSetDevice(device), "cudaSetDevice");
    auto* c = new hasty_ctx();
    c->device = device;
    c->flags = flags;
    ck(cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, device), "attr");
    *out = c;
    return HASTY_OK;
  });
}

int hasty_ctx_destroy(hasty_ctx* ctx) { delete ctx; return HASTY_OK; }

int hasty_job_load(hasty_ctx* ctx, const char* path, hasty_job** out) {
  return guarded([&] {
    if (!ctx || !path || !out) throw ApiError{HASTY_ERR_ARG, "null argument"};
    *out = load_job(ctx, path, true).release();
    return HASTY_OK;
  });
}

int hasty_jobs_load(hasty_ctx* ctx, const char* const* paths, size_t n, int32_t threads, hasty_job** out) {
  return guarded([&] {
    if (!ctx || (n && (!paths || !out))) throw ApiError{HASTY_ERR_ARG, "null argument"};
    for (size_t i = 0; i < n; ++i) {
      if (!paths[i]) throw ApiError{HASTY_ERR_ARG, "null path"};
      out[i] = nullptr;
    }
    std::vector<std::unique_ptr<hasty_job>> jobs(n);
    std::atomic<size_t> next{0};
    std::atomic<bool> failed{false};
    std::mutex mu;
    std::exception_ptr first;   // the failure of the lowest-numbered failing job
    size_t first_i = n;
    auto worker = [&] {
      cudaSetDevice(ctx->device);
      for (;;) {
        const size_t i = next.fetch_add(1);
        if (i >= n || failed.load()) return;
        try {
          jobs[i] = load_job(ctx, paths[i], true);
        } catch (...) {
          std::lock_guard<std::mutex> lk(mu);
          if (i < first_i) { first_i = i; first = std::current_exception(); }
          failed = true;
        }
      }
    };
    size_t nt = threads > 0 ? size_t(threads) : size_t(std::max(1u, std::thread::hardware_concurrency()));
    nt = std::max<size_t>(1, std::min(nt, n));
    std::vector<std::thread> pool;
    for (size_t k = 1; k < nt; ++k) {
      try {
        pool.emplace_back(worker);
      } catch (const std::system_error&) {
        break;   // fewer threads: the ones running (and this one) take the rest
      }
    }
    worker();
    for (std::thread& t : pool) t.join();
    if (first) std::rethrow_exception(first);   // the loaded jobs are freed with `jobs`
    for (size_t i = 0; i < n; ++i) out[i] = jobs[i].release();
    return HASTY_OK;
  });
}

int hasty_job_destroy(hasty_job* job) { delete job; return HASTY_OK; }

int hasty_job_info_get(hasty_job* job, hasty_job_info* out) {
  return guarded([&] {
    as_job(job);
    if (!out) throw ApiError{HASTY_ERR_ARG, "null output"};
    const HostScene& h = job->host;
    out->width = int32_t(h.settings.width); out->height = int32_t(h.settings.height);
    out->num_samples = h.settings.num_samples; out->max_depth = h.settings.max_depth;
    out->roulette_start_depth = h.settings.roulette_start; out->roulette_q = h.settings.roulette_q;
    out->use_mis = h.settings.use_mis ? 1 : 0; out->seed = job->seed;
    out->n_triangles = int64_t(h.tri_attr.size()); out->n_light_triangles = int64_t(h.light_tris.size());
    out->n_shapes = int32_t(h.n_shapes); out->n_materials = int32_t(h.mats.size());
    out->env_is_texture = h.env_texture ? 1 : 0; out->exposure = h.cam.exposure;
    out->samples_done = job->samples_done; out->bvh_depth = job->bvh_depth; out->bvh_build_ms = job->bvh_ms;
    out->device_bytes = job->bytes + job->ray_bytes;
    out->bvh_tree_ms = job->bvh_tree_ms;
    out->parse_ms = job->parse_ms;
    out->upload_ms = job->upload_ms;
    out->paths_in_flight = job->capacity;
    out->path_kernel = job->path_kernel ? 1 : 0;
    return HASTY_OK;
  });
}

int hasty_job_reset(hasty_job* job) {
  return guarded([&] {
    as_job(job);
    ck(cudaStreamSynchronize(job->stream), "sync");
    job->collect_events();
    clear_accumulators(*job);
    job->stop = false;
    ck(cudaStreamSynchronize(job->stream), "sync");
    return HASTY_OK;
  });
}

int hasty_job_set_seed(hasty_job* job, uint64_t seed) {
  int rc = hasty_job_reset(job);
  if (rc == HASTY_OK) job->seed = seed;
  return rc;
}

int hasty_job_set_paths_in_flight(hasty_job* job, int64_t paths) {
  return guarded([&] {
    as_job(job);
    int64_t npix = int64_t(job->sd.width) * job->sd.height;
    int64_t cap = paths <= 0 ? default_capacity(npix) : std::max<int64_t>(npix, (paths / npix) * npix);
    if (cap > int64_t(INT32_MAX) / 2) throw ApiError{HASTY_ERR_ARG, "too many paths in flight"};
    job->capacity = cap;   // the path buffers follow at the next render
    return HASTY_OK;
  });
}

int hasty_job_release_paths(hasty_job* job) {
  return guarded([&] {
    as_job(job);
    ck(cudaSetDevice(job->ctx->device), "cudaSetDevice");
    ck(cudaStreamSynchronize(job->stream), "sync");
    job->collect_events();
    release_path_buffers(*job, job->pd);
    release_path_buffers(*job, job->pd2);
    job->lane_free_valid[0] = job->lane_free_valid[1] = false;
    return HASTY_OK;
  });
}

int hasty_job_render_passes(hasty_job* job, int n_passes) {
  return guarded([&] {
    as_job(job);
    if (n_passes < 0) throw ApiError{HASTY_ERR_ARG, "negative pass count"};
    ck(cudaSetDevice(job->ctx->device), "cudaSetDevice");
    if (!job->pd.stats) throw ApiError{HASTY_ERR_ARG, "job was loaded for the multi-job engine only"};
    int64_t npix = int64_t(job->sd.width) * job->sd.height;
    if (n_passes == 0) return HASTY_OK;
    const int per_batch = passes_per_batch(*job, n_passes);
    ensure_paths(*job, per_batch * npix);
    int left = n_passes;
    // Device time of this call: from its first launch to its last
    // accumulation (consecutive calls chain on `stream`, so overlapped
    // batches are counted once).
    cudaEvent_t e0, e1;
    ck(cudaEventCreate(&e0), "event"); ck(cudaEventCreate(&e1), "event");
    ck(cudaEventRecord(e0, job->stream), "event record");
    if (job->lanes_wait_main) {
      ck(cudaEventRecord(job->main_ready, job->stream), "lane event");
      for (cudaStream_t ls : job->lane_stream) ck(cudaStreamWaitEvent(ls, job->main_ready, 0), "lane wait");
      job->lanes_wait_main = false;
    }
    while (left > 0) {
      if (job->stop.load()) break;
      int k = std::min(left, per_batch);
      // stage timing keeps one lane, so per-kernel times are not shared
      int lane = job->stage_timing ? 0 : job->next_lane;
      if (lane == 1) ensure_lane2(*job);
      if (job->lanes_wait_main) {          // lane 1 was just allocated on `stream`
        ck(cudaEventRecord(job->main_ready, job->stream), "lane event");
        ck(cudaStreamWaitEvent(job->lane_stream[1], job->main_ready, 0), "lane wait");
        job->lanes_wait_main = false;
      }
      render_batch(*job, k, lane, left > k);
      job->next_lane = lane ^ 1;
      left -= k;
    }
    ck(cudaEventRecord(e1, job->stream), "event record");
    job->pending_events.push_back({e0, e1, 0});
    if (job->stop.load()) throw ApiError{HASTY_ERR_STOPPED, "job stopped"};
    return HASTY_OK;
  });
}

int hasty_job_sync(hasty_job* job) {
  return guarded([&] {
    as_job(job);
    ck(cudaStreamSynchronize(job->stream), "cudaStreamSynchronize");
    job->collect_events();
    return HASTY_OK;
  });
}

int hasty_job_stop(hasty_job* job) {
  if (!job) return fail(HASTY_ERR_ARG, "null job handle");
  job->stop = true;
  return HASTY_OK;
}

int hasty_job_set_stage_timing(hasty_job* job, int on) {
  if (!job) return fail(HASTY_ERR_ARG, "null job handle");
  job->stage_timing = on != 0;
  return HASTY_OK;
}

int hasty_job_stats_get(hasty_job* job, hasty_stats* out) {
  return guarded([&] {
    as_job(job);
    if (!out) throw ApiError{HASTY_ERR_ARG, "null output"};
    ck(cudaStreamSynchronize(job->stream), "sync");
    job->collect_events();
    unsigned long long s[ST_COUNT];
    ck(cudaMemcpy(s, job->pd.stats, sizeof(s), cudaMemcpyDeviceToHost), "copy stats");
    out->rays = s[ST_RAYS]; out->shaded = s[ST_SHADED]; out->paths = s[ST_PATHS]; out->nan_samples = s[ST_NAN];
    out->media_overflow = s[ST_MEDIA_OVERFLOW]; out->trial_cap = s[ST_TRIAL_CAP];
    out->stack_overflow = s[ST_STACK_OVERFLOW];
    out->kernel_ms = job->kernel_ms;
    out->trace_ms = job->trace_ms; out->shade_ms = job->shade_ms;
    out->trace_launches = job->trace_launches; out->kernel_launches = job->kernel_launches;
    out->path_ms = job->path_ms; out->path_launches = job->path_launches;
    return HASTY_OK;
  });
}

int hasty_job_read_sums(hasty_job* job, int aov, double* host, size_t w, size_t h, int32_t* num_samples) {
  return guarded([&] {
    as_job(job);
    if (aov < 0 || aov > 2 || !host) throw ApiError{HASTY_ERR_ARG, "bad aov or buffer"};
    if (w != size_t(job->sd.width) || h != size_t(job->sd.height)) throw ApiError{HASTY_ERR_ARG, "buffer size does not match the frame"};
    ck(cudaStreamSynchronize(job->stream), "sync");
    job->collect_events();
    ck(cudaMemcpy(host, job->acc[aov], w * h * 3 * sizeof(double), cudaMemcpyDeviceToHost), "copy sums");
    if (num_samples) *num_samples = job->samples_done;
    return HASTY_OK;
  });
}

int hasty_job_read(hasty_job* job, int aov, float* host, size_t w, size_t h, int32_t* num_samples) {
  return guarded([&] {
    as_job(job);
    if (aov < 0 || aov > 2 || !host) throw ApiError{HASTY_ERR_ARG, "bad aov or buffer"};
    if (w != size_t(job->sd.width) || h != size_t(job->sd.height)) throw ApiError{HASTY_ERR_ARG, "buffer size does not match the frame"};
    int n = int(w * h * 3);
    float den = 1e-7f + float(job->samples_done);
    float scale = aov == HASTY_AOV_COLOR ? std::pow(2.0f, job->host.cam.exposure) : 1.0f;
    launch_estimate(job->acc[aov], n, den, scale, job->est, job->stream);
    ck(cudaGetLastError(), "estimate launch");
    provide_pages(host, size_t(n) * sizeof(float));       // while the passes are still rendered
    ck(cudaMemcpyAsync(host, job->est, size_t(n) * sizeof(float), cudaMemcpyDeviceToHost, job->stream), "copy estimate");
    ck(cudaStreamSynchronize(job->stream), "sync");
    job->collect_events();
    if (num_samples) *num_samples = job->samples_done;
    return HASTY_OK;
  });
}

int hasty_job_write_outputs(hasty_job* job, const char* out_dir, int write_pfm) {
  return guarded([&] {
    as_job(job);
    if (!out_dir) throw ApiError{HASTY_ERR_ARG, "null directory"};
    struct stat sb;
    if (stat(out_dir, &sb) != 0 || !S_ISDIR(sb.st_mode)) throw ApiError{HASTY_ERR_IO, std::string("not a directory: ") + out_dir};
    size_t w = size_t(job->sd.width), h = size_t(job->sd.height);
    std::vector<float> img(w * h * 3);
    const char* names[3] = {"output", "outputNormal", "outputAlbedo"};
    for (int a = 0; a < 3; ++a) {
      int rc = hasty_job_read(job, a, img.data(), w, h, nullptr);
      if (rc != HASTY_OK) return rc;
      std::string base = std::string(out_dir) + "/" + names[a];
      if (!write_exr_rgb(base + ".exr", img.data(), int(w), int(h))) throw ApiError{HASTY_ERR_IO, "could not write " + base + ".exr"};
      if (write_pfm && !write_pfm_rgb(base + ".pfm", img.data(), int(w), int(h))) throw ApiError{HASTY_ERR_IO, "could not write " + base + ".pfm"};
    }
    return HASTY_OK;
  });
}

// Enqueues snapshot slot k of the AOVs in `mask`: the estimates on the job's
// stream behind every pass enqueued so far, their copy to pinned memory on
// the copy stream. Returns without waiting.
static void enqueue_snapshot(hasty_job& j, int k, uint32_t mask) {
  if (!j.acc[0]) throw ApiError{HASTY_ERR_ARG, "job was loaded for the multi-job engine only"};
  ck(cudaSetDevice(j.ctx->device), "cudaSetDevice");
  const size_t n = size_t(j.sd.width) * size_t(j.sd.height) * 3;
  hasty_job::Snapshot& s = j.snap[k];
  if (!s.dev) {
    s.dev = j.alloc<float>(3 * n);
    ck(cudaHostAlloc(reinterpret_cast<void**>(&s.host), 3 * n * sizeof(float), cudaHostAllocDefault), "cudaHostAlloc");
    ck(cudaEventCreateWithFlags(&s.copied, cudaEventDisableTiming), "event");
  }
  if (!j.copy_stream) {
    ck(cudaStreamCreateWithFlags(&j.copy_stream, cudaStreamNonBlocking), "stream");
    ck(cudaEventCreateWithFlags(&j.snap_est, cudaEventDisableTiming), "event");
  }
  // the slot's previous copy reads `dev`: the new estimates wait for it
  if (s.pending) ck(cudaStreamWaitEvent(j.stream, s.copied, 0), "snapshot wait");
  const float den = 1e-7f + float(j.samples_done);
  for (int a = 0; a < 3; ++a) {
    if (!(mask & (1u << a))) continue;
    const float scale = a == HASTY_AOV_COLOR ? std::pow(2.0f, j.host.cam.exposure) : 1.0f;
    launch_estimate(j.acc[a], int(n), den, scale, s.dev + size_t(a) * n, j.stream);
  }
  ck(cudaGetLastError(), "estimate launch");
  ck(cudaEventRecord(j.snap_est, j.stream), "event record");
  ck(cudaStreamWaitEvent(j.copy_stream, j.snap_est, 0), "snapshot wait");
  for (int a = 0; a < 3; ++a) {
    if (!(mask & (1u << a))) continue;
    ck(cudaMemcpyAsync(s.host + size_t(a) * n, s.dev + size_t(a) * n, n * sizeof(float), cudaMemcpyDeviceToHost,
                       j.copy_stream), "copy snapshot");
  }
  ck(cudaEventRecord(s.copied, j.copy_stream), "event record");
  s.pending = true;
  s.mask = mask;
  s.samples = j.samples_done;
}

static void check_out_dir(const char* out_dir) {
  if (!out_dir) throw ApiError{HASTY_ERR_ARG, "null directory"};
  struct stat sb;
  if (stat(out_dir, &sb) != 0 || !S_ISDIR(sb.st_mode)) throw ApiError{HASTY_ERR_IO, std::string("not a directory: ") + out_dir};
}

int hasty_job_snapshot(hasty_job* job, uint32_t aov_mask) {
  return guarded([&] {
    as_job(job);
    if (aov_mask == 0 || aov_mask > 7u) throw ApiError{HASTY_ERR_ARG, "bad aov mask"};
    enqueue_snapshot(*job, 0, aov_mask);
    return HASTY_OK;
  });
}

int hasty_job_snapshot_query(hasty_job* job, int* ready) {
  return guarded([&] {
    as_job(job);
    if (!ready) throw ApiError{HASTY_ERR_ARG, "null output"};
    const hasty_job::Snapshot& s = job->snap[0];
    if (!s.pending) throw ApiError{HASTY_ERR_ARG, "no snapshot was taken"};
    const cudaError_t e = cudaEventQuery(s.copied);
    if (e == cudaErrorNotReady) {
      (void)cudaGetLastError();        // "not ready" is an answer, not an error to report later
      *ready = 0;
    } else {
      ck(e, "snapshot query");
      *ready = 1;
    }
    return HASTY_OK;
  });
}

int hasty_job_snapshot_get(hasty_job* job, int aov, const float** out, int32_t* num_samples) {
  return guarded([&] {
    as_job(job);
    if (aov < 0 || aov > 2 || !out) throw ApiError{HASTY_ERR_ARG, "bad aov or output"};
    const hasty_job::Snapshot& s = job->snap[0];
    if (!s.pending) throw ApiError{HASTY_ERR_ARG, "no snapshot was taken"};
    if (!(s.mask & (1u << aov))) throw ApiError{HASTY_ERR_ARG, "aov not in the snapshot"};
    ck(cudaEventSynchronize(s.copied), "snapshot wait");
    *out = s.host + size_t(aov) * size_t(job->sd.width) * size_t(job->sd.height) * 3;
    if (num_samples) *num_samples = s.samples;
    return HASTY_OK;
  });
}

int hasty_job_write_outputs_async(hasty_job* job, const char* out_dir, int write_pfm) {
  return guarded([&] {
    as_job(job);
    check_out_dir(out_dir);
    if (job->writer.joinable()) job->writer.join();   // the previous write reads slot 1
    enqueue_snapshot(*job, 1, 7u);
    job->writer_rc = HASTY_OK;
    job->writer_err.clear();
    const int device = job->ctx->device;
    const int w = job->sd.width, h = job->sd.height;
    hasty_job::Snapshot* s = &job->snap[1];
    hasty_job* j = job;
    std::string dir(out_dir);
    job->writer = std::thread([j, s, device, w, h, dir, write_pfm] {
      const char* names[3] = {"output", "outputNormal", "outputAlbedo"};
      cudaError_t e = cudaSetDevice(device);
      if (e == cudaSuccess) e = cudaEventSynchronize(s->copied);
      if (e != cudaSuccess) {
        j->writer_rc = HASTY_ERR_CUDA;
        j->writer_err = std::string("snapshot wait: ") + cudaGetErrorString(e);
        return;
      }
      const size_t n = size_t(w) * size_t(h) * 3;
      for (int a = 0; a < 3; ++a) {
        const float* img = s->host + size_t(a) * n;
        const std::string base = dir + "/" + names[a];
        if (!write_exr_rgb(base + ".exr", img, w, h) || (write_pfm && !write_pfm_rgb(base + ".pfm", img, w, h))) {
          j->writer_rc = HASTY_ERR_IO;
          j->writer_err = "could not write " + base;
          return;
        }
      }
    });
    return HASTY_OK;
  });
}

int hasty_job_outputs_wait(hasty_job* job) {
  return guarded([&] {
    as_job(job);
    if (job->writer.joinable()) job->writer.join();
    if (job->writer_rc != HASTY_OK) {
      const int rc = job->writer_rc;
      job->writer_rc = HASTY_OK;
      throw ApiError{rc, job->writer_err};
    }
    return HASTY_OK;
  });
}

int hasty_debug_obj_digest(const char* path, int chunks, uint64_t* digest, int64_t* n_tris, int64_t* n_shapes) {
  return guarded([&] {
    if (!path || !digest || chunks < 0 || chunks > 4096) throw ApiError{HASTY_ERR_ARG, "bad argument"};
    *digest = obj_digest(path, size_t(chunks), n_tris, n_shapes);
    return HASTY_OK;
  });
}

int hasty_debug_intersect(hasty_job* job, const float* rays, size_t n, int32_t* tri, float* t, float* u, float* v) {
  return guarded([&] {
    as_job(job);
    if (n == 0) return HASTY_OK;
    if (!rays || !tri || !t || !u || !v) throw ApiError{HASTY_ERR_ARG, "null buffer"};
    if (n > size_t(INT32_MAX)) throw ApiError{HASTY_ERR_ARG, "too many rays"};
    // Chunks of rays through two kept lists, so that a chunk's rays are copied
    // while the one before is traced. (1M rays: device allocations 0.25 ms and
    // an interleaved hit array taken apart on the host 2.1 ms, around 0.38 ms
    // of copies and tracing.)
    ck(cudaSetDevice(job->ctx->device), "cudaSetDevice");   // the lists, stream and event stay with the job
    std::lock_guard<std::mutex> lock(job->ray_mutex);
    const size_t chunk = std::min(n, hasty_job::kRayChunk);
    const int lists = n > chunk ? 2 : 1;
    for (int k = 0; k < lists; ++k) ray_list(*job, k, chunk);
    const cudaStream_t st[2] = {job->stream, job->ray_stream};
    cudaError_t err = cudaSuccess;
    auto step = [&](cudaError_t e) { if (err == cudaSuccess) err = e; };
    if (lists == 2) {
      step(cudaEventRecord(job->ray_ready, st[0]));
      step(cudaStreamWaitEvent(st[1], job->ray_ready, 0));
    }
    // A short list's results come back in one copy, taken apart on the host: four
    // copies cost more up to some 16k rays (4,510 rays: 73 us, now 54).
    if (n <= kShortRays) {
      const size_t pitch = (n + 63) / 64 * 64;
      float* at = reinterpret_cast<float*>(job->ray_lists[0].tri);
      const RayLists l = {job->ray_lists[0].rays, job->ray_lists[0].tri, at + pitch, at + 2 * pitch, at + 3 * pitch};
      std::unique_ptr<float[]> back(new float[4 * pitch]);
      step(cudaMemcpyAsync(l.rays, rays, n * 6 * sizeof(float), cudaMemcpyHostToDevice, st[0]));
      if (err == cudaSuccess) { launch_trace_rays(job->sd, l, int(n), st[0]); step(cudaGetLastError()); }
      if (err == cudaSuccess) step(cudaMemcpyAsync(back.get(), at, (3 * pitch + n) * 4, cudaMemcpyDeviceToHost, st[0]));
      const cudaError_t e = cudaStreamSynchronize(st[0]);
      step(e);
      ck(err, "debug intersect");
      std::memcpy(tri, back.get(), n * 4);
      std::memcpy(t, back.get() + pitch, n * 4);
      std::memcpy(u, back.get() + 2 * pitch, n * 4);
      std::memcpy(v, back.get() + 3 * pitch, n * 4);
      return HASTY_OK;
    }
    auto copy_back = [&](size_t first) {
      const int k = int(first / chunk & 1);
      const size_t bytes = std::min(chunk, n - first) * 4;
      const RayLists& l = job->ray_lists[k];
      step(cudaMemcpyAsync(tri + first, l.tri, bytes, cudaMemcpyDeviceToHost, st[k]));
      step(cudaMemcpyAsync(t + first, l.t, bytes, cudaMemcpyDeviceToHost, st[k]));
      step(cudaMemcpyAsync(u + first, l.u, bytes, cudaMemcpyDeviceToHost, st[k]));
      step(cudaMemcpyAsync(v + first, l.v, bytes, cudaMemcpyDeviceToHost, st[k]));
    };
    for (size_t first = 0; first < n && err == cudaSuccess; first += chunk) {
      const int k = int(first / chunk & 1);
      const size_t m = std::min(chunk, n - first);
      step(cudaMemcpyAsync(job->ray_lists[k].rays, rays + 6 * first, m * 6 * sizeof(float), cudaMemcpyHostToDevice, st[k]));
      if (err == cudaSuccess) { launch_trace_rays(job->sd, job->ray_lists[k], int(m), st[k]); step(cudaGetLastError()); }
      if (first > 0 && err == cudaSuccess) copy_back(first - chunk);
    }
    if (err == cudaSuccess) copy_back((n - 1) / chunk * chunk);
    for (int k = 0; k < lists; ++k) { const cudaError_t e = cudaStreamSynchronize(st[k]); step(e); }
    ck(err, "debug intersect");
    return HASTY_OK;
  });
}

int hasty_debug_wide_emit_check(int device, const char* job_path, int64_t* info, int32_t* identical) {
  return guarded([&] {
    if (!job_path || !identical) throw ApiError{HASTY_ERR_ARG, "null argument"};
    ck(cudaSetDevice(device), "cudaSetDevice");
    HostScene h;
    load_render_job(job_path, h);
    *identical = check_wide_emit_gpu(h.tri_pos.data(), h.n_tris(), info) ? 1 : 0;
    return HASTY_OK;
  });
}

int hasty_debug_host_trace(const char* job_path, int kind, const float* rays, size_t n, int32_t* tri, float* t, float* u,
                           float* v, int64_t* info) {
  return guarded([&] {
    if (!job_path || (n && (!rays || !tri || !t || !u || !v)) || (kind != 0 && kind != 1))
      throw ApiError{HASTY_ERR_ARG, "bad argument"};
    HostScene h;
    load_render_job(job_path, h);
    BvhHost bvh;
    if (kind == 0) build_bvh_binary(h.tri_pos.data(), h.n_tris(), 4, bvh);
    else build_bvh_wide(h.tri_pos.data(), h.n_tris(), bvh);
    std::vector<float4> nodes(bvh.nodes.size() / 4), tris(bvh.tris.size() / 4);
    std::memcpy(nodes.data(), bvh.nodes.data(), bvh.nodes.size() * sizeof(float));
    std::memcpy(tris.data(), bvh.tris.data(), bvh.tris.size() * sizeof(float));
    std::vector<float4> hits(n);
    host_trace_rays(kind, nodes.data(), tris.data(), rays, int64_t(n), hits.data());
    for (size_t i = 0; i < n; ++i) {
      int32_t id; std::memcpy(&id, &hits[i].w, 4);
      tri[i] = id; t[i] = hits[i].x; u[i] = hits[i].y; v[i] = hits[i].z;
    }
    if (info) { info[0] = int64_t(h.n_tris()); info[1] = int64_t(nodes.size() / (kind == 1 ? kWideNodeWords / 4 : 4)); info[2] = bvh.depth; }
    return HASTY_OK;
  });
}

int hasty_debug_tri_ids(hasty_job* job, int32_t* geom, int32_t* prim, size_t n) {
  return guarded([&] {
    as_job(job);
    if (n != job->host.tri_attr.size()) throw ApiError{HASTY_ERR_ARG, "n must equal the triangle count"};
    for (size_t i = 0; i < n; ++i) { geom[i] = int32_t(job->host.tri_attr[i].geom); prim[i] = int32_t(job->host.tri_attr[i].prim); }
    return HASTY_OK;
  });
}

int hasty_debug_finish_limits(hasty_job* job, int64_t* at_once, int64_t* later) {
  return guarded([&] {
    as_job(job);
    if (!at_once || !later) throw ApiError{HASTY_ERR_ARG, "null argument"};
    ck(cudaSetDevice(job->ctx->device), "cudaSetDevice");
    const FinishLimits l = finish_limits(job->sd);
    *at_once = l.at_once;
    *later = l.later;
    return HASTY_OK;
  });
}

int hasty_debug_cdf_draw(const double* cdf, size_t n, const uint64_t* draws, size_t m, uint32_t* index) {
  return guarded([&] {
    if (!cdf || n < 2 || n > size_t(INT32_MAX) || (m && (!draws || !index))) throw ApiError{HASTY_ERR_ARG, "bad argument"};
    const std::vector<double> c(cdf, cdf + n);
    uint32_t log2k = 0;
    const std::vector<uint32_t> guide = build_cdf_guide(c, log2k);
    std::vector<uint64_t> thr(n);
    for (size_t i = 0; i < n; ++i) thr[i] = cdf_threshold(c[i]);
    for (size_t i = 0; i < m; ++i) index[i] = cdf_index(thr.data(), uint32_t(n), draws[i], guide.data(), log2k);
    return HASTY_OK;
  });
}

int hasty_debug_bounds_status(uint32_t* flags) {
#ifdef HASTY_DEBUG_BOUNDS
  if (!flags) return fail(HASTY_ERR_ARG, "null argument");
  *flags = hasty::bounds_status_integrator() | hasty::bounds_status_trace() | hasty::bounds_status_photon();
  return HASTY_OK;
#else
  (void)flags;
  return fail(HASTY_ERR_MISSING, "bounds checks are compiled into the bounds-checked build only "
                                 "(python -m hastyrenderer_gb300.build --debug-bounds)");
#endif
}

int hasty_debug_bsdf(int which, const float* in, size_t n_cases, const uint32_t* replay, size_t n_replay, float* out) {
  return guarded([&] {
    if (which < 0 || which > 2 || !in || !out || (n_replay && !replay)) throw ApiError{HASTY_ERR_ARG, "bad argument"};
    if (n_cases == 0) return HASTY_OK;
    if (n_replay == 0) throw ApiError{HASTY_ERR_ARG, "replay stream must not be empty"};
    float *din = nullptr, *dout = nullptr; uint32_t* drep = nullptr;
    ck(cudaMalloc(&din, n_cases * 33 * sizeof(float)), "cudaMalloc");
    cudaError_t err = cudaMalloc(&dout, n_cases * 12 * sizeof(float));
    if (err == cudaSuccess) err = cudaMalloc(&drep, n_cases * n_replay * sizeof(uint32_t));
    if (err == cudaSuccess) err = cudaMemcpy(din, in, n_cases * 33 * sizeof(float), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) err = cudaMemcpy(drep, replay, n_cases * n_replay * sizeof(uint32_t), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) { launch_debug_bsdf(which, din, int(n_cases), drep, int(n_replay), dout, 0); err = cudaGetLastError(); }
    if (err == cudaSuccess) err = cudaMemcpy(out, dout, n_cases * 12 * sizeof(float), cudaMemcpyDeviceToHost);
    cudaFree(din); cudaFree(dout); cudaFree(drep);
    ck(err, "debug bsdf");
    return HASTY_OK;
  });
}

}  // extern "C"
