// Photon mapper, host side and C ABI (include/hasty_gpu.h, hasty_pm_*): the
// loop of the reference's renderPhotonThread (core/src/PhotonMapping.cpp:
// 814-935) for one render thread, with the photon tracing and the per-pixel
// gather on the GPU (photon.cu). The host keeps what the reference computes
// sequentially in float: the footprint angle of each pixel, the fill of
// pixels without a footprint, the hash-cell size, and the photon map's cell
// order (photons sorted by cell, then by emission index and depth, which is
// the order the reference's hash cells list them in).
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

#include "job.h"
#include "photon.h"
#include "scene_load.h"

namespace hasty {

struct PmDev {
  uint32_t W = 0, H = 0;
  bool initialised = false;
  uint32_t iteration = 0;
  PmPixelsDev px{};
  unsigned long long* stats = nullptr;     // [0] media overflow, [1] trial cap
  // photon buffers (grown on demand)
  PhotonRec* append = nullptr;
  size_t append_cap = 0;
  uint32_t* append_count = nullptr;
  uint32_t* fetch = nullptr;               // emission counter of the photon kernel
  uint8_t* stored = nullptr;
  size_t stored_cap = 0;
  float4* pos = nullptr;                   // photons in map order (PmMapDev)
  size_t pos_cap = 0;
  float4* rest = nullptr;
  size_t rest_cap = 0;
  uint32_t* start = nullptr;               // table of cell starts (PmMapDev)
  size_t start_cap = 0;
  int64_t max_table = kPmDenseCells;
  bool any_frame = false;                  // (test hook) however few pixels the frame has
  bool table_used = false;                 // by the last iteration's gather
  int4* cells = nullptr;
  size_t cells_cap = 0;
  int32_t* n_cells = nullptr;
  // map build (photon_build.cu)
  PmStatus* status = nullptr;              // device
  PmStatus* status_host = nullptr;         // pinned
  uint32_t* base = nullptr;                // first slot of each emission
  size_t base_cap = 0;
  uint32_t* scratch = nullptr;
  size_t scratch_cap = 0;
  uint32_t* src = nullptr;                 // append index of each slot
  size_t src_cap = 0;
  int32_t* coords = nullptr;               // hash cell of each slot, three planes
  size_t coords_cap = 0;
  uint32_t* perm[2] = {nullptr, nullptr};
  size_t perm_cap[2] = {0, 0};
  uint32_t* flag = nullptr;
  size_t flag_cap = 0;
  uint32_t* cell_of = nullptr;
  size_t cell_of_cap = 0;
  uint32_t* hist = nullptr;
  size_t hist_cap = 0;
  float* columns = nullptr;                // radius image, column by column
  float* radii = nullptr;                  // its host copy (pinned)
  ~PmDev() {
    if (status_host) cudaFreeHost(status_host);
    if (radii) cudaFreeHost(radii);
  }
  // last iteration
  uint64_t emitted = 0, photons = 0;
  float cell = 0.0f;
  double device_ms = 0.0, host_ms = 0.0, photon_ms = 0.0, gather_ms = 0.0, cell_ms = 0.0, map_ms = 0.0;
  uint64_t last_emitted = 0;               // sizes the next iteration's first photon batch
};

void destroy_pm(PmDev* pm) { delete pm; }

namespace {


// Camera::computeRayAngle (Camera.cpp:83-98) is 0.5 * ax + 0.5 * ay with ax
// of the pixel's column and ay of its row; this is either, for a frame `size`
// wide or high (W: its width); q = tan(fov / 2) as the camera evaluates it.
float axis_angle(float q, float x, float size, float W) {
  float l1 = (x + 0.5f - 0.5f * size) / W * 2.0f;
  float l2 = (x - 0.5f - 0.5f * size) / W * 2.0f;
  return std::fabs(std::atan(q * l1) - std::atan(q * l2));
}

// getCloseNonNegative (PhotonMapping.cpp:653-678), img[x + y * W]; the
// reference's fourth candidate per step is computed and never tested.
float close_non_negative(const float* img, int W, int H, int i, int j) {
  auto inside = [&](int x, int y) { return x >= 0 && y >= 0 && x < W && y < H; };
  auto at = [&](int x, int y) { return img[size_t(y) * size_t(W) + size_t(x)]; };
  for (int k = 1; k < std::max(H, W); ++k) {
    for (int m = 0; m <= k * 2; m++) {
      int i2 = i - k, j2 = j - k + m;
      if (inside(i2, j2) && at(i2, j2) > 0.0f) return at(i2, j2);
      i2 = i - k + m; j2 = j - k;
      if (inside(i2, j2) && at(i2, j2) > 0.0f) return at(i2, j2);
      i2 = i + k; j2 = j - k + m;
      if (inside(i2, j2) && at(i2, j2) > 0.0f) return at(i2, j2);
    }
  }
  return 1e-3f;
}

// fn(0) .. fn(n - 1), each once, on up to n threads, the calling one among them.
// It takes over what is left where the system gives no further thread, and
// joins the ones it started. fn does not throw.
template <class Fn>
void run_parts(size_t n, Fn fn) {
  std::atomic<size_t> next{0};
  auto work = [&] { for (size_t k; (k = next.fetch_add(1)) < n;) fn(k); };
  std::vector<std::thread> th;
  th.reserve(n);
  try {
    while (th.size() + 1 < n) th.emplace_back(work);
  } catch (const std::system_error&) {
  }
  work();
  for (std::thread& t : th) t.join();
}

// The cost of four cell sizes: float sums over the radii in the order given.
typedef float f4 __attribute__((vector_size(16)));
f4 cell_costs(const float* radii, size_t n, f4 c) {
  auto p3 = [](f4 f) { return f * (f * f); };        // powci<3>
  f4 s = {0.0f, 0.0f, 0.0f, 0.0f};
  for (size_t i = 0; i < n; ++i) {
    const f4 r = {radii[i], radii[i], radii[i], radii[i]};
    s += 5.0f * p3(r / c) + p3(r < c ? c : r) * 1e5f;
  }
  return s;
}

// computeCellSize (PhotonMapping.cpp:522-576): float sums in the reference's
// order (x outer, y inner), which is the order of `radii`. The reference
// evaluates cost(cs), then up to 10 trials cs *= 1.5 while they improve, then
// up to 10 trials cs *= 0.6666. A sum's additions wait for each other, so four
// costs in one vector take the time of one: the ones that the search usually
// needs are evaluated first, by three threads where that is worth starting
// them, any others when they are reached. Computed while the GPU traces photons
// (1.08 ms at 640x480): 0.84 ms, where a thread per trial value over radii in
// row order took 2.1 ms, and 0.9 ms at 17x13 (now 0.001).
float cell_size_for(const float* radii, size_t n) {
  float sum = 0.0f;
  for (size_t i = 0; i < n; ++i) sum += radii[i];
  const float cs = sum / float(uint32_t(n));
  float up[12], cu[12], down[11][12], cd[11][12];
  int n_up = 0, n_down[11] = {};
  up[0] = cs;
  for (int k = 1; k < 12; ++k) up[k] = up[k - 1] * 1.5f;
  for (int at = 0; at <= 10; ++at) {
    down[at][0] = up[at] * 0.6666f;
    for (int k = 1; k < 12; ++k) down[at][k] = down[at][k - 1] * 0.6666f;
  }
  auto more_up = [&] {
    const f4 c = cell_costs(radii, n, f4{up[n_up], up[n_up + 1], up[n_up + 2], up[n_up + 3]});
    for (int k = 0; k < 4; ++k) cu[n_up + k] = c[k];
    n_up += 4;
  };
  auto first_down = [&](int at) {                     // two trials below each of up[at], up[at + 1]
    const f4 c = cell_costs(radii, n, f4{down[at][0], down[at][1], down[at + 1][0], down[at + 1][1]});
    for (int k = 0; k < 2; ++k) { cd[at][k] = c[k]; cd[at + 1][k] = c[2 + k]; }
    n_down[at] = n_down[at + 1] = 2;
  };
  if (n >= (size_t(1) << 15)) run_parts(3, [&](size_t k) { if (k == 0) more_up(); else first_down(2 * int(k) - 2); });
  else more_up();
  float best = cu[0];
  int at = 0;
  for (int k = 1; k <= 10; ++k) {
    if (k == n_up) more_up();
    if (!(cu[k] < best)) break;
    best = cu[k];
    at = k;
  }
  float cell = up[at];
  for (int k = 0; k < 10; ++k) {
    int& have = n_down[at];
    if (k == have) {
      const float* d = down[at] + have;
      const f4 c = cell_costs(radii, n, f4{d[0], d[1], d[2], d[3]});
      for (int m = 0; m < 4; ++m) cd[at][have + m] = c[m];
      have += 4;
    }
    if (!(cd[at][k] < best)) break;
    best = cd[at][k];
    cell = down[at][k];
  }
  return cell;
}

// fn(begin, end) over [0, n) on up to 8 threads, each with at least `least`.
template <class Fn>
void parallel_ranges(size_t n, size_t least, Fn fn) {
  const size_t hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t nt = std::max<size_t>(1, std::min({n / std::max<size_t>(least, 1), hw, size_t(8)}));
  run_parts(nt, [&](size_t k) { fn(n * k / nt, n * (k + 1) / nt); });
}

// d: the pixels' distances (computeRadiusPixelFootPrint, negative: none), row
// by row, replaced by the footprint radii x 10. The angle's arctangents belong
// to a column or a row; what is left per pixel is one tangent, on several
// threads (640x480: 9.2 ms -> 1.1 ms in all).
void footprint_radii(float* d, uint32_t W, uint32_t H, const std::vector<float>& ax, const std::vector<float>& ay) {
  std::atomic<bool> holes{false};
  parallel_ranges(H, (size_t(1) << 14) / W + 1, [&](size_t y0, size_t y1) {
    bool hole = false;
    for (size_t y = y0; y < y1; y++)
      for (size_t x = 0; x < W; x++) {
        const size_t p = y * W + x;
        float fp = -1.0f;                       // computeRadiusPixelFootPrint's default
        if (d[p] >= 0.0f) {
          float angle = 0.5f * ax[x] + 0.5f * ay[y];
          fp = 0.5f * d[p] * std::tan(angle);
        }
        d[p] = 10.0f * fp;
        hole = hole || d[p] < 0.0f;
      }
    if (hole) holes = true;
  });
  if (holes)                                     // one after the other: a filled pixel counts for the next ones
    for (uint32_t y = 0; y < H; y++)
      for (uint32_t x = 0; x < W; x++)
        if (d[size_t(y) * W + x] < 0.0f) d[size_t(y) * W + x] = close_non_negative(d, int(W), int(H), int(x), int(y));
}

// The angle terms of every column and row; q = tan(fov / 2).
void footprint_angles(float q, uint32_t W, uint32_t H, std::vector<float>& ax, std::vector<float>& ay) {
  ax.resize(W);
  ay.resize(H);
  for (uint32_t x = 0; x < W; x++) ax[x] = axis_angle(q, float(x) + 0.5f, float(W), float(W));
  for (uint32_t y = 0; y < H; y++) ay[y] = axis_angle(q, float(y) + 0.5f, float(H), float(W));
}

template <class T>
T* grow(hasty_job& j, T* old, size_t& cap, size_t need, size_t keep) {
  if (need <= cap) return old;
  size_t n = std::max(need, cap + cap / 2);
  T* p = j.alloc<T>(n);
  if (old && keep) ck(cudaMemcpyAsync(p, old, keep * sizeof(T), cudaMemcpyDeviceToDevice, j.stream), "grow");
  if (old) { ck(cudaStreamSynchronize(j.stream), "grow"); j.release(old); }
  cap = n;
  return p;
}

PmDev& pm_state(hasty_job& j) {
  if (!j.pm) {
    auto* pm = new PmDev();
    j.pm = pm;
    const uint32_t W = uint32_t(j.sd.width), H = uint32_t(j.sd.height);
    const size_t n = size_t(W) * H;
    pm->W = W; pm->H = H;
    pm->px.radius = j.alloc<float>(n);
    pm->px.N = j.alloc<float>(n);
    pm->px.Ne = j.alloc<float>(n);
    pm->px.flux = j.alloc<float4>(n);
    pm->px.lsum = j.alloc<float4>(n);
    pm->px.radii = j.alloc<float>(n);
    pm->px.color = j.alloc<float>(3 * n);
    pm->px.normal = j.alloc<float>(3 * n);
    pm->px.albedo = j.alloc<float>(3 * n);
    pm->stats = j.alloc<unsigned long long>(2);
    pm->append_count = j.alloc<uint32_t>(1);
    pm->fetch = j.alloc<uint32_t>(1);
    pm->n_cells = j.alloc<int32_t>(1);
    pm->status = j.alloc<PmStatus>(1);
    pm->columns = j.alloc<float>(n);
    ck(cudaHostAlloc(reinterpret_cast<void**>(&pm->status_host), sizeof(PmStatus), cudaHostAllocDefault), "cudaHostAlloc");
    ck(cudaHostAlloc(reinterpret_cast<void**>(&pm->radii), n * sizeof(float), cudaHostAllocDefault), "cudaHostAlloc");
  }
  return *j.pm;
}

// Enqueues the copy of the radius image to pm.radii.
void read_radii(hasty_job& j, PmDev& pm) {
  launch_pm_transpose(pm.px.radii, pm.columns, pm.W, pm.H, j.stream);
  ck(cudaGetLastError(), "radii launch");
  ck(cudaMemcpyAsync(pm.radii, pm.columns, size_t(pm.W) * pm.H * sizeof(float), cudaMemcpyDeviceToHost, j.stream), "radii");
}

// Pixel statistics cleared and the radius image set up (renderPhotonThread,
// PhotonMapping.cpp:828-833: footprint radii x 10 with a surface light, else 1).
void pm_init(hasty_job& j, PmDev& pm) {
  const uint32_t W = pm.W, H = pm.H;
  const size_t n = size_t(W) * H;
  launch_pm_fill(pm.px.radius, n, -1.0f, j.stream);
  ck(cudaMemsetAsync(pm.px.N, 0, n * sizeof(float), j.stream), "pm init");
  ck(cudaMemsetAsync(pm.px.Ne, 0, n * sizeof(float), j.stream), "pm init");
  ck(cudaMemsetAsync(pm.px.flux, 0, n * sizeof(float4), j.stream), "pm init");
  ck(cudaMemsetAsync(pm.px.lsum, 0, n * sizeof(float4), j.stream), "pm init");
  ck(cudaMemsetAsync(pm.px.color, 0, 3 * n * sizeof(float), j.stream), "pm init");
  ck(cudaMemsetAsync(pm.px.normal, 0, 3 * n * sizeof(float), j.stream), "pm init");
  ck(cudaMemsetAsync(pm.px.albedo, 0, 3 * n * sizeof(float), j.stream), "pm init");
  ck(cudaMemsetAsync(pm.stats, 0, 2 * sizeof(unsigned long long), j.stream), "pm init");
  if (j.sd.n_light_tris > 0) {
    float* d = pm.radii;                         // distances, then radii, row by row
    launch_pm_footprint(j.sd, j.seed, pm.px.radii, j.stream);
    ck(cudaGetLastError(), "footprint launch");
    ck(cudaMemcpyAsync(d, pm.px.radii, n * sizeof(float), cudaMemcpyDeviceToHost, j.stream), "footprint");
    std::vector<float> ax, ay;
    footprint_angles(j.sd.cam.q, W, H, ax, ay);
    ck(cudaStreamSynchronize(j.stream), "footprint");
    footprint_radii(d, W, H, ax, ay);
    ck(cudaMemcpyAsync(pm.px.radii, d, n * sizeof(float), cudaMemcpyHostToDevice, j.stream), "radii");
  } else {
    launch_pm_fill(pm.px.radii, n, 1.0f, j.stream);
  }
  read_radii(j, pm);
  ck(cudaStreamSynchronize(j.stream), "pm init");
  pm.initialised = true;
  pm.iteration = 0;
}

// One iteration of renderPhotonThread's loop (PhotonMapping.cpp:848-931).
// The GPU traces photon batches and scans their store counts; the hash-cell
// size is computed on the host meanwhile (it needs only the radii of the
// previous iteration); then the photon map is built and gathered on the GPU.
void pm_iteration(hasty_job& j, PmDev& pm) {
  const uint32_t W = pm.W, H = pm.H, t = pm.iteration;
  const auto h0 = std::chrono::steady_clock::now();
  cudaEvent_t ev[6];
  for (cudaEvent_t& e : ev) ck(cudaEventCreate(&e), "event");
  auto elapsed = [&](int a, int b) {
    float ms = 0.f;
    ck(cudaEventElapsedTime(&ms, ev[a], ev[b]), "event time");
    return double(ms);
  };
  double photon_ms = 0.0, cell_ms = 0.0;
  float cell = 0.0f;
  bool have_cell = false;
  auto compute_cell = [&] {
    const auto c0 = std::chrono::steady_clock::now();
    cell = cell_size_for(pm.radii, size_t(W) * H);
    cell_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - c0).count();
    have_cell = true;
  };
  uint32_t emitted = 0, kept = 0, appended = 0;
  const int count_threshold = int(0.5f * float(H) * float(W));
  if (j.sd.n_light_tris > 0 && count_threshold > 0) {
    const int trace_threshold = int(10.f * float(H) * float(W));
    const int depth_slots = std::max(1, j.sd.max_depth - 1);   // photons one emitted photon can store
    const float min_q = 1.0f - std::pow(0.1f, 1.0f / j.sd.max_depth);
    uint32_t first = 0;
    // first batch: what the previous iteration needed (+10%), else 2x the stored target
    size_t chunk = std::max<size_t>(size_t(1) << 16, pm.last_emitted ? size_t(pm.last_emitted * 1.1) + 1024
                                                                     : 2 * size_t(count_threshold));
    ck(cudaMemsetAsync(pm.append_count, 0, sizeof(uint32_t), j.stream), "photon count");
    ck(cudaMemsetAsync(pm.status, 0, sizeof(PmStatus), j.stream), "photon status");
    for (;;) {
      const uint32_t n = uint32_t(std::min<uint64_t>(chunk, uint64_t(trace_threshold) - first));
      pm.append = grow(j, pm.append, pm.append_cap, size_t(appended) + size_t(n) * depth_slots, appended);
      pm.stored = grow(j, pm.stored, pm.stored_cap, n, 0);
      pm.base = grow(j, pm.base, pm.base_cap, size_t(first) + n, first);
      pm.scratch = grow(j, pm.scratch, pm.scratch_cap, size_t(n) / 2048 + 2, 0);
      PmEmitOut out{pm.append, pm.append_count, uint32_t(pm.append_cap), pm.stored, pm.stats, pm.fetch};
      ck(cudaEventRecord(ev[0], j.stream), "event");
      launch_pm_emit(j.sd, j.seed, t, first, n, min_q, out, j.stream);
      launch_pm_emit_scan(pm.stored, n, first, uint32_t(count_threshold), pm.base, pm.scratch, pm.status, j.stream);
      ck(cudaGetLastError(), "photon launch");
      ck(cudaEventRecord(ev[1], j.stream), "event");
      ck(cudaMemcpyAsync(&pm.status->appended, pm.append_count, sizeof(uint32_t), cudaMemcpyDeviceToDevice, j.stream),
         "photon count");
      ck(cudaMemcpyAsync(pm.status_host, pm.status, sizeof(PmStatus), cudaMemcpyDeviceToHost, j.stream), "photon status");
      ck(cudaEventRecord(ev[2], j.stream), "event");
      if (!have_cell) compute_cell();           // overlaps the photon tracing
      ck(cudaEventSynchronize(ev[2]), "photons");
      photon_ms += elapsed(0, 1);
      appended = pm.status_host->appended;
      if (appended > pm.append_cap) throw ApiError{HASTY_ERR_CUDA, "photon buffer overflow"};
      // the reference emits photon i while fewer than count_threshold are stored
      if (pm.status_host->done) { emitted = pm.status_host->emitted; kept = pm.status_host->kept; break; }
      first += n;
      if (first >= uint32_t(trace_threshold)) { emitted = first; kept = pm.status_host->cum; break; }
      chunk *= 2;
    }
  }
  if (!have_cell) compute_cell();
  // Photon map: the kept photons in emission order (slot = the emission's
  // first slot + the photon's index within it), then a stable radix sort by
  // hash cell, so each cell lists its photons in the order the reference
  // stored them.
  const uint32_t cap = std::max<uint32_t>(kept, 1u);
  const uint32_t tiles = pm_sort_tiles(cap);
  pm.src = grow(j, pm.src, pm.src_cap, cap, 0);
  pm.perm[0] = grow(j, pm.perm[0], pm.perm_cap[0], cap, 0);
  pm.perm[1] = grow(j, pm.perm[1], pm.perm_cap[1], cap, 0);
  pm.flag = grow(j, pm.flag, pm.flag_cap, cap, 0);
  pm.cell_of = grow(j, pm.cell_of, pm.cell_of_cap, cap, 0);
  pm.hist = grow(j, pm.hist, pm.hist_cap, size_t(256) * tiles, 0);
  pm.scratch = grow(j, pm.scratch, pm.scratch_cap, size_t(cap) / 2048 + size_t(tiles) / 8 + 2, 0);
  pm.pos = grow(j, pm.pos, pm.pos_cap, cap, 0);
  pm.rest = grow(j, pm.rest, pm.rest_cap, 2 * size_t(cap), 0);
  pm.cells = grow(j, pm.cells, pm.cells_cap, cap, 0);
  // coordinates: three planes of `coords_cap / 3` slots
  if (pm.coords_cap < 3 * size_t(cap)) {
    j.release(pm.coords);
    pm.coords = nullptr;
    pm.coords_cap = 0;
    pm.coords = grow(j, pm.coords, pm.coords_cap, 3 * size_t(cap), 0);
  }
  const uint32_t plane = uint32_t(pm.coords_cap / 3);
  ck(cudaEventRecord(ev[3], j.stream), "event");
  launch_pm_place(pm.append, appended, pm.base, emitted, pm.status, cell, pm.src, pm.coords, plane, j.stream);
  ck(cudaGetLastError(), "photon map launch");
  const uint32_t* perm = nullptr;
  if (kept > 0) {
    ck(cudaMemcpyAsync(pm.status_host, pm.status, sizeof(PmStatus), cudaMemcpyDeviceToHost, j.stream), "cell bounds");
    ck(cudaStreamSynchronize(j.stream), "cell bounds");
  }
  if (kept > 1) {
    int which = 0;
    for (int axis = 2; axis >= 0; --axis) {      // least significant key first: z, y, x
      const uint32_t range = uint32_t(int64_t(pm.status_host->hi[axis]) - int64_t(pm.status_host->lo[axis]));
      for (int shift = 0; shift < 32 && (range >> shift) != 0; shift += 8) {
        launch_pm_sort_pass(pm.coords + size_t(axis) * plane, pm.status_host->lo[axis], shift, kept, perm,
                            pm.perm[which], pm.hist, pm.scratch, j.stream);
        perm = pm.perm[which];
        which ^= 1;
      }
    }
  }
  launch_pm_cells(pm.append, pm.src, pm.coords, plane, kept, perm, pm.pos, pm.rest, pm.flag, pm.cell_of, pm.scratch,
                  pm.cells, pm.n_cells, j.stream);
  ck(cudaGetLastError(), "photon map launch");
  PmMapDev map{};
  map.pos = pm.pos;
  map.rest = pm.rest;
  map.cells = pm.cells;
  map.n_cells = pm.n_cells;
  map.n = int32_t(kept);
  map.cell = cell;
  int64_t cells = 1;                             // of the bounds, at most kPmDenseCells + 1
  for (int a = 0; a < 3; ++a) {
    map.lo[a] = kept > 0 ? pm.status_host->lo[a] : 0;
    map.hi[a] = kept > 0 ? pm.status_host->hi[a] : -1;
    const int64_t d = int64_t(map.hi[a]) - map.lo[a] + 1;
    cells = d > kPmDenseCells ? kPmDenseCells + 1 : std::min<int64_t>(cells * d, kPmDenseCells + 1);
  }
  // The table of cell starts for 2.3 million cells takes 0.03 ms and saves the
  // gather of 307,200 pixels 0.26 ms of 1.86 (640x480 room): it would pay up to
  // about 70 cells a pixel there, and is made up to half of that.
  if (cells > 0 && cells <= pm.max_table && (pm.any_frame || cells <= 32 * int64_t(W) * H)) {
    try {
      pm.start = grow(j, pm.start, pm.start_cap, size_t(cells) + 1, 0);
      map.start = pm.start;
    } catch (const ApiError&) {
      cudaGetLastError();                        // no memory for the table: the gather searches the cells
    }
    if (map.start) launch_pm_starts(map, pm.start, cells, j.stream);
  }
  pm.table_used = map.start != nullptr;
  ck(cudaGetLastError(), "photon map launch");
  ck(cudaEventRecord(ev[4], j.stream), "event");
  const float ox = halton_value(2, t), oy = halton_value(3, t);
  launch_pm_gather(j.sd, map, pm.px, j.seed, t, ox, oy, int(emitted), pm.stats, pm.fetch, j.stream);
  ck(cudaGetLastError(), "gather launch");
  ck(cudaEventRecord(ev[5], j.stream), "event");
  read_radii(j, pm);
  ck(cudaStreamSynchronize(j.stream), "radii");
  const double map_ms = elapsed(3, 4), gather_ms = elapsed(4, 5);
  for (cudaEvent_t e : ev) cudaEventDestroy(e);
  const double dev_ms = photon_ms + map_ms + gather_ms;
  pm.emitted = emitted;
  pm.photons = kept;
  pm.cell = cell;
  pm.iteration = t + 1;
  pm.device_ms += dev_ms;
  pm.photon_ms += photon_ms;
  pm.gather_ms += gather_ms;
  pm.map_ms += map_ms;
  pm.cell_ms += cell_ms;
  pm.last_emitted = emitted;
  pm.host_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - h0).count() - dev_ms;
}

hasty_job* pm_job(hasty_job* j) {
  if (!j) throw ApiError{HASTY_ERR_ARG, "null job handle"};
  if (j->sd.max_depth > kPmMaxDepth)
    throw ApiError{HASTY_ERR_ARG, "photon mapping supports max_depth <= " + std::to_string(kPmMaxDepth)};
  ck(cudaSetDevice(j->ctx->device), "cudaSetDevice");
  return j;
}

}  // namespace
}  // namespace hasty

using namespace hasty;

extern "C" {

int hasty_pm_render(hasty_job* job, int iterations) {
  return guarded([&] {
    pm_job(job);
    if (iterations < 0) throw ApiError{HASTY_ERR_ARG, "negative iteration count"};
    ck(cudaStreamSynchronize(job->stream), "sync");
    PmDev& pm = pm_state(*job);
    if (!pm.initialised) pm_init(*job, pm);
    for (int k = 0; k < iterations; ++k) {
      if (job->stop.load()) throw ApiError{HASTY_ERR_STOPPED, "job stopped"};
      pm_iteration(*job, pm);
    }
    return HASTY_OK;
  });
}

int hasty_pm_reset(hasty_job* job) {
  return guarded([&] {
    pm_job(job);
    if (job->pm) job->pm->initialised = false;
    return HASTY_OK;
  });
}

int hasty_pm_read(hasty_job* job, int aov, float* host, size_t w, size_t h) {
  return guarded([&] {
    pm_job(job);
    if (aov < 0 || aov > 2 || !host) throw ApiError{HASTY_ERR_ARG, "bad aov or buffer"};
    if (w != size_t(job->sd.width) || h != size_t(job->sd.height)) throw ApiError{HASTY_ERR_ARG, "buffer size does not match the frame"};
    if (!job->pm || !job->pm->initialised) throw ApiError{HASTY_ERR_ARG, "no photon-mapping iteration rendered"};
    const float* src = aov == 0 ? job->pm->px.color : (aov == 1 ? job->pm->px.normal : job->pm->px.albedo);
    ck(cudaMemcpyAsync(host, src, w * h * 3 * sizeof(float), cudaMemcpyDeviceToHost, job->stream), "read");
    ck(cudaStreamSynchronize(job->stream), "read");
    if (aov == HASTY_AOV_COLOR) {            // image *= 2^exposure, PhotonMappingViewer.cpp:154
      const float scale = std::pow(2.0f, job->host.cam.exposure);
      for (size_t k = 0; k < w * h * 3; ++k) host[k] *= scale;
    }
    return HASTY_OK;
  });
}

int hasty_pm_read_radii(hasty_job* job, float* host, size_t w, size_t h) {
  return guarded([&] {
    pm_job(job);
    if (!host) throw ApiError{HASTY_ERR_ARG, "null buffer"};
    if (w != size_t(job->sd.width) || h != size_t(job->sd.height)) throw ApiError{HASTY_ERR_ARG, "buffer size does not match the frame"};
    if (!job->pm || !job->pm->initialised) throw ApiError{HASTY_ERR_ARG, "no photon-mapping iteration rendered"};
    for (size_t y = 0; y < h; ++y)
      for (size_t x = 0; x < w; ++x) host[y * w + x] = job->pm->radii[x * h + y];
    return HASTY_OK;
  });
}

int hasty_pm_stats_get(hasty_job* job, hasty_pm_stats* out) {
  return guarded([&] {
    pm_job(job);
    if (!out) throw ApiError{HASTY_ERR_ARG, "null argument"};
    std::memset(out, 0, sizeof(*out));
    if (!job->pm) return HASTY_OK;
    const PmDev& pm = *job->pm;
    out->iterations = int32_t(pm.iteration);
    out->photons_emitted = int64_t(pm.emitted);
    out->photons_stored = int64_t(pm.photons);
    out->cell_size = pm.cell;
    out->device_ms = pm.device_ms;
    out->host_ms = pm.host_ms;
    unsigned long long st[2] = {0, 0};
    if (pm.stats) {
      ck(cudaMemcpyAsync(st, pm.stats, sizeof(st), cudaMemcpyDeviceToHost, job->stream), "stats");
      ck(cudaStreamSynchronize(job->stream), "stats");
    }
    out->media_overflow = st[0];
    out->trial_cap = st[1];
    out->photon_ms = pm.photon_ms;
    out->gather_ms = pm.gather_ms;
    out->cell_ms = pm.cell_ms;
    out->map_ms = pm.map_ms;
    return HASTY_OK;
  });
}

int hasty_debug_pm_table(hasty_job* job, int64_t max_cells) {
  return guarded([&] {
    pm_job(job);
    pm_state(*job).max_table = std::min(max_cells, kPmDenseCells);
    pm_state(*job).any_frame = true;
    return HASTY_OK;
  });
}

int hasty_debug_pm_table_used(hasty_job* job, int32_t* used) {
  return guarded([&] {
    pm_job(job);
    if (!used) throw ApiError{HASTY_ERR_ARG, "null argument"};
    if (!job->pm || !job->pm->initialised) throw ApiError{HASTY_ERR_ARG, "no photon-mapping iteration rendered"};
    *used = job->pm->table_used ? 1 : 0;
    return HASTY_OK;
  });
}

int hasty_debug_pm_host(float* dist, size_t w, size_t h, float q, float* cell) {
  return guarded([&] {
    if (!dist || !cell || w == 0 || h == 0 || w > size_t(INT32_MAX) / h) throw ApiError{HASTY_ERR_ARG, "bad argument"};
    std::vector<float> ax, ay;
    footprint_angles(q, uint32_t(w), uint32_t(h), ax, ay);
    footprint_radii(dist, uint32_t(w), uint32_t(h), ax, ay);
    *cell = cell_size_for(dist, w * h);
    return HASTY_OK;
  });
}

int hasty_debug_pm_map(hasty_job* job, float* xyz, uint32_t* emission, uint32_t* index, int32_t* cells,
                       int64_t* n_photons, int64_t* n_cells, float* cell) {
  return guarded([&] {
    pm_job(job);
    if (!n_photons || !n_cells || !cell) throw ApiError{HASTY_ERR_ARG, "null count output"};
    if (!job->pm || !job->pm->initialised || job->pm->iteration == 0)
      throw ApiError{HASTY_ERR_ARG, "no photon-mapping iteration rendered"};
    const PmDev& pm = *job->pm;
    int32_t nc = 0;
    ck(cudaMemcpyAsync(&nc, pm.n_cells, sizeof(int32_t), cudaMemcpyDeviceToHost, job->stream), "map");
    ck(cudaStreamSynchronize(job->stream), "map");
    *n_photons = int64_t(pm.photons);
    *n_cells = nc;
    *cell = pm.cell;
    if (xyz && emission && index && pm.photons) {
      std::vector<float4> pos(pm.photons), rest(2 * pm.photons);
      ck(cudaMemcpyAsync(pos.data(), pm.pos, pos.size() * sizeof(float4), cudaMemcpyDeviceToHost, job->stream), "map");
      ck(cudaMemcpyAsync(rest.data(), pm.rest, rest.size() * sizeof(float4), cudaMemcpyDeviceToHost, job->stream), "map");
      ck(cudaStreamSynchronize(job->stream), "map");
      for (size_t q = 0; q < pos.size(); ++q) {
        xyz[3 * q] = pos[q].x; xyz[3 * q + 1] = pos[q].y; xyz[3 * q + 2] = pos[q].z;
        std::memcpy(&emission[q], &rest[2 * q].w, 4);
        std::memcpy(&index[q], &rest[2 * q + 1].w, 4);
      }
    }
    if (cells && nc > 0) {
      std::vector<int4> c(static_cast<size_t>(nc));
      ck(cudaMemcpyAsync(c.data(), pm.cells, c.size() * sizeof(int4), cudaMemcpyDeviceToHost, job->stream), "map");
      ck(cudaStreamSynchronize(job->stream), "map");
      for (size_t k = 0; k < c.size(); ++k) {
        cells[5 * k] = c[k].x; cells[5 * k + 1] = c[k].y; cells[5 * k + 2] = c[k].z;
        cells[5 * k + 3] = c[k].w;
        cells[5 * k + 4] = (k + 1 < c.size() ? c[k + 1].w : int32_t(pm.photons)) - c[k].w;
      }
    }
    return HASTY_OK;
  });
}

}  // extern "C"
