// Photon mapper kernels: the reference's stochastic progressive photon
// mapper (core/src/PhotonMapping.cpp) on the GPU, in persistent kernels whose
// lanes take the next photon or pixel when theirs has ended and go through each
// bounce in stages with their block. Compiled without FMA contraction like
// integrator.cu, and
// with the same device shading routines (device_common.cuh) and traversal
// (traverse.cuh), so each photon path and each gather path computes what the
// CPU restatement computes for the same random stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include "device_common.cuh"
#include "photon.h"
#include "traverse.cuh"
#include "wavefront.h"

namespace hasty {
namespace {
using namespace dev;

constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ Hit trace_ray(const SceneDev& sc, V3 o, V3 d) {
  return sc.bvh_kind == 1 ? trace_wide(sc.nodes, sc.isect_tris, o.x, o.y, o.z, d.x, d.y, d.z)
                          : trace_binary(sc.nodes, sc.isect_tris, o.x, o.y, o.z, d.x, d.y, d.z);
}

// The photon and gather kernels run in stages separated by block barriers
// (closest hits, then the code of the vertices they reach), so that the warps
// of a block share one region of code at a time: one thread per photon or
// pixel through the whole kernel waited for instructions 15-17 cycles per
// issue, with 6-7 lanes active. The rays of a block live in shared memory.
// One block per SM, so that all its warps share: four iterations of the
// 640x480 room took the photon kernel 4.34 ms with 512 threads, 4.92 with two
// blocks of 256 and 5.88 with four of 128 (gather: 6.4, 6.7, 9.3); more
// threads than 512 spill (3 x 256: 5.53, gather 8.72).
constexpr int kStageThreads = 512;
template <int KIND> struct StageTrav { using T = TravBinary; };
template <> struct StageTrav<1> { using T = TravWide; };

// Rays of one warp (two per lane, ray 2 * lane + k) and their hits.
struct WarpRays {
  float o[64][3], d[64][3];
  float4 hit[64];            // t, u, v, triangle
  int list[64];
  __device__ void put(int ray, V3 ro, V3 rd) {
    o[ray][0] = ro.x; o[ray][1] = ro.y; o[ray][2] = ro.z;
    d[ray][0] = rd.x; d[ray][1] = rd.y; d[ray][2] = rd.z;
  }
  __device__ V3 origin(int ray) const { return V3(o[ray][0], o[ray][1], o[ray][2]); }
  __device__ V3 dir(int ray) const { return V3(d[ray][0], d[ray][1], d[ray][2]); }
  __device__ Hit result(int ray) const {
    const float4 h = hit[ray];
    Hit r;
    r.t = h.x; r.u = h.y; r.v = h.z; r.tri = __float_as_int(h.w);
    return r;
  }
};

// Closest hits of the warp's rays (this lane's ray 2 * lane if r0, the next
// one if r1), taken by its lanes one after the other. All lanes call it.
template <int KIND>
__device__ __forceinline__ void trace_stage(const SceneDev& sc, WarpRays& w, bool r0, bool r1) {
  using Trav = typename StageTrav<KIND>::T;
  const uint32_t lane = threadIdx.x & 31u;
  const unsigned m0 = __ballot_sync(kFull, r0), m1 = __ballot_sync(kFull, r1), below = (1u << lane) - 1u;
  const uint32_t n0 = uint32_t(__popc(m0)), n = n0 + uint32_t(__popc(m1));
  if (r0) w.list[__popc(m0 & below)] = int(2 * lane);
  if (r1) w.list[n0 + __popc(m1 & below)] = int(2 * lane + 1);
  __syncwarp();
  uint32_t next = 0;
  trace_rays_of_queue<Trav, 4>(
      n, [&](uint32_t n_idle) { const uint32_t base = next; next += n_idle; return base; },
      [&](uint32_t k, Trav& tr, const float4*& nodes, const float4*& tris, int& id) {
        id = w.list[k];
        tr.init(w.o[id][0], w.o[id][1], w.o[id][2], w.d[id][0], w.d[id][1], w.d[id][2]);
        HASTY_TRAV_LIMITS(tr, sc.n_nodes, sc.n_tris);
        nodes = sc.nodes;
        tris = sc.isect_tris;
      },
      [&](int id, const Hit& h) { w.hit[id] = make_float4(h.t, h.u, h.v, __int_as_float(h.tri)); });
}

// LightRayInfo (core/src/LightRayInfo.cpp): the band and the medium stack of
// one path, at most kMaxMedia deep (a deeper push is dropped and counted).
struct PmMedia {
  int wl = -1;
  int n = 0;
  V3 T[kMaxMedia];
  float ior[kMaxMedia];
  int geom[kMaxMedia];
  __device__ V3 transmittance() const { return n > 0 ? T[0] : V3(1.f, 1.f, 1.f); }
  // getOutsideIOR, LightRayInfo.cpp:80-126
  __device__ float outside_ior(const Inter& it, V3 wfrom) const {
    if (dot(wfrom, it.ng) < 0.0f) {
      int idx = -1;
      for (int i = 0; i < n; ++i) if (geom[i] == int(it.geom)) { idx = i; break; }
      if (idx == -1 || n == 1) return 1.0f;
      return idx == 0 ? ior[1] : ior[0];
    }
    return n == 0 ? 1.0f : ior[0];
  }
  // sampleOrGetWavelength, LightRayInfo.cpp:52-79
  __device__ float sample_wavelength(Rng& r, bool vary) {
    if (wl == -1 && vary) {
      float p3 = 1.0f / 3.0f;
      float xi = r.u01();
      if (xi < p3) wl = 0; else if (xi < p3 + p3) wl = 1; else wl = 2;
      return p3;
    }
    return 1.0f;
  }
  // updateMedia, LightRayInfo.cpp:8-38; returns 1 when a push overflowed
  __device__ int update(const SceneDev& sc, const MaterialDev& m, const Inter& it, V3 wfrom, V3 wto) {
    float nf = dot(it.ng, wfrom), nt = dot(it.ng, wto);
    if (nf >= 0.0f && nt < 0.0f) {
      if (n >= kMaxMedia) return 1;
      T[n] = mat_albedo(sc, m, it); ior[n] = mat_ior(m, wl); geom[n] = int(it.geom); ++n;
    } else if (nf < 0.0f && nt >= 0.0f) {
      for (int i = 0; i < n; ++i) {
        if (geom[i] == int(it.geom)) {
          for (int j = i; j < n - 1; ++j) { T[j] = T[j + 1]; ior[j] = ior[j + 1]; geom[j] = geom[j + 1]; }
          --n;
          break;
        }
      }
    }
    return 0;
  }
};

// PrincipledBRDF::hasDiffuseLobe, BRDF.cpp:743-750
__device__ __forceinline__ bool has_diffuse_lobe(const SceneDev& sc, const MaterialDev& m, const Inter& it) {
  float met = mat_scalar(sc, m.metallic, m.metallic_tex, it);
  return (1.0f - 0.5f * m.specular) * (1.0 - double(m.transmission)) * (1.0 - double(met)) > 0.0f;
}

// Scene::sampleBRDFConcentrated, Scene.cpp:339-352
__device__ __forceinline__ BsdfSample sample_concentrated(const SceneDev& sc, const MaterialDev& m, const Inter& it, V3 wo,
                                                          PmMedia& lr, Rng& r, bool adjoint, int& capped) {
  float prob = lr.sample_wavelength(r, m.vary_ior != 0);
  float eta_out = lr.outside_ior(it, wo);
  const ShadeCtx cx = shade_ctx(sc, m, it, wo);
  const Prob p = lobe_probability(cx, m, mat_ior(m, lr.wl), eta_out, kLobeConcentrated);
  BsdfSample s = bsdf_sample(cx, m, it, wo, lr.wl, eta_out, p, r, capped, adjoint);
  s.thrD = s.thrD / prob;
  s.thrC = s.thrC / prob;
  return s;
}

// ---- footprint: computeRadiusPixelFootPrint (PhotonMapping.cpp:578-651) ----
__global__ void __launch_bounds__(128) k_pm_footprint(SceneDev sc, uint64_t seed, float* dist) {
  const int npix = sc.width * sc.height;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npix) return;
  const int i = p % sc.width, j = p / sc.width;
  Rng r; r.seed(path_key(seed, uint32_t(p), kFootprintPass));
  V3 o, d; int capped = 0;
  camera_ray(sc.cam, r, float(i) + 0.5f, float(j) + 0.5f, float(sc.width), float(sc.height), o, d, capped);
  Hit h = trace_ray(sc, o, d);
  if (h.tri < 0) { dist[p] = -1.0f; return; }
  Inter it = inter_from_hit(sc, h.tri, h.u, h.v);
  float dd = norm(ld3(sc.cam.pos) - it.x);
  if (!has_diffuse_lobe(sc, sc.mats[it.mat], it)) {
    for (int k = 0; k < sc.max_depth; k++) {
      const MaterialDev& m = sc.mats[it.mat];
      if (has_diffuse_lobe(sc, m, it)) break;
      V3 wo = -d;
      BsdfSample s;
      int tries = 0;
      do {
        PmMedia fresh;
        s = sample_concentrated(sc, m, it, wo, fresh, r, false, capped);
        tries += 1;
      } while (is_zero(s.thrC) && tries < 3);
      if (is_zero(s.thrC)) break;
      V3 o2 = ray_x(it, s.outside);
      Hit h2 = trace_ray(sc, o2, s.dir);
      if (h2.tri < 0 || h2.tri == it.tri) { dist[p] = -1.0f; return; }
      Inter it2 = inter_from_hit(sc, h2.tri, h2.u, h2.v);
      dd += norm(it.x - it2.x);
      it = it2;
      d = s.dir;
    }
  }
  dist[p] = dd;
}

// ---- photon tracing: sampleLightRay + tracePhoton(causticsMap = true) -------
// Scene.cpp:527-537 and PhotonMapping.cpp:191-270. Persistent: every lane
// carries one photon and, when its photon ends, takes the next emission
// index from `out.fetch`, so warps stay full although most photons end at
// their first diffuse hit and a few bounce through glass and metal. Each
// round of the loop traces one segment per lane and processes the vertex
// it reaches; the random stream is drawn in tracePhoton's order.
template <int KIND>
__global__ void __launch_bounds__(kStageThreads, 1) k_pm_emit(SceneDev sc, uint64_t seed, uint32_t iter, uint32_t first, uint32_t n,
                                                 float minQ, PmEmitOut out) {
  __shared__ WarpRays s_rays[kStageThreads / 32];
  __shared__ int s_more;
  WarpRays& w = s_rays[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u;
  const int ray = int(2 * lane);
  bool active = false, drained = false;
  uint32_t k = 0, stored = 0;
  Rng r;
  V3 flux, tt;
  PmMedia lr;
  int depth = 0, prev_tri = -1, pend_ovf = 0;
  bool first_seg = true;
  int capped = 0, overflow = 0;                 // this lane's photon
  uint32_t n_ovf = 0, n_cap = 0;                // photons of this lane with either
  for (;;) {
    if (!drained) {
      const unsigned idle = __ballot_sync(kFull, !active);
      const uint32_t n_idle = uint32_t(__popc(idle));
      if (n_idle) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(out.fetch, n_idle);
        base = __shfl_sync(kFull, base, 0);
        if (base >= n || n - base <= n_idle) drained = true;
        if (!active) {
          const uint32_t kk = base + uint32_t(__popc(idle & ((1u << lane) - 1u)));
          if (kk < n) {
            // sampleLightRay: area-weighted light triangle, uniform point, cosine direction
            k = kk;
            r.seed(path_key(seed ^ kPhotonKeyMix, first + k, iter));
            capped = overflow = 0;
            const uint32_t li_k = sample_cdf(sc.light_cdf, uint32_t(sc.n_light_tris), r, sc.light_guide, sc.light_guide_log2);
            const int ltri = sc.light_tris[li_k];
            TriRec lrec = tri_record(sc, ltri);
            lrec.ng = normalize(cross(lrec.x1 - lrec.x0, lrec.x2 - lrec.x0));
            const V3 bb = triangle_uniform(r);
            const Inter li = make_inter(sc, ltri, lrec, bb);
            float pdir;
            const V3 dir = hemisphere_cos(r, li.ng, pdir, capped);
            const V3 Le = ld3(sc.mats[li.mat].emission) * HINVPI_F;
            flux = Le * (fabsf(dot(li.ng, dir)) / (sc.light_pdf_area * pdir));
            w.put(ray, ray_x(li, true), dir);
            lr = PmMedia();
            depth = 0; stored = 0; prev_tri = -1; pend_ovf = 0;
            first_seg = true;
            active = true;
          }
        }
      }
    }
    if (threadIdx.x == 0) s_more = 0;
    __syncthreads();
    if (active || !drained) s_more = 1;
    __syncthreads();
    if (!s_more) break;
    trace_stage<KIND>(sc, w, active, false);
    __syncthreads();
    bool end = false, sample = false;
    if (active) {
      const Hit h = w.result(ray);
      const V3 o = w.origin(ray), d = w.dir(ray);
      Inter it;
      if (first_seg) {
        if (h.tri < 0) {
          end = true;
        } else {
          it = inter_from_hit(sc, h.tri, h.u, h.v);
          flux = cwise(flux, beers(lr.transmittance(), norm(it.x - o)));
        }
      } else if (h.tri < 0 || h.tri == prev_tri) {
        end = true;
      } else {
        // the previous vertex's medium update (already applied) counts once the ray arrives
        it = inter_from_hit(sc, h.tri, h.u, h.v);
        overflow |= pend_ovf;
        tt = cwise(tt, beers(lr.transmittance(), norm(it.x - o)));
        const float q = fmaxf(minQ, 1.0f - norm(tt));
        if (r.u01() <= q) {
          end = true;
        } else {
          flux = cwise(flux, tt) / (1.0f - q);
          depth += 1;
        }
      }
      // the vertex at `depth`: one round of tracePhoton's loop, its sampling in a
      // stage of its own (4 x 0.88M photons: 4.32 -> 3.41 ms)
      if (!end && (depth >= sc.max_depth || !(isfinite(flux.x) && isfinite(flux.y) && isfinite(flux.z)))) end = true;
      if (!end) {
        const MaterialDev& m = sc.mats[it.mat];
        const V3 wo = -d;
        if (has_diffuse_lobe(sc, m, it) && depth > 0) {
          const uint32_t slot = atomicAdd(out.count, 1u);
          if (slot < out.cap) {
            PhotonRec rec;
            rec.xn = make_float4(it.x.x, it.x.y, it.x.z, dot(it.ng, wo));
            rec.wi = make_float4(wo.x, wo.y, wo.z, __uint_as_float(first + k));
            rec.flux = make_float4(flux.x, flux.y, flux.z, __uint_as_float(stored));   // k-th photon of this emission
            out.photons[slot] = rec;
          }
          ++stored;
        }
        sample = true;
      }
    }
    __syncthreads();
    if (sample) {
      const Hit h = w.result(ray);
      const Inter it = inter_from_hit(sc, h.tri, h.u, h.v);
      const MaterialDev& m = sc.mats[it.mat];
      const V3 wo = -w.dir(ray);
      const BsdfSample bs = sample_concentrated(sc, m, it, wo, lr, r, true, capped);
      tt = bs.thrD + bs.thrC;
      if (is_zero(tt)) {
        end = true;
      } else {
        pend_ovf = lr.update(sc, m, it, wo, bs.dir);
        w.put(ray, ray_x(it, bs.outside), bs.dir);
        prev_tri = it.tri;
        first_seg = false;
      }
    }
    if (active && end) {
      out.stored[k] = uint8_t(stored < 255u ? stored : 255u);
      n_ovf += overflow ? 1u : 0u;
      n_cap += capped ? 1u : 0u;
      active = false;
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    n_ovf += __shfl_down_sync(kFull, n_ovf, off);
    n_cap += __shfl_down_sync(kFull, n_cap, off);
  }
  if (lane == 0) {
    if (n_ovf) atomicAdd(&out.stats[0], (unsigned long long)n_ovf);
    if (n_cap) atomicAdd(&out.stats[1], (unsigned long long)n_cap);
  }
}

// ---- gather: pathTraceWithCausticsMap (PhotonMapping.cpp:404-503) -----------
// Light from one sampling strategy's child is accumulated into its parent in
// the reference's order; the walk keeps, per continuing vertex, the partial
// sums after its light-strategy child and the weights of its BSDF child, and
// adds the BSDF child's result on the way back up.
struct PmRes { V3 pf, ll, lr, ls; int M; };
struct PmFrame { V3 pf, lr, ls, tD, tC; int M; };

// First cell of the photon map not before (x, y, z) in lexicographic order.
__device__ __forceinline__ int lower_cell(const PmMapDev& map, int n_cells, int x, int y, int z) {
  int lo = 0, hi = n_cells;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    int4 c = map.cells[mid];
    bool less = c.x < x || (c.x == x && (c.y < y || (c.y == y && c.z < z)));
    if (less) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Photons [q, qe) of the map's cells (i, j, lz..hz) (within its bounds),
// which follow each other.
__device__ __forceinline__ void column_range(const PmMapDev& map, int i, int j, int lz, int hz, int& q, int& qe) {
  q = qe = 0;
  if (map.start) {
    const int ny = map.hi[1] - map.lo[1] + 1, nz = map.hi[2] - map.lo[2] + 1;
    const uint32_t* col = map.start + (int64_t(i - map.lo[0]) * ny + (j - map.lo[1])) * nz;
    q = int(col[lz - map.lo[2]]);
    qe = int(col[hz - map.lo[2] + 1]);
    return;
  }
  const int n_cells = *map.n_cells;
  const int c0 = lower_cell(map, n_cells, i, j, lz), c1 = lower_cell(map, n_cells, i, j, hz + 1);
  if (c0 >= c1) return;
  q = map.cells[c0].w;
  qe = c1 < n_cells ? map.cells[c1].w : map.n;
}

// What a vertex's photon estimate needs of it.
struct PmQuery { V3 x, ng, ns, alb; float met, specular, transmission, radius; };
constexpr int kQueryFloats = 16;

// One warp's photon search. A "column" is the cells of one (x, y) that a
// query's cube meets, whose photons follow each other in the map.
constexpr int kCols = 64;                        // columns at a time
constexpr int kTests = 128;                      // photons tested at a time
constexpr int kEval = 64;                        // photons evaluated at a time
struct WarpSearch {
  float q[kQueryFloats][32];                     // the lanes' queries
  unsigned long long first[32];                  // columns of the lanes before
  int last[32];                                  // end of the lane's columns among the current ones
  int ly[32], ny[32], lx[32], lz[32], hz[32];
  int end[kCols], photon[kCols];                 // end of the column's tests; photon of test t is t + photon
  uint8_t col_owner[kCols];
  int found[kEval + kTests];                     // photons within the radius, waiting
  uint8_t owner[kEval + kTests];
  uint8_t seg[2][32];                            // the lane's part of the evaluated photons
  float term[kEval][3];
};
union WarpShared {
  WarpRays rays;                                 // dead during the search
  WarpSearch search;
};

// Evaluates the first n waiting photons (their lanes add them in order).
__device__ __forceinline__ void photon_evaluate(const PmMapDev& map, WarpSearch& s, int n, V3& est, int& count) {
  const int lane = int(threadIdx.x & 31u);
  s.seg[0][lane] = s.seg[1][lane] = 0;
  __syncwarp();
  float xw[kEval / 32];
  float4 pw[kEval / 32], pf[kEval / 32];
#pragma unroll
  for (int k = 0; k < kEval / 32; ++k) {
    const int e = 32 * k + lane;
    if (e < n) {
      const size_t ph = size_t(s.found[e]);
      xw[k] = __ldg(&map.pos[ph].w);
      pw[k] = __ldg(&map.rest[2 * ph]);
      pf[k] = __ldg(&map.rest[2 * ph + 1]);
    }
  }
#pragma unroll
  for (int k = 0; k < kEval / 32; ++k) {
    const int e = 32 * k + lane;
    if (e >= n) continue;
    const int o = s.owner[e];
    if (e == 0 || s.owner[e - 1] != o) s.seg[0][o] = uint8_t(e);
    if (e == n - 1 || s.owner[e + 1] != o) s.seg[1][o] = uint8_t(e + 1);
    const V3 ng(s.q[3][o], s.q[4][o], s.q[5][o]), ns(s.q[6][o], s.q[7][o], s.q[8][o]), alb(s.q[9][o], s.q[10][o], s.q[11][o]);
    const V3 wi(pw[k].x, pw[k].y, pw[k].z);
    const float nswi = dot(ns, wi);
    const float nsc = normal_scale(wi, ns, ng);
    const V3 fD = eval_diffuse(nswi, alb, nsc, s.q[12][o], s.q[13][o], s.q[14][o]);
    const float fc = fabsf(dot(wi, ng)) / (1e-7f + fabsf(xw[k]));
    const V3 t = cwise(V3(pf[k].x, pf[k].y, pf[k].z) * fc, fD + V3());
    s.term[e][0] = t.x; s.term[e][1] = t.y; s.term[e][2] = t.z;
  }
  __syncwarp();
  const int b = s.seg[0][lane], e = s.seg[1][lane];
  for (int k = b; k < e; ++k) est = est + V3(s.term[k][0], s.term[k][1], s.term[k][2]);
  count += e - b;
  __syncwarp();
}

// photonMapFluxEstimate (PhotonMapping.cpp:271-302) with the hash-cell radius
// search (HashCells.h:71-101) for the lanes that `need` it: cells in (x, y,
// z) order, photons in the order they were stored. The warp shares the work
// of its lanes' queries: their columns, then the columns' photons and then
// those within the radius are each one list taken 32 * k at a time, so every
// load has the whole warp behind it; the terms return to the query's lane,
// which adds them in list order. All lanes call it.
// What bounds it is the latency of the dependent loads (column, photon,
// photon's flux): a search by each lane for itself met it some 75 times per
// warp (387,000 queries with 9 columns, 54 photons and 19 within the radius
// each: 107,000 cycles per warp) and took 8.7 of the gather's 12 ms in four
// iterations of the 640x480 room; this one takes 3.2 of 6.4.
__device__ V3 photon_estimate(const PmMapDev& map, const PmQuery& v, bool need, WarpSearch& s, int& count) {
  const int lane = int(threadIdx.x & 31u);
  V3 est;
  __syncwarp();
  unsigned long long mine = 0;
  if (need) {
    const V3 r3(v.radius, v.radius, v.radius), lo = v.x - r3, hi = v.x + r3;
    const int lx = max(floor_int32(lo.x / map.cell), map.lo[0]), hx = min(floor_int32(hi.x / map.cell), map.hi[0]);
    const int ly = max(floor_int32(lo.y / map.cell), map.lo[1]), hy = min(floor_int32(hi.y / map.cell), map.hi[1]);
    const int lz = max(floor_int32(lo.z / map.cell), map.lo[2]), hz = min(floor_int32(hi.z / map.cell), map.hi[2]);
    if (lx <= hx && ly <= hy && lz <= hz) {
      const unsigned ny = unsigned(hy) - unsigned(ly) + 1u;
      mine = (unsigned long long)(unsigned(hx) - unsigned(lx) + 1u) * ny;
      s.lx[lane] = lx; s.ly[lane] = ly; s.ny[lane] = int(ny); s.lz[lane] = lz; s.hz[lane] = hz;
      const float f[kQueryFloats] = {v.x.x, v.x.y, v.x.z, v.ng.x, v.ng.y, v.ng.z, v.ns.x, v.ns.y, v.ns.z,
                                     v.alb.x, v.alb.y, v.alb.z, v.met, v.specular, v.transmission, v.radius * v.radius};
#pragma unroll
      for (int k = 0; k < kQueryFloats; ++k) s.q[k][lane] = f[k];
    }
  }
  unsigned long long upto = mine;                // columns of the lanes up to this one
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned long long a = __shfl_up_sync(kFull, upto, off);
    if (lane >= off) upto += a;
  }
  s.first[lane] = upto - mine;
  const unsigned long long all = __shfl_sync(kFull, upto, 31);
  int n_found = 0;
  for (unsigned long long c0 = 0; c0 < all;) {
    // Columns c0.. of the warp; one at a time where the tests of kCols columns
    // might not fit an int.
    const int nc = map.n < (1 << 24) ? int(all - c0 < kCols ? all - c0 : kCols) : 1;
    s.last[lane] = upto <= c0 ? 0 : int(upto - c0 < kCols ? upto - c0 : kCols);
    __syncwarp();
    int off[kCols / 32], len[kCols / 32];
#pragma unroll
    for (int k = 0; k < kCols / 32; ++k) {
      const int c = 32 * k + lane;
      off[k] = len[k] = 0;
      if (c < nc) {
        int o = 0;                               // first lane with last > c
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) if (s.last[o + step - 1] <= c) o += step;
        const unsigned long long at = c0 + unsigned(c) - s.first[o];
        const unsigned ny = unsigned(s.ny[o]);
        unsigned di, dj;
        if (at >> 32) { di = unsigned(at / ny); dj = unsigned(at % ny); }
        else { di = unsigned(at) / ny; dj = unsigned(at) - di * ny; }
        int qe;
        column_range(map, int(unsigned(s.lx[o]) + di), int(unsigned(s.ly[o]) + dj), s.lz[o], s.hz[o], off[k], qe);
        len[k] = qe - off[k];
        s.col_owner[c] = uint8_t(o);
      }
    }
    int total = 0;
#pragma unroll
    for (int k = 0; k < kCols / 32; ++k) {
      int incl = len[k];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int a = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += a;
      }
      s.end[32 * k + lane] = total + incl;
      s.photon[32 * k + lane] = off[k] - (total + incl - len[k]);
      total += __shfl_sync(kFull, incl, 31);
    }
    __syncwarp();
    int t0 = 0;
    do {
      int ph[kTests / 32], o[kTests / 32];
      float4 xn[kTests / 32];
#pragma unroll
      for (int k = 0; k < kTests / 32; ++k) {
        const int t = t0 + 32 * k + lane;
        o[k] = 0;
        if (t < total) {
          int c = 0;                             // first column with end > t
#pragma unroll
          for (int step = kCols / 2; step > 0; step >>= 1) if (s.end[c + step - 1] <= t) c += step;
          ph[k] = t + s.photon[c];
          o[k] = s.col_owner[c];
          xn[k] = __ldg(&map.pos[ph[k]]);
        }
      }
#pragma unroll
      for (int k = 0; k < kTests / 32; ++k) {
        const bool in = t0 + 32 * k + lane < total &&
                        norm_sq(V3(xn[k].x, xn[k].y, xn[k].z) - V3(s.q[0][o[k]], s.q[1][o[k]], s.q[2][o[k]])) <= s.q[15][o[k]];
        const unsigned hit = __ballot_sync(kFull, in);
        if (in) {
          const int at = n_found + __popc(hit & ((1u << lane) - 1u));
          s.found[at] = ph[k];
          s.owner[at] = uint8_t(o[k]);
        }
        n_found += __popc(hit);
      }
      __syncwarp();
      t0 += kTests;
      while (n_found >= kEval) {
        photon_evaluate(map, s, kEval, est, count);
        n_found -= kEval;
        // the ones that wait move up
#pragma unroll
        for (int k = 0; k < kTests / 32; ++k) {
          const int e = 32 * k + lane;
          int f = 0;
          uint8_t w = 0;
          if (e < n_found) { f = s.found[kEval + e]; w = s.owner[kEval + e]; }
          __syncwarp();
          if (e < n_found) { s.found[e] = f; s.owner[e] = w; }
          __syncwarp();
        }
      }
    } while (t0 < total);
    c0 += unsigned(nc);
    __syncwarp();
  }
  if (n_found > 0) photon_evaluate(map, s, n_found, est, count);
  return est;
}

// Pixel p's new statistics and image values: the chain of frames unwound from
// the path's last vertex `leaf`, then PMRenderJob's update.
__device__ __forceinline__ void finish_pixel(const PmPixelsDev& px, int p, const PmFrame* fr, int top, const PmRes& leaf,
                                             float radius, V3 normal, V3 albedo, int emitted) {
  // back up the chain: each continuing vertex adds its BSDF child's result
  PmRes res = leaf;
  for (int k = top; k >= 0; --k) {
    const PmFrame& F = fr[k];
    const V3 t2 = F.tD + F.tC;
    PmRes up;
    up.ls = F.ls + cwise(res.ll + res.ls, F.tC);
    up.lr = F.lr + (cwise(res.lr, t2) + cwise(res.ll, F.tD));
    up.pf = F.pf + cwise(res.pf, t2);
    up.M = F.M + res.M;
    up.ll = V3();
    res = up;
  }
  // PMRenderJob::unlockAndUpdateStatistic (PhotonMapping.h:62-106) or unlock
  const V3 L = res.ll + res.lr + res.ls;
  float4 ls4 = px.lsum[p];
  V3 LSum(ls4.x, ls4.y, ls4.z);
  int Nd = __float_as_int(ls4.w);
  V3 Lnew;
  if (has_nan(L) || has_nan(res.pf)) {
    Lnew = LSum / (1e-7f + float(Nd));
  } else {
    const float alpha = 0.4f;
    const int M = res.M;
    float prad = px.radius[p], pN = px.N[p], pNe = px.Ne[p];
    float4 f4v = px.flux[p];
    V3 pflux(f4v.x, f4v.y, f4v.z);
    LSum = LSum + L;
    Nd += 1;
    V3 Lflux;
    if (prad < 0.0f) {
      if (!(radius < 0.0f)) {
        prad = radius;
        pN += alpha * M;
        pNe += emitted;
        pflux = res.pf;
        Lflux = pNe == 0 ? V3() : pflux / (prad * prad * HPI_F * pNe);
      }
    } else {
      float rold = prad;
      float Ni = pN;
      if (Ni + M > 0) prad *= sqrtf((Ni + alpha * M) / (Ni + M));
      pN += alpha * M;
      pNe += emitted;
      pflux = (pflux + res.pf) * (prad * prad) / (rold * rold);
      Lflux = pNe == 0 ? V3() : pflux / (prad * prad * HPI_F * pNe);
      radius = prad;
    }
    Lnew = Lflux + LSum / float(Nd);
    px.radius[p] = prad; px.N[p] = pN; px.Ne[p] = pNe;
    px.flux[p] = make_float4(pflux.x, pflux.y, pflux.z, 0.f);
    px.lsum[p] = make_float4(LSum.x, LSum.y, LSum.z, __int_as_float(Nd));
  }
  px.radii[p] = radius;
  px.color[3 * p] = Lnew.x; px.color[3 * p + 1] = Lnew.y; px.color[3 * p + 2] = Lnew.z;
  px.normal[3 * p] = normal.x; px.normal[3 * p + 1] = normal.y; px.normal[3 * p + 2] = normal.z;
  px.albedo[3 * p] = albedo.x; px.albedo[3 * p + 1] = albedo.y; px.albedo[3 * p + 2] = albedo.z;
}

// A pixel's path between two stages: the vertex whose light and BSDF rays are
// being traced.
struct PmVertex {
  PmRes R;                   // the vertex's own sums
  V3 thr;                    // transmittance (and roulette) factor
  V3 fD, fC, TL;             // light ray: lobes, transmittance of its medium
  V3 tDB, tCB;               // BSDF ray: lobe weights
  float cosL, pBL, pdfB;     // light ray: |cos| and BSDF pdf; BSDF ray: its pdf
  int tri, ltri;             // the vertex's triangle; the light triangle sampled (-1: environment)
};

// One persistent thread per pixel's path; a thread whose path has ended takes
// the next pixel. A round: closest hits of the pending rays (the camera ray,
// or a vertex's light and BSDF rays); the vertex's two children and the next
// vertex; its photon estimate; its samples. Random numbers are drawn
// in the reference's order (the light ray's result draws none).
template <int KIND>
__global__ void __launch_bounds__(kStageThreads, 1) k_pm_gather(SceneDev sc, PmMapDev map, PmPixelsDev px, uint64_t seed, uint32_t iter,
                                                   float ox, float oy, int emitted, unsigned long long* stats,
                                                   uint32_t* fetch) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  WarpShared* s_warp = reinterpret_cast<WarpShared*>(s_dyn);
  __shared__ int s_more;
  WarpRays& w = s_warp[threadIdx.x >> 5].rays;
  const uint32_t lane = threadIdx.x & 31u;
  const int rB = int(2 * lane), rL = rB + 1;
  const uint32_t npix = uint32_t(sc.width) * uint32_t(sc.height);
  const bool two = sc.two_strategies != 0;
  uint32_t n_ovf = 0, n_cap = 0;                // pixels of this lane with either
  int p = -1;                                   // this lane's pixel
  bool drained = false;                         // warp-uniform
  bool pendB = false, pendL = false, camera = false;
  Rng r;
  int capped = 0, overflow = 0, ovB = 0, ovL = 0, depth = 0, top = -1;
  float radius = 0.0f;
  V3 normal, albedo;
  PmMedia lr;
  PmVertex v;
  PmFrame fr[kPmMaxDepth];
  for (;;) {
    // ---- new pixels for lanes without one
    const unsigned need = __ballot_sync(kFull, p < 0);
    if (need && !drained) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(fetch, uint32_t(__popc(need)));
      base = __shfl_sync(kFull, base, 0);
      if (base >= npix || npix - base <= uint32_t(__popc(need))) drained = true;
      const uint32_t k = base + uint32_t(__popc(need & ((1u << lane) - 1u)));
      if (p < 0 && k < npix) {
        p = int(k);
        r.seed(path_key(seed, uint32_t(p), iter));
        capped = overflow = 0;
        V3 o, d;
        camera_ray(sc.cam, r, float(p % sc.width) + ox, float(p / sc.width) + oy, float(sc.width), float(sc.height), o, d, capped);
        if (px.radius[p] == -1.0f) px.radius[p] = px.radii[p];        // PMRenderJob::lock
        radius = px.radius[p];
        normal = V3(); albedo = V3();
        lr = PmMedia();
        depth = 0; top = -1;
        w.put(rB, o, d);
        pendB = camera = true;
        pendL = false;
      }
    }
    if (threadIdx.x == 0) s_more = 0;
    __syncthreads();
    if (p >= 0 || !drained) s_more = 1;
    __syncthreads();
    if (!s_more) break;
    // ---- closest hits
    trace_stage<KIND>(sc, w, pendB, pendL);
    __syncthreads();
    // ---- the children of the vertex the rays left
    bool end = false;                           // the path's last vertex is `leaf`
    PmRes leaf;
    leaf.M = 0;
    Hit h;
    h.tri = -1;
    if (p >= 0 && !camera) {
      float pdfs[2] = {0.0f, 0.0f};
      if (pendL) {                              // LightSamplingStrategy::sample, MIS.cpp:32-54
        const Hit hL = w.result(rL);
        const V3 oL = w.origin(rL), dL = w.dir(rL);
        TriRec recL;
        recL.mat = -1;
        V3 x2;
        if (hL.tri >= 0) { recL = tri_record(sc, hL.tri); x2 = tri_point(recL, hit_weights(hL.u, hL.v)); }
        bool vis = v.ltri >= 0 ? hL.tri == v.ltri : (hL.tri < 0 || sc.mats[recL.mat].is_light);
        float pdfL = vis ? light_density(sc, oL, dL, recL.mat, x2, recL.ng) : 0.0f;
        V3 tDL, tCL;
        if (vis && pdfL != 0.0f) {
          float mm = v.cosL / pdfL;
          tDL = v.fD * mm; tCL = v.fC * mm;
        }
        pdfs[0] = pdfL;
        if (!is_zero(tDL + tCL) && hL.tri != v.tri) {
          pdfs[1] = v.pBL;
          float ssum = 0.0f;
          for (int k = 0; k < 2; ++k) ssum += pdfs[k] * pdfs[k];
          float wt = pdfs[0] * pdfs[0] / ssum;
          overflow |= ovL;
          V3 tD = cwise(v.thr, tDL) * wt, tC = cwise(v.thr, tCL) * wt, t2 = tD + tC;
          PmRes rs; rs.M = 0;                   // the light child (a light or the sky)
          if (depth + 1 < sc.max_depth) {
            if (hL.tri < 0) {
              rs.lr = cwise(beers(v.TL, 1e6f), env_eval(sc, dL));
            } else if (sc.mats[recL.mat].is_light) {
              rs.ll = rs.ll + cwise(beers(v.TL, norm(x2 - oL)), emission(sc, recL.mat, recL.ng, -dL));
            }
          }
          v.R.ls = v.R.ls + cwise(rs.ll + rs.ls, tC);
          v.R.lr = v.R.lr + (cwise(rs.lr, t2) + cwise(rs.ll, tD));
          v.R.pf = v.R.pf + cwise(rs.pf, t2);
          v.R.M += rs.M;
        }
      }
      // BRDFSamplingStrategy::sample, MIS.cpp:6-26
      if (pendB) h = w.result(rB);
      if (pendB && h.tri != v.tri && top + 1 < kPmMaxDepth) {
        const int sb = two ? 1 : 0;
        pdfs[sb] = v.pdfB;
        if (two) {
          TriRec recB;
          recB.mat = -1;
          V3 xB;
          if (h.tri >= 0) { recB = tri_record(sc, h.tri); xB = tri_point(recB, hit_weights(h.u, h.v)); }
          pdfs[0] = light_density(sc, w.origin(rB), w.dir(rB), recB.mat, xB, recB.ng);
        }
        int ns = two ? 2 : 1;
        float ssum = 0.0f;
        for (int k = 0; k < ns; ++k) ssum += pdfs[k] * pdfs[k];
        float wt = pdfs[sb] * pdfs[sb] / ssum;
        overflow |= ovB;
        PmFrame& F = fr[++top];
        F.pf = v.R.pf; F.lr = v.R.lr; F.ls = v.R.ls; F.M = v.R.M;
        F.tD = cwise(v.thr, v.tDB) * wt;
        F.tC = cwise(v.thr, v.tCB) * wt;
        ++depth;
      } else {
        leaf = v.R;
        end = true;
      }
    }
    // ---- the next vertex, up to its photon estimate
    const bool child_end = end;
    bool shade = false, need_est = false;
    Inter it;
    V3 wo;
    ShadeCtx cx;
    PmQuery qv;
    qv.radius = 0.0f;
    if (p >= 0 && !end) {
      if (camera) h = w.result(rB);
      camera = false;
      const V3 o = w.origin(rB), d = w.dir(rB);
      v.R = PmRes();
      v.R.M = 0;
      if (depth >= sc.max_depth) {
        end = true;
      } else if (h.tri < 0) {
        v.R.lr = cwise(beers(lr.transmittance(), 1e6f), env_eval(sc, d));
        if (depth == 0) { normal = V3(); albedo = v.R.lr; }
        end = true;
      } else {
        it = inter_from_hit(sc, h.tri, h.u, h.v);
        const MaterialDev& m = sc.mats[it.mat];
        if (depth == 0) { normal = it.ns; albedo = mat_albedo(sc, m, it); }
        v.thr = beers(lr.transmittance(), norm(it.x - o));
        if (m.is_light) {
          v.R.ll = v.R.ll + cwise(v.thr, emission(sc, it.mat, it.ng, -d));
          end = true;
        } else {
          wo = -d;
          cx = shade_ctx(sc, m, it, wo);
          need_est = has_diffuse_lobe(sc, m, it);
          qv.x = it.x; qv.ng = it.ng; qv.ns = cx.ns; qv.alb = cx.alb;
          qv.met = cx.met; qv.specular = m.specular; qv.transmission = m.transmission; qv.radius = radius;
          shade = true;
        }
      }
    }
    __syncthreads();
    // ---- its photon estimate and roulette
    {
      int cnt = 0;
      const V3 est = photon_estimate(map, qv, need_est, s_warp[threadIdx.x >> 5].search, cnt);
      if (need_est) {
        v.R.M += cnt;
        v.R.pf = v.R.pf + cwise(v.thr, est);
      }
    }
    if (shade) {
      float q = depth >= sc.rr_start ? sc.rr_q : 0.0f;
      if (r.u01() <= q) {
        end = true;
        shade = false;
      } else {
        v.thr = v.thr / (1.0f - q);
      }
    }
    if (end && !child_end) leaf = v.R;
    pendB = pendL = false;
    __syncthreads();
    // ---- its light and BSDF samples
    if (shade) {
      const MaterialDev& m = sc.mats[it.mat];
      v.tri = it.tri;
      ovB = ovL = 0;
      if (two) {
        float xi = r.u01();
        V3 oL, dL;
        v.ltri = -1;
        if (xi < sc.p_surface) {
          uint32_t kk = sample_cdf(sc.light_cdf, uint32_t(sc.n_light_tris), r, sc.light_guide, sc.light_guide_log2);
          v.ltri = sc.light_tris[kk];
          V3 bb = triangle_uniform(r);
          V3 xl = tri_point(tri_record(sc, v.ltri), bb);
          oL = ray_x(it, dot(it.ng, xl - it.x) >= 0.0f);
          dL = normalize(xl - oL);
        } else {
          float dens;
          dL = env_sample(sc, r, dens, capped);
          oL = ray_x(it, dot(it.ng, dL) >= 0.0f);
        }
        const BsdfEval ev = bsdf_eval(cx, m, it, wo, dL);
        if (!(is_zero(ev.fD) && is_zero(ev.fC))) {
          v.fD = ev.fD; v.fC = ev.fC;
          v.cosL = fabsf(dot(dL, it.ng));
          v.pBL = bsdf_pdf(cx, lobe_probability(cx, m, m.ior, lr.outside_ior(it, wo)), wo, dL);
          PmMedia lrL = lr;
          ovL = lrL.update(sc, m, it, wo, dL);
          v.TL = lrL.transmittance();
          w.put(rL, oL, dL);
          pendL = true;
        }
      }
      float prob = lr.sample_wavelength(r, m.vary_ior != 0);
      float eta_out = lr.outside_ior(it, wo);
      BsdfSample bs = bsdf_sample(cx, m, it, wo, lr.wl, eta_out, lobe_probability(cx, m, mat_ior(m, lr.wl), eta_out), r, capped);
      v.tDB = bs.thrD / prob;
      v.tCB = bs.thrC / prob;
      v.pdfB = bs.pdf;
      if (bs.pdf != 0.0f && !is_zero(v.tDB + v.tCB)) {
        w.put(rB, ray_x(it, bs.outside), bs.dir);
        pendB = true;
        // the medium the path continues in (the update counts once it does)
        ovB = lr.update(sc, m, it, wo, bs.dir);
      }
      if (!pendB && !pendL) { leaf = v.R; end = true; }
    }
    __syncthreads();
    if (end) {
      finish_pixel(px, p, fr, top, leaf, radius, normal, albedo, emitted);
      n_ovf += overflow ? 1u : 0u;
      n_cap += capped ? 1u : 0u;
      p = -1;
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    n_ovf += __shfl_down_sync(kFull, n_ovf, off);
    n_cap += __shfl_down_sync(kFull, n_cap, off);
  }
  if (lane == 0) {
    if (n_ovf) atomicAdd(&stats[0], (unsigned long long)n_ovf);
    if (n_cap) atomicAdd(&stats[1], (unsigned long long)n_cap);
  }
}

}  // namespace

void launch_pm_footprint(const SceneDev& sc, uint64_t seed, float* dist, cudaStream_t st) {
  const int npix = sc.width * sc.height;
  k_pm_footprint<<<(npix + 127) / 128, 128, 0, st>>>(sc, seed, dist);
}

namespace {
// Launch of a staged kernel over n photons or pixels: one block per SM, its
// threads no more than an even share of n (whole warps).
struct StageGrid { int blocks, threads; };
StageGrid stage_grid(int64_t n) {
  static const int sms = [] {
    int dev = 0, count = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    return std::max(1, count);
  }();
  const int64_t warps = (n + 31) / 32, per_block = std::min<int64_t>((warps + sms - 1) / sms, kStageThreads / 32);
  return {int(std::min<int64_t>((warps + per_block - 1) / per_block, sms)), int(per_block) * 32};
}
}  // namespace

void launch_pm_emit(const SceneDev& sc, uint64_t seed, uint32_t iter, uint32_t first, uint32_t n, float min_q,
                    const PmEmitOut& out, cudaStream_t st) {
  if (n == 0) return;
  cudaMemsetAsync(out.fetch, 0, sizeof(uint32_t), st);
  const StageGrid g = stage_grid(n);
  if (sc.bvh_kind == 1) k_pm_emit<1><<<g.blocks, g.threads, 0, st>>>(sc, seed, iter, first, n, min_q, out);
  else k_pm_emit<0><<<g.blocks, g.threads, 0, st>>>(sc, seed, iter, first, n, min_q, out);
}

void launch_pm_gather(const SceneDev& sc, const PmMapDev& map, const PmPixelsDev& px, uint64_t seed, uint32_t iter,
                      float ox, float oy, int emitted, unsigned long long* stats, uint32_t* fetch, cudaStream_t st) {
  const int64_t npix = int64_t(sc.width) * sc.height;
  constexpr int most = int(sizeof(WarpShared)) * (kStageThreads / 32);
  cudaFuncSetAttribute(k_pm_gather<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  cudaFuncSetAttribute(k_pm_gather<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  cudaMemsetAsync(fetch, 0, sizeof(uint32_t), st);
  const StageGrid g = stage_grid(npix);
  const int shared = int(sizeof(WarpShared)) * (g.threads / 32);
  if (sc.bvh_kind == 1) k_pm_gather<1><<<g.blocks, g.threads, shared, st>>>(sc, map, px, seed, iter, ox, oy, emitted, stats, fetch);
  else k_pm_gather<0><<<g.blocks, g.threads, shared, st>>>(sc, map, px, seed, iter, ox, oy, emitted, stats, fetch);
}

}  // namespace hasty

// Status word of this file's bounds checks (bounds-checked build).
HASTY_BOUNDS_READER(bounds_status_photon)
