// Closest-hit traversal of the compressed 8-wide BVH and the binary BVH
// (per-ray step machines, exact ray/triangle test), host + device. Shared by
// the closest-hit kernels (trace.cu) and the photon mapper (photon.cu); every
// including translation unit gets its own copy (anonymous namespace). All
// rounding is explicit (mulr/addr/subr/divr, fmaf), so the results do not
// depend on the compiler's FMA contraction setting.
//
// The ray/triangle test is Moeller-Trumbore in Embree's sign conventions and
// rounds every product and sum separately (no FMA contraction), so t, u, v
// and the chosen triangle are the ones the CPU oracle computes. The far
// limit is applied to the divided distance and ties at equal t go to the
// smaller triangle id, so the answer does not depend on traversal order.
// Binary-BVH box tests round each step once and are padded by
// 1 +/- 2*gamma(3), so no box that holds the closest hit is culled by
// rounding (Ize 2013); the wide BVH's one-FMA child planes carry an absolute
// error bound instead (plane_terms). The far limit at the current closest
// hit is padded by 1 + 2*gamma(3) in both.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstring>

#include "bounds.cuh"
#include "hasty_types.h"

namespace hasty {
namespace {

#define HDI __host__ __device__ __forceinline__

constexpr unsigned kFullMask = 0xFFFFFFFFu;

struct Hit { float t, u, v; int tri; };

HDI float mulr(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  return a * b;        // host objects are built with -ffp-contract=off
#endif
}
HDI float addr(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  return a + b;
#endif
}
HDI float subr(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fsub_rn(a, b);
#else
  return a - b;
#endif
}
HDI float divr(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fdiv_rn(a, b);
#else
  return a / b;
#endif
}
HDI uint32_t f2u(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t u; std::memcpy(&u, &f, 4); return u;
#endif
}
HDI float u2f(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f; std::memcpy(&f, &u, 4); return f;
#endif
}
HDI uint32_t popc(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __popc(x);
#else
  return uint32_t(__builtin_popcount(x));
#endif
}
HDI uint32_t highest_bit(uint32_t x) {   // x != 0
#ifdef __CUDA_ARCH__
  return 31u - __clz(x);
#else
  return 31u - uint32_t(__builtin_clz(x));
#endif
}
HDI uint32_t lowest_bit(uint32_t x) {    // x != 0
#ifdef __CUDA_ARCH__
  return uint32_t(__ffs(x)) - 1u;
#else
  return uint32_t(__builtin_ctz(x));
#endif
}
// 32 bytes at a 32-byte boundary: one load on the GPU with WIDE, else two.
// Rays that read different nodes and triangles cost the L1 about one lookup
// per ray and load instruction, whatever its width, so the wide loads serve
// the persistent kernels; warps whose rays share a few nodes (tiny BVHs) are
// served faster by 16-byte loads. ms per render of closest hits, 16-byte ->
// 32-byte loads: 1.02M-triangle field 17.67 -> 17.33, textured room 2.91 ->
// 2.82, Cornell box (36 triangles) 1.81 -> 2.12.
struct Ld32 { float4 a, b; };
template <bool WIDE>
HDI Ld32 ld32(const float4* p) {
  Ld32 r;
#ifdef __CUDA_ARCH__
  if (WIDE) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y), "=f"(r.b.z), "=f"(r.b.w)
        : "l"(p));
  } else {
    r.a = __ldg(p); r.b = __ldg(p + 1);
  }
#else
  r.a = p[0]; r.b = p[1];
#endif
  return r;
}
HDI float dotr(float ax, float ay, float az, float bx, float by, float bz) {
  return addr(addr(mulr(ax, bx), mulr(ay, by)), mulr(az, bz));
}

// Leaf-ordered triangle ti (kLeafTriWords), its normal as the layout writers
// round it: e2 x e1, every product and difference once.
template <bool WIDE>
HDI void tri_test(float ox, float oy, float oz, float dx, float dy, float dz, const float4* tris, int ti, Hit& best) {
  const float4* tp = tris + kLeafTriWords / 4 * int64_t(ti);
  const Ld32 t0 = ld32<WIDE>(tp), t1 = ld32<WIDE>(tp + 2);
  const float4 v0 = t0.a, e1 = t0.b, e2 = t1.a;
  const float nx = e1.w, ny = e2.w, nz = t1.b.x;
  float cx = subr(v0.x, ox), cy = subr(v0.y, oy), cz = subr(v0.z, oz);
  float rx = subr(mulr(cy, dz), mulr(cz, dy));
  float ry = subr(mulr(cz, dx), mulr(cx, dz));
  float rz = subr(mulr(cx, dy), mulr(cy, dx));
  float den = dotr(nx, ny, nz, dx, dy, dz);
  float ad = fabsf(den);
  float sg = den < 0.f ? -1.f : 1.f;
  float U = mulr(dotr(rx, ry, rz, e2.x, e2.y, e2.z), sg);
  float V = mulr(dotr(rx, ry, rz, e1.x, e1.y, e1.z), sg);
  if (!(den != 0.f && U >= 0.f && V >= 0.f && addr(U, V) <= ad)) return;
  float T = mulr(dotr(nx, ny, nz, cx, cy, cz), sg);
  if (!(mulr(ad, 1e-6f) < T)) return;
  float t = divr(T, ad);
  int id = int(f2u(v0.w));
  if (t < best.t || (t == best.t && (best.tri < 0 || id < best.tri))) {
    best.t = t; best.u = divr(U, ad); best.v = divr(V, ad); best.tri = id;
  }
}

HDI float slab(float b, float o, float id) { return mulr(subr(b, o), id); }

constexpr float kPadHi = 1.0000008f;   // 1 + 2*gamma(3), rounded up
constexpr float kPadLo = 0.9999992f;
constexpr float kInf = __builtin_huge_valf();

struct RayInv { float ix, iy, iz; };
HDI RayInv inverse_dir(float dx, float dy, float dz) {
  const float eps = 1e-20f;
  RayInv r;
  r.ix = 1.0f / (fabsf(dx) > eps ? dx : copysignf(eps, dx));
  r.iy = 1.0f / (fabsf(dy) > eps ? dy : copysignf(eps, dy));
  r.iz = 1.0f / (fabsf(dz) > eps ? dz : copysignf(eps, dz));
  return r;
}

// ---------------------------------------------------------- binary BVH ----
constexpr int kStack = 64;

// Traversal state of one ray. init() sets it up; each step() walks inner
// nodes to the next leaf, tests the leaf's triangles and pops the next
// subtree; it returns true once the ray is finished (result in `best`).
// Whole-ray traversal is init() + step() until true; the persistent GPU
// kernels interleave steps of many rays, with identical results per ray.
// The traversal stack is kept outside the struct (passed to step()) so the
// scalar state can stay in registers.
struct TravBinary {
  using Entry = int;
  static constexpr int kDepth = kStack;
  float ox, oy, oz, dx, dy, dz;
  RayInv iv;
  bool neg_x, neg_y, neg_z;
  Hit best;
  int link, sp;
  bool any;   // stop at the first triangle hit (visibility only); set after init
  bool overflow;   // a subtree was skipped because the stack was full
#ifdef HASTY_DEBUG_BOUNDS
  int32_t lim_nodes = 0x7FFFFFFF, lim_tris = 0x7FFFFFFF;   // bounds-checked build: array sizes
#endif

  HDI void init(float ox_, float oy_, float oz_, float dx_, float dy_, float dz_) {
    ox = ox_; oy = oy_; oz = oz_; dx = dx_; dy = dy_; dz = dz_;
    any = false;
    overflow = false;
    best.t = kInf; best.u = best.v = 0.f; best.tri = -1;
    iv = inverse_dir(dx, dy, dz);
    neg_x = iv.ix < 0.f; neg_y = iv.iy < 0.f; neg_z = iv.iz < 0.f;
    sp = 0;
    link = 0;   // root (always an inner node)
  }

  HDI bool step(const float4* nodes, const float4* tris, int* stack) {
    while (link >= 0) {
#ifdef HASTY_DEBUG_BOUNDS
      if (!HASTY_IN_BOUNDS(link < lim_nodes, BB_NODE)) return true;
#endif
      const Ld32 b0 = ld32<true>(&nodes[4 * link]), b1 = ld32<true>(&nodes[4 * link + 2]);
      const float4 n0 = b0.a, n1 = b0.b, n2 = b1.a, n3 = b1.b;
      float tlim = best.t * kPadHi;
      // near/far planes by the direction sign: (b - o) * id is monotonic in b,
      // so this picks exactly what per-axis min/max would
      float t0min = fmaxf(fmaxf(slab(neg_x ? n0.y : n0.x, ox, iv.ix), slab(neg_y ? n0.w : n0.z, oy, iv.iy)),
                          fmaxf(slab(neg_z ? n2.y : n2.x, oz, iv.iz), 0.0f)) * kPadLo;
      float t0max = fminf(fminf(fminf(slab(neg_x ? n0.x : n0.y, ox, iv.ix), slab(neg_y ? n0.z : n0.w, oy, iv.iy)),
                                slab(neg_z ? n2.x : n2.y, oz, iv.iz)) * kPadHi, tlim);
      float t1min = fmaxf(fmaxf(slab(neg_x ? n1.y : n1.x, ox, iv.ix), slab(neg_y ? n1.w : n1.z, oy, iv.iy)),
                          fmaxf(slab(neg_z ? n2.w : n2.z, oz, iv.iz), 0.0f)) * kPadLo;
      float t1max = fminf(fminf(fminf(slab(neg_x ? n1.x : n1.y, ox, iv.ix), slab(neg_y ? n1.z : n1.w, oy, iv.iy)),
                                slab(neg_z ? n2.z : n2.w, oz, iv.iz)) * kPadHi, tlim);
      bool h0 = t0min <= t0max, h1 = t1min <= t1max;
      int l0 = int(f2u(n3.x)), l1 = int(f2u(n3.y));
      if (h0 && h1) {
        int far_l = l1;
        link = l0;
        if (t1min < t0min) { link = l1; far_l = l0; }
        if (sp < kStack) stack[sp++] = far_l; else overflow = true;
      } else if (h0) {
        link = l0;
      } else if (h1) {
        link = l1;
      } else {
        if (sp == 0) return true;
        link = stack[--sp];
      }
    }
    // leaf: link = ~(first << 3 | count)
    int code = ~link;
    int first = code >> 3, cnt = code & 7;
    for (int k = 0; k < cnt; ++k) {
      int ti = first + k;
#ifdef HASTY_DEBUG_BOUNDS
      if (!HASTY_IN_BOUNDS(ti >= 0 && ti < lim_tris, BB_LEAF_TRI)) return true;
#endif
      tri_test<true>(ox, oy, oz, dx, dy, dz, tris, ti, best);
    }
    if (sp == 0 || (any && best.tri >= 0)) return true;
    link = stack[--sp];
    return false;
  }
};

HDI Hit trace_binary(const float4* nodes, const float4* tris, float ox, float oy, float oz, float dx, float dy, float dz) {
  TravBinary tr;
  int stack[kStack];
  tr.init(ox, oy, oz, dx, dy, dz);
  while (!tr.step(nodes, tris, stack)) {}
  return tr.best;
}

// ------------------------------------------------- compressed 8-wide BVH ----
// Node groups of Ylitie, Karras and Laine 2017: (base index, mask) where bits
// 24..31 are children still to visit, each at bit 24 + (slot ^ octant) so the
// highest bit is the nearest child, and bits 0..7 hold the parent's
// inner-child mask; for triangle groups bits 0..23 are triangles to test.
// Child boxes are decoded as the builder verified them (fma of the 8-bit
// coordinate and the power-of-two step) and tested with the padded slabs.
constexpr int kWideStack = 32;

HDI uint32_t byte_of(uint32_t w, uint32_t k) { return (w >> (8 * k)) & 0xFFu; }

// Byte k (0..7) of the 8-byte value (lo, hi).
HDI uint32_t byte_at(uint32_t lo, uint32_t hi, uint32_t k) {
#ifdef __CUDA_ARCH__
  return __byte_perm(lo, hi, k) & 0xFFu;
#else
  return byte_of(k < 4 ? lo : hi, k & 3u);
#endif
}

// x with its bits exchanged at distance d within pairs of groups (low groups
// m): d is that distance, or 0 for none.
HDI uint32_t swap_bits(uint32_t x, uint32_t d, uint32_t m) { return ((x >> d) & m) | ((x << d) & ~m); }

// 2^23 + byte k of w as a float, exactly: one byte permute places the byte
// in the mantissa of 2^23 (the offset is folded into the planes' b terms).
HDI float byte_biased(uint32_t w, uint32_t k) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(__byte_perm(w, 0x4B000000u, k | 0x7540u));
#else
  return 8388608.0f + float(byte_of(w, k));
#endif
}

// (q0, q1) * a + b, each rounded once: one packed FMA on the GPU.
HDI float2 fma2(float q0, float q1, float a, float b) {
#ifdef __CUDA_ARCH__
  uint64_t q, aa, bb, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "f"(q0), "f"(q1));
  asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a));
  asm("mov.b64 %0, {%1, %1};" : "=l"(bb) : "f"(b));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(q), "l"(aa), "l"(bb));
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(r));
  return f;
#else
  return make_float2(fmaf(q0, a, b), fmaf(q1, a, b));
#endif
}

// Same contract as TravBinary: a step tests the pending triangle group and
// opens one node.
// Per-node, per-axis terms of the child slab test t = fma(q, a, b). A child
// plane is x = fma(q, s, p0) rounded once (the float plane the layout writer
// makes conservative); the slab parameter is T = (x - o) / d. Here a = s * inv
// is exact (s is a power of two, inv = fl(1/d)) and b = (p0 - o) * inv, so
//   fma(q, a, b) = T (1 + th), |th| <= gamma(2),  plus  R,
//   |R| <= u |inv| (|p0| + 255 s + 2 |p0 - o|) (1 + 4u),  u = 2^-24,
// R coming from x's own rounding (which this form skips) and from b's two
// roundings; and |T| <= (|p0 - o| + 255 s) |inv| (1 + u). With the rounding
// of b -/+ eps, the total error is below u |inv| (|p0| + 765 s + 5 |p0 - o|)
// to first order; eps = 2^-22 |inv| (|p0| + 1024 s + 6 |p0 - o|) + 1e-37
// covers it at least twice over (the constant covers products in the
// subnormal range). Near planes use b - eps and far planes b + eps, so each
// near value is at most, and each far value at least, the exact T: the box
// test needs no further padding and culls no box the ray enters.
// (Coordinates and grid steps are assumed below 2^120, far beyond any scene.)
struct PlaneTerms { float a, b_near, b_far; };
HDI PlaneTerms plane_terms(float p0, float o, float inv, float s) {
  PlaneTerms t;
  const float d = subr(p0, o);
  const float b = mulr(d, inv);
  const float mag = fmaf(6.0f, fabsf(d), fmaf(1024.0f, s, fabsf(p0)));
  const float eps = fmaf(mulr(mag, fabsf(inv)), 2.384185791015625e-07f, 1e-37f);   // 2^-22
  t.a = mulr(s, inv);
  // The child loop evaluates fma(2^23 + q, a, b') with b' = b -/+ eps - 2^23 a
  // (2^23 a is exact; the FMA forms (2^23 + q) a exactly). The one extra
  // rounding, of b' itself, is at most u (2^23 |a| + |b| + eps) = s |inv| / 2
  // + u (|b| + eps): half a grid step, added to eps with a relative margin
  // of 1e-6; the u |b| part is inside eps's factor-two margin.
  const float half = mulr(mulr(0.5000005f, s), fabsf(inv));
  const float e = addr(eps, half);
  const float a23 = mulr(-8388608.0f, t.a);
  t.b_near = addr(subr(b, e), a23);
  t.b_far = addr(addr(b, e), a23);
  return t;
}

template <bool WIDE>
struct TravWideOf {
  using Entry = uint2;
  static constexpr int kDepth = kWideStack;
  static constexpr uint32_t kNone = 0xFFFFFFFFu;
  float ox, oy, oz, dx, dy, dz;
  RayInv iv;
  bool neg_x, neg_y, neg_z;
  uint32_t oct;
  Hit best;
  uint32_t node;   // node to open next (kNone: none left)
  uint2 tg;        // triangles to test before it
  int sp;
  // Visibility only: stop at the first triangle hit (best is then a hit,
  // not necessarily the closest). Set after init.
  bool any;
  bool overflow;   // a node group was skipped because the stack was full
#ifdef HASTY_DEBUG_BOUNDS
  int32_t lim_nodes = 0x7FFFFFFF, lim_tris = 0x7FFFFFFF;   // bounds-checked build: array sizes
#endif

  HDI void init(float ox_, float oy_, float oz_, float dx_, float dy_, float dz_) {
    ox = ox_; oy = oy_; oz = oz_; dx = dx_; dy = dy_; dz = dz_;
    any = false;
    overflow = false;
    best.t = kInf; best.u = best.v = 0.f; best.tri = -1;
    iv = inverse_dir(dx, dy, dz);
    neg_x = iv.ix < 0.f; neg_y = iv.iy < 0.f; neg_z = iv.iz < 0.f;
    oct = (neg_x ? 4u : 0u) | (neg_y ? 2u : 0u) | (neg_z ? 1u : 0u);
    sp = 0;
    node = 0;
    tg = make_uint2(0u, 0u);
  }

  // A step tests the pending triangles, opens `node` and chooses the node
  // after it. Which node that is does not depend on the triangles, so it is
  // chosen (and its line fetched ahead) before they are tested.
  HDI bool step(const float4* nodes, const float4* tris, uint2* stack) {
    while (tg.y) {
      uint32_t b = lowest_bit(tg.y);
      tg.y &= tg.y - 1u;
      int ti = int(tg.x + b);
#ifdef HASTY_DEBUG_BOUNDS
      if (!HASTY_IN_BOUNDS(ti >= 0 && ti < lim_tris, BB_LEAF_TRI)) return true;
#endif
      tri_test<WIDE>(ox, oy, oz, dx, dy, dz, tris, ti, best);
    }
    if (node == kNone || (any && best.tri >= 0)) return true;
#ifdef HASTY_DEBUG_BOUNDS
    if (!HASTY_IN_BOUNDS(node < uint32_t(lim_nodes), BB_NODE)) return true;
#endif
    const float4* np = nodes + kWideNodeWords / 4 * int64_t(node);
    const Ld32 l0 = ld32<WIDE>(np), l1 = ld32<WIDE>(np + 2), l2 = ld32<WIDE>(np + 4);
    const float4 f0 = l0.a, f1 = l0.b, f2 = l1.a, f3 = l1.b, f4 = l2.a;
    const uint32_t node_imask = f2u(f0.w) >> 24;
    const float sx = l2.b.x, sy = l2.b.y, sz = l2.b.z;
    // Child plane t = q * A + B per axis (one FMA per plane), A = 2^e * inv
    // (exact), B = (p0 - o) * inv moved by eps to the conservative side.
    const PlaneTerms px = plane_terms(f0.x, ox, iv.ix, sx);
    const PlaneTerms py = plane_terms(f0.y, oy, iv.iy, sy);
    const PlaneTerms pz = plane_terms(f0.z, oz, iv.iz, sz);
    uint32_t child_base = f2u(f1.x), tri_base = f2u(f1.y);
    uint32_t meta_w[2] = {f2u(f1.z), f2u(f1.w)};
    // near and far planes per axis, chosen once by the ray's direction sign
    const uint32_t nx[2] = {neg_x ? f2u(f3.z) : f2u(f2.x), neg_x ? f2u(f3.w) : f2u(f2.y)};
    const uint32_t fx[2] = {neg_x ? f2u(f2.x) : f2u(f3.z), neg_x ? f2u(f2.y) : f2u(f3.w)};
    const uint32_t ny[2] = {neg_y ? f2u(f4.x) : f2u(f2.z), neg_y ? f2u(f4.y) : f2u(f2.w)};
    const uint32_t fy[2] = {neg_y ? f2u(f2.z) : f2u(f4.x), neg_y ? f2u(f2.w) : f2u(f4.y)};
    const uint32_t nz[2] = {neg_z ? f2u(f4.z) : f2u(f3.x), neg_z ? f2u(f4.w) : f2u(f3.y)};
    const uint32_t fz[2] = {neg_z ? f2u(f3.x) : f2u(f4.z), neg_z ? f2u(f3.y) : f2u(f4.w)};
    const float tlim = best.t * kPadHi;
    uint32_t hits = 0;          // children hit, by slot
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (uint32_t k = 0; k < 4; k += 2) {
        const float2 nx2 = fma2(byte_biased(nx[h], k), byte_biased(nx[h], k + 1), px.a, px.b_near);
        const float2 fx2 = fma2(byte_biased(fx[h], k), byte_biased(fx[h], k + 1), px.a, px.b_far);
        const float2 ny2 = fma2(byte_biased(ny[h], k), byte_biased(ny[h], k + 1), py.a, py.b_near);
        const float2 fy2 = fma2(byte_biased(fy[h], k), byte_biased(fy[h], k + 1), py.a, py.b_far);
        const float2 nz2 = fma2(byte_biased(nz[h], k), byte_biased(nz[h], k + 1), pz.a, pz.b_near);
        const float2 fz2 = fma2(byte_biased(fz[h], k), byte_biased(fz[h], k + 1), pz.a, pz.b_far);
        if (fmaxf(fmaxf(nx2.x, ny2.x), fmaxf(nz2.x, 0.0f)) <= fminf(fminf(fx2.x, fy2.x), fminf(fz2.x, tlim))) hits |= 1u << (4 * h + k);
        if (fmaxf(fmaxf(nx2.y, ny2.y), fmaxf(nz2.y, 0.0f)) <= fminf(fminf(fx2.y, fy2.y), fminf(fz2.y, tlim))) hits |= 2u << (4 * h + k);
      }
    }
    // inner children hit, slot k at bit k ^ octant: three conditional swaps
    uint32_t in = hits & node_imask;
    in = swap_bits(in, oct & 1u, 0x55u);
    in = swap_bits(in, oct & 2u, 0x33u);
    in = swap_bits(in, oct & 4u, 0x0Fu);
    uint2 ng = make_uint2(child_base, (in << 24) | node_imask);
    // triangles of the leaf children hit: unary count in a meta byte's top
    // three bits, first triangle in the others (an empty slot's byte is 0)
    uint32_t tb = 0;
    for (uint32_t leaf = hits & ~node_imask; leaf; leaf &= leaf - 1u) {
      const uint32_t m = byte_at(meta_w[0], meta_w[1], lowest_bit(leaf));
      tb |= (m >> 5) << (m & 31u);
    }
    tg = make_uint2(tri_base, tb);
    // the next node: the nearest inner child hit, else of the last group pushed
    if (!in) {
      if (sp == 0) { node = kNone; return tb == 0; }
      ng = stack[--sp];
    }
    const uint32_t bit = highest_bit(ng.y);
    const uint32_t slot = (bit - 24u) ^ oct;
    node = ng.x + popc(ng.y & 0xFFu & ~(0xFFFFFFFFu << slot));
    ng.y &= ~(1u << bit);
    if (ng.y > 0x00FFFFFFu) {
      if (sp < kWideStack) stack[sp++] = ng; else overflow = true;
    }
    return false;
  }
};

using TravWide = TravWideOf<true>;

// Array sizes for the bounds-checked build's traversal checks (no-op otherwise).
#ifdef HASTY_DEBUG_BOUNDS
#define HASTY_TRAV_LIMITS(tr, n_nodes, n_tris) ((tr).lim_nodes = (n_nodes), (tr).lim_tris = (n_tris))
#else
#define HASTY_TRAV_LIMITS(tr, n_nodes, n_tris) ((void)0)
#endif

HDI Hit trace_wide(const float4* nodes, const float4* tris, float ox, float oy, float oz, float dx, float dy, float dz) {
  TravWide tr;
  uint2 stack[kWideStack];
  tr.init(ox, oy, oz, dx, dy, dz);
  while (!tr.step(nodes, tris, stack)) {}
  return tr.best;
}

#ifdef __CUDACC__
// A warp's traversal of rays 0..n-1 of a queue. Whenever REFILL lanes are
// idle the warp takes that many rays, take(n_idle) giving the index of the
// first; fetch(k, traversal, nodes, tris, id) starts ray k. A finished ray's
// result stays in its lane until the warp refills, so that the results are
// written by several lanes at once (done(id, hit)) instead of by one or two
// in each step. Returns the number of this lane's rays whose traversal stack
// overflowed.
template <class Trav, int REFILL, class Take, class Fetch, class Done>
__device__ __forceinline__ uint32_t trace_rays_of_queue(uint32_t n, Take take, Fetch fetch, Done done) {
  Trav tr;
  typename Trav::Entry stack[Trav::kDepth];
  const float4* nodes = nullptr;
  const float4* tris = nullptr;
  int rid = -1;                         // ray of this lane, -1: none
  uint32_t overflows = 0;
  bool active = false;                  // its traversal goes on
  bool drained = false;                 // warp-uniform: the queue has been handed out
  const uint32_t lane = threadIdx.x & 31u;
  auto finish = [&] {
    done(rid, tr.best);
    overflows += tr.overflow ? 1u : 0u;
    rid = -1;
  };
  for (;;) {
    const unsigned idle = __ballot_sync(kFullMask, !active);
    if (!drained) {
      const uint32_t n_idle = uint32_t(__popc(idle));
      if (n_idle >= uint32_t(REFILL)) {
        const uint32_t base = take(n_idle);
        if (!active && rid >= 0) finish();
        if (base >= n || n - base <= n_idle) drained = true;
        if (!active) {
          const uint32_t k = base + uint32_t(__popc(idle & ((1u << lane) - 1u)));
          if (k < n) {
            fetch(k, tr, nodes, tris, rid);
            active = true;
          }
        }
        if (__ballot_sync(kFullMask, active) == 0) break;
      }
    } else if (idle == kFullMask) {
      break;
    }
    if (active && tr.step(nodes, tris, stack)) active = false;
  }
  if (rid >= 0) finish();
  return overflows;
}
#endif

template <int KIND>
HDI Hit trace_any(const float4* nodes, const float4* tris, float ox, float oy, float oz, float dx, float dy, float dz) {
  if (KIND == 1) return trace_wide(nodes, tris, ox, oy, oz, dx, dy, dz);
  return trace_binary(nodes, tris, ox, oy, oz, dx, dy, dz);
}

}  // namespace
}  // namespace hasty
