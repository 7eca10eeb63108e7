// traverse.cuh -- BVH traversal and primitive tests on the device.
//
// Reference: BVHAccel::intersect_p / ::intersect (src/accelerator/bvh.cpp:112-185),
// Bounds3::intersect_p (src/utility/geometry.hpp:837-864),
// Triangle::intersect(_p) (src/shape/triangle.cpp:117-174),
// sphere::intersect(_p) + TransformedShape::to_local (src/shape/sphere.cpp:15-47,
// src/shape/transformed_shape.hpp:17-21), GeometricPrimitive::intersect_p
// (src/shape/geometry.cpp:49-60).
//
// Order and culling match the reference exactly on child-pair nodes:
//  * the reference pops a node, tests its box against the CURRENT ray.t_max,
//    and pushes the children near-last (near = second child when
//    dir_is_neg[split_axis]);
//  * a box test is "slab overlap and tMax > 0" (independent of t_max) and
//    "tMin < t_max". Here both children of a visited node are tested at once;
//    the near child is entered immediately (no t_max change can happen in
//    between in the reference), the far child is pushed with its tMin and
//    the tMin < t_max part is re-evaluated when it is popped.
// Triangle arithmetic: the two cross products run in double and round to
// float, the dot products in float, exactly as the reference (no FMA: this
// file is compiled with --fmad=false).
#pragma once

#include "scene_types.h"

namespace trg {

struct RayIn {
  f3 o, d;
  float t_min, t_max;
};

struct Hit {
  int prim;       // -1: miss
  float t_attr;   // the accepted primitive's own parameter (triangle t, local sphere t)
  float alpha, beta;
};

__device__ __forceinline__ float4 ldg4(const float4* p) { return __ldg(p); }

// Two float4 in one 32-byte load (p 32-byte aligned). Not in the persistent
// render kernel: ptxas 13.0 does not compile that with it.
__device__ __forceinline__ void ldg8(const float4* p, float4& a, float4& b) {
#if defined(TRG_MATH_OUT_OF_LINE)
  a = ldg4(p);
  b = ldg4(p + 1);
#else
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
#endif
}

// The shared-memory treelet (DScene::treelet, staged by each block of a
// traversal kernel into its dynamic shared memory). Float4 k of treelet node j
// sits at 4 * j + (k ^ ((j >> 1) & 3)): eight lanes reading the same field of
// eight consecutive nodes then hit eight different bank groups (without the
// swizzle a 64-byte node stride leaves only two).
extern __shared__ float4 trav_smem[];

__device__ __forceinline__ int treelet_slot(int j, int k) { return 4 * j + (k ^ ((j >> 1) & 3)); }

// Copies the first n treelet nodes into shared memory; every thread of the
// block calls it once, before any traversal.
__device__ __forceinline__ void stage_treelet(const DScene& sc, int n) {
  const float4* src = reinterpret_cast<const float4*>(sc.treelet);
  for (int i = threadIdx.x; i < 4 * n; i += blockDim.x) trav_smem[treelet_slot(i >> 2, i & 3)] = __ldg(src + i);
  __syncthreads();
}

// Slab test with the reference's arithmetic. Returns the t_max-independent
// part ("pass"), and tmin for the "tMin < ray.t_max" part.
// Written without branches (the reference's early returns become flags;
// each conditional assignment is a select with the same NaN behaviour), so
// the lanes of a warp never diverge inside a box test. tmin is meaningful
// only when the test passes.
__device__ __forceinline__ bool box_pass(float lx, float ly, float lz, float hx, float hy, float hz, f3 o,
                                         f3 inv, bool n0, bool n1, bool n2, float& tmin) {
  float tMin = ((n0 ? hx : lx) - o.x) * inv.x;
  float tMax = slab_scale(((n0 ? lx : hx) - o.x) * inv.x);
  const float tyMin = ((n1 ? hy : ly) - o.y) * inv.y;
  const float tyMax = slab_scale(((n1 ? ly : hy) - o.y) * inv.y);
  const float tzMin = ((n2 ? hz : lz) - o.z) * inv.z;
  const float tzMax = slab_scale(((n2 ? lz : hz) - o.z) * inv.z);
  const bool miss_y = (tMin > tyMax) | (tyMin > tMax);
  tMin = tyMin > tMin ? tyMin : tMin;
  tMax = tyMax < tMax ? tyMax : tMax;
  const bool miss_z = (tMin > tzMax) | (tzMin > tMax);
  tMin = tzMin > tMin ? tzMin : tMin;
  tMax = tzMax < tMax ? tzMax : tMax;
  tmin = tMin;
  return !miss_y & !miss_z & (tMax > 0.0f);
}

// Three-operand minimum and maximum of numbers (sm_103 has them as one
// instruction each).
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// (a.x + b, a.y + b) and (a.x * b, a.y * b), each rounded once.
__device__ __forceinline__ float2 add2(float ax, float ay, float b) {
  float2 r;
  asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\tadd.rn.f32x2 p, p, q;\n\t"
      "mov.b64 {%0, %1}, p;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(ax), "f"(ay), "f"(b));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float b) {
  float2 r;
  asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\tmul.rn.f32x2 p, p, q;\n\t"
      "mov.b64 {%0, %1}, p;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b));
  return r;
}

// Both boxes of a child pair for an ordinary ray: origin and reciprocal
// direction finite, no reciprocal zero, and boxes with lo <= hi (no NaN can
// arise, and rounding keeps order). Then box_pass's chain of comparisons is
//   max(near x, y, z) <= slab_scale(min(far x, y, z)),  slab_scale(...) > 0,
// with near and far the smaller and larger of an axis's two quotients:
//  * a slab's quotients are ordered as its planes are (by the sign of the
//    reciprocal), so picking by sign is picking the smaller;
//  * slab_scale never decreases when its argument grows, so it commutes
//    with the minimum: one evaluation instead of three;
//  * box_pass compares each near value with the OTHER axes' far values;
//    comparing with its own axis as well changes nothing, since
//    near <= far before scaling and scaling moves far away from zero: it can
//    only fall below near when it is negative, where the last test fails.
// The walk is bound by instruction issue and by its dependent loads; this
// halves the comparisons and selects of a visit (the half-rate ALU pipe).
// Measured with tri_surely_missed below: 2M closest-hit and 2M shadow rays
// against 1M triangles 5.00 -> 4.67 ms, the 1024x768x16 occluded room 238 ->
// 229 ms, the 256x256x16 Cornell box 10.05 -> 8.97 ms.
__device__ __forceinline__ void pair_boxes(float4 x, float4 y, float4 z, f3 o, f3 inv, float& tl, float& tr, bool& hl,
                                           bool& hr) {
  const float2 x0 = mul2(add2(x.x, x.y, -o.x), inv.x), x1 = mul2(add2(x.z, x.w, -o.x), inv.x);
  const float2 y0 = mul2(add2(y.x, y.y, -o.y), inv.y), y1 = mul2(add2(y.z, y.w, -o.y), inv.y);
  const float2 z0 = mul2(add2(z.x, z.y, -o.z), inv.z), z1 = mul2(add2(z.z, z.w, -o.z), inv.z);
  tl = max3f(fminf(x0.x, x1.x), fminf(y0.x, y1.x), fminf(z0.x, z1.x));
  tr = max3f(fminf(x0.y, x1.y), fminf(y0.y, y1.y), fminf(z0.y, z1.y));
  const float fl = slab_scale(min3f(fmaxf(x0.x, x1.x), fmaxf(y0.x, y1.x), fmaxf(z0.x, z1.x)));
  const float fr = slab_scale(min3f(fmaxf(x0.y, x1.y), fmaxf(y0.y, y1.y), fmaxf(z0.y, z1.y)));
  hl = tl <= fl && fl > 0.0f;
  hr = tr <= fr && fr > 0.0f;
}

// Möller-Trumbore as the reference writes it. A = s0.xyz, AB = s1.xyz, AC = s2.xyz.
__device__ __forceinline__ bool tri_test(float4 s0, float4 s1, float4 s2, f3 o, f3 d, float t_min, float t_max,
                                         float& t, float& alpha, float& beta) {
  const f3 A = mk3(s0.x, s0.y, s0.z), AB = mk3(s1.x, s1.y, s1.z), AC = mk3(s2.x, s2.y, s2.z);
  const f3 S1 = cross(d, AC);
  const float div = dot(S1, AB);
  if (!div) return false;
  const float inv_div = 1.0f / div;
  const f3 AO = o - A;
  alpha = dot(AO, S1) * inv_div;
  if (alpha < 0.0f) return false;
  const f3 S2 = cross(AO, AB);
  beta = dot(d, S2) * inv_div;
  if (beta < 0.0f || alpha + beta > 1.0f) return false;
  t = dot(AC, S2) * inv_div;
  if (t < t_min || t > t_max) return false;
  return true;
}

// Whether tri_test certainly rejects a triangle, from the same quantities in
// plain fused arithmetic. tri_test rounds its cross products as the
// reference's doubles do (about 100 operations each); most triangles a walk
// reaches are missed by far more than any rounding, and those need not be
// evaluated that way.
//
// e = tri_margin() = 64 u M (u = 2^-24, M the largest |component| of AB and
// AC, +inf outside [2^-20, 2^20]); |d| components at most 1.001, the largest
// at least 0.5; t_min >= 0. With O the largest |AO| component, each of
//   div = d x AC . AB,  na = AO . d x AC,  nb = d . AO x AB,  nt = AC . AO x AB
// is a sum of at most six products of three factors, evaluated here and in
// tri_test with at most 51 u times the product of the factors' bounds
// between the two results (3 u a cross component here, 2 u there, and the
// roundings of the dot products). So within e M of div, e O of na and nb and
// e O M of nt lies what tri_test computes; the comparisons below take twice
// these margins, which also covers the roundings of 1 / div, of the products
// with it and of alpha + beta (at most 8 u relative). O is taken as at least
// 2^-60 and tested below 2^40: nothing underflows or overflows. A NaN or
// infinity rejects nothing.
__device__ __forceinline__ bool tri_surely_missed(f3 AB, f3 AC, float e, f3 AO, f3 d, float t_max) {
  const f3 s1 = mk3(__fmaf_rn(d.y, AC.z, -(d.z * AC.y)), __fmaf_rn(d.z, AC.x, -(d.x * AC.z)),
                    __fmaf_rn(d.x, AC.y, -(d.y * AC.x)));
  const f3 s2 = mk3(__fmaf_rn(AO.y, AB.z, -(AO.z * AB.y)), __fmaf_rn(AO.z, AB.x, -(AO.x * AB.z)),
                    __fmaf_rn(AO.x, AB.y, -(AO.y * AB.x)));
  const float div = __fmaf_rn(s1.z, AB.z, __fmaf_rn(s1.y, AB.y, s1.x * AB.x));
  const float sign = copysignf(1.0f, div);
  const float na = sign * __fmaf_rn(AO.z, s1.z, __fmaf_rn(AO.y, s1.y, AO.x * s1.x));
  const float nb = sign * __fmaf_rn(d.z, s2.z, __fmaf_rn(d.y, s2.y, d.x * s2.x));
  const float nt = sign * __fmaf_rn(AC.z, s2.z, __fmaf_rn(AC.y, s2.y, AC.x * s2.x));
  const float O = fmaxf(max3f(fabsf(AO.x), fabsf(AO.y), fabsf(AO.z)), 8.6736174e-19f);  // 2^-60
  const float M = e * 262144.0f;                                                        // 2^18
  const float a = fabsf(div), em = 2.0f * e * M, eo = 2.0f * e * O, et = eo * M;
  const bool sure = a > em && O < 1.0995116e12f;  // 2^40
  return sure && (na < -eo || nb < -eo || na + nb > a + (2.0f * eo + em) || nt < -et ||
                  nt > t_max * (a + em) + et);
}

// tri_surely_missed's per-triangle margin.
TR_HD float tri_margin(f3 AB, f3 AC) {
  float m = 0.0f;
  const float c[6] = {AB.x, AB.y, AB.z, AC.x, AC.y, AC.z};
  for (int k = 0; k < 6; ++k) m = fmaxf(m, fabsf(c[k]));
  return m >= 9.5367432e-07f && m <= 1048576.0f ? m * 3.8146973e-06f : INFINITY;  // 2^-20, 2^20, 2^-18
}

// Local ray of a TransformedShape: origin by the inverse point transform,
// direction by the inverse vector transform then the Ray constructor's
// double normalisation.
__device__ __forceinline__ void sphere_local(const DSphere& s, f3 o, f3 d, f3& lo, f3& ld) {
  lo = xform_point(s.inv, o);
  ld = normalize(xform_vec(s.inv, d));
}

// sphere::get_abc + the quadratic (src/shape/sphere.cpp:7-47). C widens to
// double in the reference; for float operands that equals the float
// difference (an inexact double difference needs an exponent gap > 29 bits,
// where both roundings give the larger operand).
__device__ __forceinline__ bool sphere_roots(f3 lo, f3 ld, float radius, float& t0, float& t1) {
  const float A = len2f(ld);
  const float B = 2.0f * dot(ld, lo);
  const float C = len2f(lo) - radius * radius;
  float delta = B * B - 4.0f * A * C;
  if (delta < 0.0f) return false;
  delta = sqrtf(delta);
  const float inv2A = 0.5f / A;
  t0 = (-B - delta) * inv2A;
  t1 = (-B + delta) * inv2A;
  return true;
}

// Boxes tested and leaf primitives tested by one traversal (the per-ray
// units of the traversal's algorithmic-bytes figure).
struct VisitCount {
  unsigned int boxes = 0, prims = 0;
  unsigned int cache_hits = 0;  // any-hit rays answered by a remembered occluder
};

// Tests one leaf slot. Returns true when `any` and the ray is occluded.
// quick: the ray meets tri_surely_missed's conditions.
__device__ __forceinline__ bool test_slot(const DScene& sc, int slot, f3 o, f3 d, float t_min, float& t_max, Hit& h,
                                          bool any, bool quick) {
  const float4 s0 = ldg4(sc.slots + 3 * slot);
  const float4 s1 = ldg4(sc.slots + 3 * slot + 1);
  const int kind = __float_as_int(s1.w);
  if (kind < 0) {
    const float4 s2 = ldg4(sc.slots + 3 * slot + 2);
    if (quick && tri_surely_missed(mk3(s1.x, s1.y, s1.z), mk3(s2.x, s2.y, s2.z), s2.w,
                                   o - mk3(s0.x, s0.y, s0.z), d, t_max))
      return false;
    float t, a, b;
    if (tri_test(s0, s1, s2, o, d, t_min, t_max, t, a, b)) {
      if (any) return true;
      t_max = t;
      h.prim = __float_as_int(s0.w);
      h.t_attr = t;
      h.alpha = a;
      h.beta = b;
    }
  } else {
    const DSphere& s = sc.spheres[kind];
    f3 lo, ld;
    sphere_local(s, o, d, lo, ld);
    float t0, t1;
    if (!sphere_roots(lo, ld, s.radius, t0, t1)) return false;
    if (any) return (t_min <= t0 && t0 <= t_max) || (t_min <= t1 && t1 <= t_max);
    if (t_max < t0 || t1 < t_min) return false;
    const bool not_t0 = t0 < t_min;
    if (not_t0 && t1 > t_max) return false;
    // Sphere::intersect_p never writes its hit_t argument, so
    // GeometricPrimitive stores 0 into ray.t_max (src/shape/sphere.cpp:98-119,
    // src/shape/geometry.cpp:49-57).
    t_max = 0.0f;
    h.prim = __float_as_int(s0.w);
    h.t_attr = not_t0 ? t1 : t0;
    h.alpha = 0.0f;
    h.beta = 0.0f;
  }
  return false;
}

// Any hit through a remembered occluder: slot s, tested after the box of its
// BVH leaf (stored in the leaf's parent node). The slab test passes a box
// whenever it passes a box inside it (rounding is monotone, a child's box
// lies in its parent's, and the NaN cases of a slab plane through the origin
// act like the parent's infinities), and the culling bound t_max is fixed for
// any hits; so a ray that passes the leaf's box passes every box above it,
// the reference's walk reaches the slot, and a hit there is the walk's answer
// (occluded). A miss here says nothing: the walk follows.
__device__ __forceinline__ bool occluded_by_slot(const DScene& sc, int scene, int s, f3 o, f3 d, float t_min,
                                                 float t_max) {
  const int lp = __ldg(sc.slot_leaf + s);
  float lx, ly, lz, hx, hy, hz;
  if (lp >= 0) {
    const float4* np = reinterpret_cast<const float4*>(sc.nodes + (lp >> 1));
    const float4 x = ldg4(np), y = ldg4(np + 1), z = ldg4(np + 2);
    const bool right = (lp & 1) != 0;
    lx = right ? x.y : x.x; hx = right ? x.w : x.z;
    ly = right ? y.y : y.x; hy = right ? y.w : y.z;
    lz = right ? z.y : z.x; hz = right ? z.w : z.z;
  } else {
    const SceneRoot& R = sc.roots[scene];
    lx = R.lo[0]; ly = R.lo[1]; lz = R.lo[2]; hx = R.hi[0]; hy = R.hi[1]; hz = R.hi[2];
  }
  const f3 inv = mk3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
  float tmin;
  if (!box_pass(lx, ly, lz, hx, hy, hz, o, inv, inv.x < 0.0f, inv.y < 0.0f, inv.z < 0.0f, tmin) || !(tmin < t_max))
    return false;
  Hit h;
  float tm = t_max;
  return test_slot(sc, s, o, d, t_min, tm, h, true, false);
}

// ---------------------------------------------------------------------------
// Persistent traversal with dynamic fetch. Each lane runs the same per-ray
// algorithm as BVHAccel's loops (same order, same culling, same tests), cut
// into steps so that a warp can keep its lanes busy: interior steps repeat
// until fewer than kWalkLanes lanes are without a leaf, then the lanes that
// have one test its primitives; when fewer than `refill` lanes still hold a
// ray, the finished lanes take new rays from the work queue (one atomic per
// warp). Every loop decision is warp-uniform; all 32 lanes stay in the loop
// until the queue is exhausted, so the kernel must be launched with whole
// warps and no lane may return early.

// The traversal stack, in (L1-cached) local memory: 8 bytes per entry, one
// 8-byte store per push. An entry holds the child reference shifted left by
// 5 with its primitive count in the low 5 bits (count 31 stands for "31 or
// more": the true count is then kept in a rarely touched second array) and
// the child's box entry t. Child references stay below 2^26 (checked on
// upload). A stack in shared memory was slower: shared memory takes its
// space from the L1 that serves the node and triangle reads.
constexpr int kStackBinary = 96;               // entries (a binary walk pushes at most one per level)
constexpr int kMaxDepth = kStackBinary - 4;      // the host rejects binary trees this many levels deep
constexpr int kStackWide = 96;                   // entries; the host keeps four-wide trees whose stack bound fits

// MIXED: each ray is a closest-hit or an any-hit ray by the member `any`
// (ANY is ignored).
template <bool ANY, bool COUNT, bool WIDE = false, bool MIXED = false>
struct TravLane {
  static_assert(ANY || !WIDE, "closest-hit traversal keeps the binary order");
  static_assert(!(MIXED && (COUNT || WIDE)), "mixed rays walk the binary tree, uncounted");
  static constexpr int kStack = WIDE ? kStackWide : kStackBinary;
  static constexpr unsigned kGeneral = 8u, kExactTri = 16u;
  f3 o, d, inv;
  unsigned neg;  // bit k: inv component k is negative; kGeneral: the ray takes box_pass; kExactTri: no quick rejection
  float t_min, t_max;
  int cur, cnt, sp;  // current node: cnt 0 interior, > 0 leaf, -1 none (stack ran dry, a leaf is postponed)
  int pl, pc;        // postponed leaf (pc > 0), speculative traversal
  float path_t;      // largest box entry t on the path taken since the last pop
  Hit h;
  bool occluded, failed;
  bool any;  // MIXED: this ray wants any hit
  __device__ __forceinline__ bool is_any() const { return MIXED ? any : ANY; }
  int2 st[kStack];      // (ref << 5 | min(count, 31), t bits)
  int big_cnt[kStack];  // counts of 31 or more, by stack index

  __device__ __forceinline__ void push(int ref, int c, float t) {
    if (c >= 31) big_cnt[sp] = c;
    st[sp++] = make_int2((ref << 5) | min(c, 31), __float_as_int(t));
  }

  // Starts a ray in scene `scene` of the set; returns false when it misses
  // the root box (done at once).
  // tl: the block staged scene 0's treelet (its root is treelet node 0).
  __device__ __forceinline__ bool start(const DScene& sc, int scene, f3 o_, f3 d_, float tmin_, float tmax_,
                                        VisitCount& vc, bool tl) {
    o = o_;
    d = d_;
    t_min = tmin_;
    t_max = tmax_;
    h.prim = -1;
    occluded = false;
    failed = false;
    sp = 0;
    pc = 0;
    path_t = -INFINITY;
    const SceneRoot& R = sc.roots[scene];
    if (R.kind == 0) return false;
    if (COUNT) ++vc.boxes;
    inv = mk3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    const bool n0 = inv.x < 0.0f, n1 = inv.y < 0.0f, n2 = inv.z < 0.0f;
    neg = (n0 ? 1u : 0u) | (n1 ? 2u : 0u) | (n2 ? 4u : 0u);
    const float big = max3f(fabsf(inv.x), fabsf(inv.y), fabsf(inv.z)), far = max3f(fabsf(o.x), fabsf(o.y), fabsf(o.z));
    const bool num = !isnan(inv.x) && !isnan(inv.y) && !isnan(inv.z) && !isnan(o.x) && !isnan(o.y) && !isnan(o.z);
    // pair_boxes' conditions (an infinite direction component has reciprocal 0)
    if (!(num && big <= kRealMax && far <= kRealMax && inv.x != 0.0f && inv.y != 0.0f && inv.z != 0.0f && sc.box_order))
      neg |= kGeneral;
    const float dm = max3f(fabsf(d.x), fabsf(d.y), fabsf(d.z));
    if (!(dm >= 0.5f && dm <= 1.001f && t_min >= 0.0f)) neg |= kExactTri;
    float tmin;
    if (!box_pass(R.lo[0], R.lo[1], R.lo[2], R.hi[0], R.hi[1], R.hi[2], o, inv, n0, n1, n2, tmin) || !(tmin < t_max))
      return false;
    cur = WIDE && R.kind == 1 ? R.offset4 : R.offset;
    if (!WIDE && tl && scene == 0 && R.kind == 1) cur = kTreeletRef;
    cnt = R.kind == 2 ? R.count : 0;
    return true;
  }

  // Next entry from the stack whose box entry is still before t_max;
  // returns false when the traversal is over.
  __device__ __forceinline__ bool pop() {
    while (sp > 0) {
      const int2 e = st[--sp];
      if (__int_as_float(e.y) < t_max) {
        cur = e.x >> 5;
        cnt = e.x & 31;
        if (cnt == 31) cnt = big_cnt[sp];
        path_t = __int_as_float(e.y);
        return true;
      }
    }
    return false;
  }

  // One child-pair visit at interior node `cur`; returns false when done.
  __device__ __forceinline__ bool interior(const DScene& sc, int* err, VisitCount& vc) {
    float4 a, b, c, dd;
    if (cur & kTreeletRef) {
      const int j = cur & (kTreeletRef - 1);
      a = trav_smem[treelet_slot(j, 0)];
      b = trav_smem[treelet_slot(j, 1)];
      c = trav_smem[treelet_slot(j, 2)];
      dd = trav_smem[treelet_slot(j, 3)];
    } else {
      const float4* np = reinterpret_cast<const float4*>(sc.nodes + cur);
      ldg8(np, a, b);
      ldg8(np + 2, c, dd);
    }
    if (COUNT) vc.boxes += 2;
    float tl, tr;
    bool hl, hr;
    if (neg & kGeneral) {
      const bool n0 = neg & 1u, n1 = neg & 2u, n2 = neg & 4u;
      hl = box_pass(a.x, b.x, c.x, a.z, b.z, c.z, o, inv, n0, n1, n2, tl);
      hr = box_pass(a.y, b.y, c.y, a.w, b.w, c.w, o, inv, n0, n1, n2, tr);
    } else {
      pair_boxes(a, b, c, o, inv, tl, tr, hl, hr);
    }
    hl = hl && tl < t_max;
    hr = hr && tr < t_max;
    bool second_near = (neg >> __float_as_int(dd.w)) & 1u;
    if (is_any() && !COUNT && sc.any_order != 0) {
      // any hit: the answer does not depend on the order, only the visits do
      // (the counting walk keeps the reference's visits)
      if (sc.any_order == 1) {
        second_near = !second_near;  // the far child first
      } else {  // the child with the larger box surface first
        const float lx = a.z - a.x, ly = b.z - b.x, lz = c.z - c.x;
        const float rx = a.w - a.y, ry = b.w - b.y, rz = c.w - c.y;
        second_near = rx * ry + ry * rz + rz * rx > lx * ly + ly * lz + lz * lx;
      }
    }
    const int lref = __float_as_int(dd.x), rref = __float_as_int(dd.y);
    const unsigned cc = (unsigned)__float_as_int(dd.z);
    const int lcnt = (int)(cc & 0xffffu), rcnt = (int)(cc >> 16);
    if (hl && hr) {
      if (sp >= kStack) {
        atomicOr(err, 1);
        h.prim = -1;
        occluded = false;
        failed = true;
        return false;
      }
      if (second_near) {
        push(lref, lcnt, tl);
        cur = rref;
        cnt = rcnt;
        path_t = fmaxf(path_t, tr);
      } else {
        push(rref, rcnt, tr);
        cur = lref;
        cnt = lcnt;
        path_t = fmaxf(path_t, tl);
      }
      return true;
    }
    if (hl) {
      cur = lref;
      cnt = lcnt;
      path_t = fmaxf(path_t, tl);
      return true;
    }
    if (hr) {
      cur = rref;
      cnt = rcnt;
      path_t = fmaxf(path_t, tr);
      return true;
    }
    return pop();
  }

  // Speculative traversal: the leaf just reached is postponed and the walk
  // goes on from the stack (with the t_max from before the leaf's tests).
  __device__ __forceinline__ void postpone() {
    pl = cur;
    pc = cnt;
    if (!pop()) cnt = -1;
  }

  // Tests the postponed leaf; returns false when the traversal is over.
  // Closest hit: the walk made since the postponement used a t_max that the
  // leaf may have lowered. Every box entry t on the current path (path_t is
  // their maximum, counted from the last pop) still below the new t_max means
  // the reference, testing the leaf first, takes the same path and pushes
  // the same entries; otherwise the reference would have culled a box on it:
  // the path is dropped and the next entry popped (entries pushed along it
  // are culled when popped, their boxes lying inside the dropped one).
  __device__ __forceinline__ bool postponed_leaf(const DScene& sc, VisitCount& vc) {
    for (int i = 0; i < pc; ++i) {
      if (COUNT) ++vc.prims;
      if (test_slot(sc, pl + i, o, d, t_min, t_max, h, is_any(), !(neg & kExactTri))) {
        occluded = true;
        h.prim = pl + i;  // any hit: the occluding slot
        return false;
      }
    }
    pc = 0;
    if (!is_any() && cnt >= 0 && !(path_t < t_max)) cnt = -1;
    if (cnt < 0) return pop();
    return true;
  }

  // One visit of four-wide node `cur` (any-hit only): the children whose
  // boxes pass are all taken, the nearest entered and the others pushed;
  // returns false when done.
  __device__ __forceinline__ bool interior4(const DScene& sc, int* err, VisitCount& vc) {
    const float4* np = reinterpret_cast<const float4*>(sc.nodes4 + cur);
    const float4 lx = ldg4(np), ly = ldg4(np + 1), lz = ldg4(np + 2);
    const float4 hx = ldg4(np + 3), hy = ldg4(np + 4), hz = ldg4(np + 5);
    const float4 rf = ldg4(np + 6), ct = ldg4(np + 7);
    const int refs[4] = {__float_as_int(rf.x), __float_as_int(rf.y), __float_as_int(rf.z), __float_as_int(rf.w)};
    const int cnts[4] = {__float_as_int(ct.x), __float_as_int(ct.y), __float_as_int(ct.z), __float_as_int(ct.w)};
    float t[4];
    bool hit[4];
    const bool n0 = neg & 1u, n1 = neg & 2u, n2 = neg & 4u;
    hit[0] = cnts[0] >= 0 && box_pass(lx.x, ly.x, lz.x, hx.x, hy.x, hz.x, o, inv, n0, n1, n2, t[0]) && t[0] < t_max;
    hit[1] = cnts[1] >= 0 && box_pass(lx.y, ly.y, lz.y, hx.y, hy.y, hz.y, o, inv, n0, n1, n2, t[1]) && t[1] < t_max;
    hit[2] = cnts[2] >= 0 && box_pass(lx.z, ly.z, lz.z, hx.z, hy.z, hz.z, o, inv, n0, n1, n2, t[2]) && t[2] < t_max;
    hit[3] = cnts[3] >= 0 && box_pass(lx.w, ly.w, lz.w, hx.w, hy.w, hz.w, o, inv, n0, n1, n2, t[3]) && t[3] < t_max;
    if (COUNT) vc.boxes += (cnts[0] >= 0) + (cnts[1] >= 0) + (cnts[2] >= 0) + (cnts[3] >= 0);
    int best = -1;
    float bt = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (hit[i] && (best < 0 || t[i] < bt)) {
        best = i;
        bt = t[i];
      }
    if (best < 0) return pop();
    const int npush = hit[0] + hit[1] + hit[2] + hit[3] - 1;
    if (sp + npush > kStack) {
      atomicOr(err, 1);
      h.prim = -1;
      occluded = false;
      failed = true;
      return false;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (hit[i] && i != best) push(refs[i], cnts[i], t[i]);
    cur = best == 0 ? refs[0] : best == 1 ? refs[1] : best == 2 ? refs[2] : refs[3];
    cnt = best == 0 ? cnts[0] : best == 1 ? cnts[1] : best == 2 ? cnts[2] : cnts[3];
    return true;
  }

  // The primitives of leaf `cur`; returns false when done.
  __device__ __forceinline__ bool leaf(const DScene& sc, VisitCount& vc) {
    for (int i = 0; i < cnt; ++i) {
      if (COUNT) ++vc.prims;
      if (test_slot(sc, cur + i, o, d, t_min, t_max, h, is_any(), !(neg & kExactTri))) {
        occluded = true;
        h.prim = cur + i;  // any hit: the occluding slot
        return false;
      }
    }
    return pop();
  }
};

// Job: unsigned count() const;
//      unsigned load(unsigned i, f3& o, f3& d, float& t_min, float& t_max, int& scene);
//        ray i of the queue; what it returns names the ray to cached and store
//      int cached(unsigned i) const;  any hits: a slot to test first (occluded_by_slot), or -1
//      void store(unsigned i, const Hit& h, float t_max, bool occluded).
// For an occluded any-hit ray h.prim is the occluding slot.
// tl_n: treelet nodes to stage in shared memory (the launch gives the block
// at least tl_n * 64 bytes of dynamic shared memory; 0: none). The four-wide
// walk does not use the treelet.
// Lanes still looking for a leaf below which the warp tests the leaves it has:
// waiting for the last few costs more than coming back for them. 1024x768x16
// room 165 -> 158 ms (its any hits 37.3 -> 32.9 ms), 2M closest + 2M any hits
// in 1M triangles 4.94 -> 4.79 ms, the sphere grid 48.9 -> 50.1 ms; with 8:
// 160, 4.80, 51.0. With the 32-byte node loads and the queue entry kept in the
// lane: 155, 4.55, 49.4 ms.
constexpr int kWalkLanes = 4;

template <bool ANY, bool COUNT, bool WIDE = false, class Job>
__device__ __forceinline__ void persistent_traverse(const DScene& sc, Job& job, unsigned int* fetch, int* err,
                                                    VisitCount& vc, int refill, int tl_n = 0) {
  const bool tl = !WIDE && tl_n > 0;
  if (tl) stage_treelet(sc, tl_n);
  const unsigned int n = job.count();
  const unsigned int lane = threadIdx.x & 31u;
  const unsigned int below = (1u << lane) - 1u;
  TravLane<ANY, COUNT, WIDE> L;
  unsigned int item = 0;
  bool live = false, exhausted = false;
  for (;;) {
    const unsigned int need = __ballot_sync(0xffffffffu, !live && !exhausted);
    if (need) {
      const int leader = __ffs(need) - 1;
      unsigned int base = 0;
      if ((int)lane == leader) base = atomicAdd(fetch, (unsigned int)__popc(need));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (!live && !exhausted) {
        item = base + (unsigned int)__popc(need & below);
        if (item < n) {
          f3 o, d;
          float tmin, tmax;
          int scene;
          item = job.load(item, o, d, tmin, tmax, scene);
          const int cs = ANY ? job.cached(item) : -1;
          if (ANY && cs >= 0 && occluded_by_slot(sc, scene, cs, o, d, tmin, tmax)) {
            ++vc.cache_hits;
            L.h.prim = cs;
            job.store(item, L.h, tmax, true);
            live = false;
          } else {
            live = L.start(sc, scene, o, d, tmin, tmax, vc, tl);
            if (!live) job.store(item, L.h, L.t_max, false);
          }
        } else {
          exhausted = true;
        }
      }
    }
    if (!__any_sync(0xffffffffu, live)) {
      if (__all_sync(0xffffffffu, exhausted)) break;
      continue;
    }
    if (COUNT) {
      // the reference's walk step for step (its box and primitive counts)
      for (;;) {
        while (__any_sync(0xffffffffu, live && L.cnt == 0)) {
          if (live && L.cnt == 0) {
            live = WIDE ? L.interior4(sc, err, vc) : L.interior(sc, err, vc);
            if (!live) job.store(item, L.h, L.t_max, L.occluded);
          }
        }
        if (live) {
          live = L.leaf(sc, vc);
          if (!live) job.store(item, L.h, L.t_max, L.occluded);
        }
        if (__popc(__ballot_sync(0xffffffffu, live)) < refill) break;
      }
    } else {
      // speculative while-while: interior steps go on while kWalkLanes lanes
      // have not found a leaf; a lane holding a postponed leaf keeps walking
      // (and waits at a second leaf); then the postponed leaves are tested
      for (;;) {
        for (;;) {
          if (live && L.cnt > 0 && L.pc == 0) L.postpone();
          const unsigned int walking = __ballot_sync(0xffffffffu, live && L.pc == 0);
          if (__popc(walking) < kWalkLanes && (walking == 0 || __any_sync(0xffffffffu, live && L.pc > 0))) break;
          if (live && L.cnt == 0) {
            const bool more = WIDE ? L.interior4(sc, err, vc) : L.interior(sc, err, vc);
            if (!more) {
              if (L.failed || L.pc == 0) {
                live = false;
                job.store(item, L.h, L.t_max, L.occluded);
              } else {
                L.cnt = -1;
              }
            }
          }
        }
        if (live && L.pc > 0) {
          live = L.postponed_leaf(sc, vc);
          if (!live) job.store(item, L.h, L.t_max, L.occluded);
        }
        if (__popc(__ballot_sync(0xffffffffu, live)) < refill) break;
      }
    }
  }
}

}  // namespace trg
