// wide_bvh.cuh — binary BVHs two levels at a time, with the binary traversal's answers.
//
// What bounds an incoherent walk here is the L1 data path: every lane reads another node, so a
// load costs one wavefront per lane whatever its width up to 32 bytes. A wide node holds the
// four grandchildren of an interior node (slots 0, 1 under its left child, 2, 3 under the
// right), where the binary tree takes six loads (three pairs of 64 bytes).
//
// A scene has one wide tree: the top-level BVH's wide nodes, and below its leaves the wide
// nodes of every mesh that is placed once and untransformed, so that a walk goes from the
// scene into its meshes without any per-object work. Other primitives are object leaves.
//
// Why the answers are the binary traversal's (trace_mesh.cuh, scene_device.cuh). There a leaf is
// visited when its own box is hit over [near, far] and its entry distance is below the nearest
// hit at its turn; the boxes above it add nothing, being exact unions under a monotone slab test.
//   - Any hit: a hit counts only if its leaf's exact box is hit. No order matters, so those
//     walks take boxes rounded outwards to a 256-step grid over the node's own box: 64 bytes,
//     two loads. The slab test on them is conservative (the margin m below).
//   - Nearest hit: the leaves' order is fixed by one comparison per interior node, of the entry
//     distances of its two children, whatever has been hit. A walk of the exact boxes, 128
//     bytes and four loads, takes the same leaves in the same order with the same tests, and so
//     ends with the same hit, also where rounding or a scaled object puts a hit before its
//     box's entry. (The grid's boxes for nearest hits too, in the order of their own entries, save
//     two loads: 717 us against 768 for 16,777,216 rays and 327,680 triangles, 705 against 805 for
//     1,500,000 rays and 10,000 spheres. But a leaf dropped unseen, entered beyond the nearest
//     hit, may be one that the binary order visits first and hits nearer: 1 in 1,000 of the rays
//     aimed at spheres 10^4 radii away, whose distances round that far.)
// Rays this arithmetic does not cover (a direction component of zero or outside
// [2^-40, 2^40], near < 0, coordinates beyond 2^40) or whose interval is empty or ends in a NaN use
// the binary nodes from the start.
#pragma once

#include <cfloat>

#include "trace_mesh.cuh"

namespace pbrt {

constexpr uint32_t kLeafRef = 0x80000000u;
constexpr int kWideStack = 128;  // three pending slots per two levels (upload_scene checks the depths)
constexpr float kWideLimit = 1.099511627776e12f;  // 2^40

// A wide node for nearest hits: the slots' own boxes.
struct __align__(128) ExactNode {
  float lo_x[4], hi_x[4];
  float lo_y[4], hi_y[4];
  float lo_z[4], hi_z[4];
  uint32_t ref[4];  // 0: empty; kLeafRef | leaf (triangle_ref, object slot); else a wide node
  uint32_t pad[4];
};
static_assert(sizeof(ExactNode) == 128, "an exact node is one cache line");

// The same for any hits: the boxes rounded outwards to a grid.
struct __align__(64) WideNode {
  float org[3];      // the node's own lower corner
  float step[3];     // the grid's step / 256 per axis
  uint32_t lo_x, hi_x, lo_y, hi_y, lo_z, hi_z;  // the slots' planes, a byte each
  uint32_t ref[4];   // as ExactNode's
};
static_assert(sizeof(WideNode) == 64, "a wide node is two 32-byte loads");

// A reference: 0, a wide node's index, or a leaf. A triangle leaf holds its first triangle and
// its count in 26 + 4 bits; a count that does not fit (code 15), and every count in scenes of
// more than 2^26 triangles (then the first triangle takes 30 bits), is read from the leaf's node.
// An object leaf holds its slot in the scene's primitive order.
constexpr uint32_t kObjectRef = 0x40000000u;

__host__ PBRT_DEV uint32_t triangle_ref(uint32_t first, uint32_t count, bool direct) {
  if (!direct) return kLeafRef | first;
  return kLeafRef | ((count <= 15u ? count - 1u : 15u) << 26) | first;
}

// A scene's wide tree and what its triangle leaves name, all meshes' arrays end to end.
struct WideView {
  const ExactNode* exact;
  const WideNode* wide;
  const float4* tri;    // 2 float4 per triangle
  const float2* tri_c;
  const uint2* leaf;    // at a leaf's first triangle: the leaf's node in `nodes`, the object's leaf index
  const float4* nodes;  // the meshes' binary nodes
  const uint32_t* slot_node;  // per primitive slot: the top-level node that is its leaf
  uint32_t root;        // 0: nothing bounded
  uint32_t count;       // wide nodes: no walk visits more
  bool direct;          // triangle references hold their counts
  bool bounded;         // every coordinate lies where the grid's arithmetic holds
};

PBRT_DEV void triangle_range(const WideView& w, uint32_t ref, uint32_t& first, uint32_t& count) {
  const uint32_t code = (ref >> 26) & 15u;
  first = w.direct ? ref & 0x3FFFFFFu : ref & 0x3FFFFFFFu;
  count = code + 1u;
  if (!w.direct || code == 15u) count = __float_as_uint(__ldg(&w.nodes[2 * size_t(__ldg(&w.leaf[first]).x) + 1]).w);
}

// The least float above x; +inf above FLT_MAX, -FLT_MAX above -inf; a NaN gives -inf (nothing
// is below it: an interval that ends in a NaN holds no hit).
PBRT_DEV float next_up(float x) {
  if (!(x == x)) return __int_as_float(0xff800000);
  if (x == 0.f) return __int_as_float(1);
  const uint32_t b = __float_as_uint(x);
  if (x > 0.f) return x > FLT_MAX ? x : __uint_as_float(b + 1u);
  return __uint_as_float(b - 1u);
}

struct WRay {
  F3 o, d, inv;
  bool exact;  // walks the binary nodes
};

PBRT_DEV WRay wide_ray(const F3& o, const F3& d, float near, float far, bool bounded) {
  WRay r;
  r.o = o;
  r.d = d;
  r.inv = mk3(frcp(d.x), frcp(d.y), frcp(d.z));
  // (sums of magnitudes: a NaN or an infinity anywhere fails them)
  const float so = fabsf(o.x) + fabsf(o.y) + fabsf(o.z), si = fabsf(r.inv.x) + fabsf(r.inv.y) + fabsf(r.inv.z);
  const float least = fminf(fminf(fabsf(r.inv.x), fabsf(r.inv.y)), fabsf(r.inv.z));
  r.exact = !(bounded && near >= 0.f && near <= far && so <= kWideLimit && si <= kWideLimit && least >= 1.f / kWideLimit);
  return r;
}

// Pending slots of a walk: reference and entry distance.
struct WideStack {
  uint2 s[kWideStack];
};

// (No check against kWideStack: a walk has at most three slots pending per two levels, and
// upload_scene lets no ray walk a scene whose trees are too deep for that.)
PBRT_DEV void wide_push(WideStack& st, int& sp, uint32_t ref, float e) {
  st.s[sp] = make_uint2(ref, __float_as_uint(e));
  ++sp;
}

// The next pending slot whose entry distance is below lim (the pop that drops entries at or
// beyond the nearest hit, bvh.rs:470-472); 0 when none is left.
PBRT_DEV uint32_t wide_pop(const WideStack& st, int& sp, float lim, float& e) {
  while (sp > 0) {
    const uint2 v = st.s[--sp];
    e = __uint_as_float(v.y);
    if (e < lim) return v.x;
  }
  return 0u;
}
PBRT_DEV uint32_t wide_pop(const WideStack& st, int& sp, float lim) {
  float e;
  return wide_pop(st, sp, lim, e);
}

namespace wide {
PBRT_DEV unsigned long long pack(float a, float b) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
PBRT_DEV void unpack(unsigned long long v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
PBRT_DEV unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}
PBRT_DEV float max3(float a, float b, float c) {
  float v;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(a), "f"(b), "f"(c));
  return v;
}
PBRT_DEV float min3(float a, float b, float c) {
  float v;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(a), "f"(b), "f"(c));
  return v;
}
// Byte j of w as the float 2^23 + 256 * byte.
template <int j>
PBRT_DEV float grid(uint32_t w) {
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7604u | (j << 4)));
}

PBRT_DEV unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
PBRT_DEV unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
PBRT_DEV void load256(const void* p, unsigned long long& a, unsigned long long& b, unsigned long long& c,
                      unsigned long long& d) {
  asm("ld.global.nc.v4.b64 {%0,%1,%2,%3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
}

// One axis of the four exact boxes: distances to the nearer and farther planes, each rounded as
// slab_axis_fast rounds it.
PBRT_DEV void exact_planes(const float* p, float o, float inv, float (&t0)[4], float (&t1)[4]) {
  unsigned long long l01, l23, h01, h23;
  load256(p, l01, l23, h01, h23);
  const unsigned long long no = pack(-o, -o), iv = pack(inv, inv);
  const bool neg = inv < 0.f;
  unpack(mul2(add2(neg ? h01 : l01, no), iv), t0[0], t0[1]);
  unpack(mul2(add2(neg ? h23 : l23, no), iv), t0[2], t0[3]);
  unpack(mul2(add2(neg ? l01 : h01, no), iv), t1[0], t1[1]);
  unpack(mul2(add2(neg ? l23 : h23, no), iv), t1[2], t1[3]);
}

// Entry distances of the four slots of an exact node (+inf: not hit within [near, inf), not below
// reach, or empty), and of the two children they lie under: on each axis a child's near plane is the
// nearer of its slots' two, so its distance is the smaller of their distances. The widening by
// 2*gamma(3) is monotone, so it is applied once to the largest entry and the smallest exit; where
// near >= 0 a negative distance needs no absolute value (it is clamped to near, or misses).
PBRT_DEV void exact_slots(const ExactNode* nd, const WRay& r, float near, float reach, float (&e)[4], float& el,
                          float& er, uint32_t (&ref)[4]) {
  float ax[4], bx[4], ay[4], by[4], az[4], bz[4];
  exact_planes(nd->lo_x, r.o.x, r.inv.x, ax, bx);
  exact_planes(nd->lo_y, r.o.y, r.inv.y, ay, by);
  exact_planes(nd->lo_z, r.o.z, r.inv.z, az, bz);
  const uint4 f = __ldg(reinterpret_cast<const uint4*>(nd->ref));
  ref[0] = f.x;
  ref[1] = f.y;
  ref[2] = f.z;
  ref[3] = f.w;
  float x[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    e[i] = max3(ax[i], ay[i], az[i]);
    x[i] = min3(bx[i], by[i], bz[i]);
  }
  el = max3(fminf(ax[0], ax[1]), fminf(ay[0], ay[1]), fminf(az[0], az[1]));
  er = max3(fminf(ax[2], ax[3]), fminf(ay[2], ay[3]), fminf(az[2], az[3]));
  const float W = PBRT_SLAB_WIDENING_F32;
  const unsigned long long up = pack(W, W), down = pack(-W, -W);
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    unsigned long long v = pack(e[i], e[i + 1]);
    unpack(add2(v, mul2(v, down)), e[i], e[i + 1]);
    v = pack(x[i], x[i + 1]);
    unpack(add2(v, mul2(v, up)), x[i], x[i + 1]);
  }
  const unsigned long long v = pack(el, er);
  unpack(add2(v, mul2(v, down)), el, er);
  el = fmaxf(el, near);
  er = fmaxf(er, near);
  const float inf = __int_as_float(0x7f800000);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    e[i] = fmaxf(e[i], near);
    e[i] = x[i] >= e[i] && e[i] < reach && (i % 2 == 0 || ref[i] != 0u) ? e[i] : inf;
  }
}

// Distances to the four slots' near (t0) and far (t1) planes on one axis, rounded outwards.
// The plane is at org + 256 * byte * step, its distance fma(2^23 + 256 * byte, k, c) with
// k = step * inv, p = (org - o) * inv and c = p -+ m - 2^23 * k. The roundings of k, p, c and the
// fma stay below 2^-21.9 |p| + 0.52 |k|, the exact test's own roundings and its widening by
// 2*gamma(3) below 2^-21 of the distance, which is at most |p| + 2^16 |k| (0.03 |k|), and a plane
// stands at most 0.26 |k| inside its box's (k_widen): m covers their sum.
PBRT_DEV void planes(float org, float step, uint32_t lo, uint32_t hi, float o, float inv, float (&t0)[4],
                     float (&t1)[4]) {
  const float p = fm(fs(org, o), inv), k = fm(step, inv);
  const float m = fa(fm(fabsf(p), 0x1p-20f), fabsf(k));
  float c0, c1;
  unpack(fma2(pack(-8388608.f, -8388608.f), pack(k, k), pack(fs(p, m), fa(p, m))), c0, c1);
  const bool neg = inv < 0.f;
  const uint32_t a = neg ? hi : lo, b = neg ? lo : hi;
  const unsigned long long kk = pack(k, k), cc0 = pack(c0, c0), cc1 = pack(c1, c1);
  unpack(fma2(pack(grid<0>(a), grid<1>(a)), kk, cc0), t0[0], t0[1]);
  unpack(fma2(pack(grid<2>(a), grid<3>(a)), kk, cc0), t0[2], t0[3]);
  unpack(fma2(pack(grid<0>(b), grid<1>(b)), kk, cc1), t1[0], t1[1]);
  unpack(fma2(pack(grid<2>(b), grid<3>(b)), kk, cc1), t1[2], t1[3]);
}

// Entry distances of the four slots of a node (+inf: not hit within [near, far] or empty).
PBRT_DEV void slots(const WideNode* nd, const WRay& r, float near, float far, float (&e)[4], uint32_t (&ref)[4]) {
  float4 a, b, c, d;
  load_node(reinterpret_cast<const float4*>(nd), a, b);
  load_node(reinterpret_cast<const float4*>(nd) + 2, c, d);
  float x0[4], x1[4], y0[4], y1[4], z0[4], z1[4];
  planes(a.x, a.w, __float_as_uint(b.z), __float_as_uint(b.w), r.o.x, r.inv.x, x0, x1);
  planes(a.y, b.x, __float_as_uint(c.x), __float_as_uint(c.y), r.o.y, r.inv.y, y0, y1);
  planes(a.z, b.y, __float_as_uint(c.z), __float_as_uint(c.w), r.o.z, r.inv.z, z0, z1);
  ref[0] = __float_as_uint(d.x);
  ref[1] = __float_as_uint(d.y);
  ref[2] = __float_as_uint(d.z);
  ref[3] = __float_as_uint(d.w);
  const float inf = __int_as_float(0x7f800000);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float t0 = fmaxf(max3(x0[i], y0[i], z0[i]), near);
    const float t1 = fminf(min3(x1[i], y1[i], z1[i]), far);
    e[i] = t0 <= t1 && (i % 2 == 0 || ref[i] != 0u) ? t0 : inf;
  }
}

PBRT_DEV void order(bool s, float& a, float& b, uint32_t& p, uint32_t& q) {  // exchanges when s
  const float t = s ? b : a;
  const uint32_t u = s ? q : p;
  b = s ? a : b;
  q = s ? p : q;
  a = t;
  p = u;
}
}  // namespace wide

// Visits one exact node: the slots entered below `reach`, in the binary traversal's order (of two
// siblings the right one first only when strictly nearer, bvh.rs:503-506). The first is returned,
// the others are pushed; the next pending one when none is entered; 0 when none is left.
PBRT_DEV uint32_t wide_step(const ExactNode* nd, const WRay& r, float near, float reach, WideStack& st, int& sp,
                            float& e) {
  float k[4], el, er;
  uint32_t f[4];
  wide::exact_slots(nd, r, near, reach, k, el, er, f);
  wide::order(k[1] < k[0], k[0], k[1], f[0], f[1]);
  wide::order(k[3] < k[2], k[2], k[3], f[2], f[3]);
  const float inf = __int_as_float(0x7f800000);
  // (the order of the pairs is the children's only when both have a slot to visit)
  const bool s = k[0] == inf || (er < el && k[2] < inf);
  wide::order(s, k[0], k[2], f[0], f[2]);
  wide::order(s, k[1], k[3], f[1], f[3]);
  if (k[3] < inf) wide_push(st, sp, f[3], k[3]);
  if (k[2] < inf) wide_push(st, sp, f[2], k[2]);
  if (k[1] < inf) wide_push(st, sp, f[1], k[1]);
  e = k[0];
  return k[0] < inf ? f[0] : wide_pop(st, sp, reach, e);
}
PBRT_DEV uint32_t wide_step(const ExactNode* nd, const WRay& r, float near, float reach, WideStack& st, int& sp) {
  float e;
  return wide_step(nd, r, near, reach, st, sp, e);
}

// The next pending slot of an any-hit walk, whose far end does not change; 0 when none is left.
PBRT_DEV uint32_t wide_pop_any(const WideStack& st, int& sp) { return sp > 0 ? st.s[--sp].x : 0u; }

// Visits one wide node of an any-hit walk, whose answer does not depend on the order: the slots
// entered within [near, far], in slot order.
PBRT_DEV uint32_t wide_step_any(const WideNode* nd, const WRay& r, float near, float far, WideStack& st, int& sp) {
  float k[4];
  uint32_t f[4];
  wide::slots(nd, r, near, far, k, f);
  const float inf = __int_as_float(0x7f800000);
#pragma unroll
  for (int i = 3; i > 0; --i)
    if (k[i] < inf) wide_push(st, sp, f[i], k[i]);
  return k[0] < inf ? f[0] : wide_pop_any(st, sp);
}

// The exact test of a leaf's box (its node) for a ray of the wide walk: box_hit where no
// direction component is zero.
PBRT_DEV bool leaf_hit(const float4* node, const WRay& r, float near, float& e) {
  float4 lo, hi;
  load_node(node, lo, hi);
  float x = __int_as_float(0x7f800000);
  e = near;
  slab_axis_fast(r.o.x, r.inv.x, r.inv.x < 0.f, lo.x, hi.x, e, x);
  slab_axis_fast(r.o.y, r.inv.y, r.inv.y < 0.f, lo.y, hi.y, e, x);
  slab_axis_fast(r.o.z, r.inv.z, r.inv.z < 0.f, lo.z, hi.z, e, x);
  return !(x < e);
}

// The first of a leaf's nearest triangles within [near, reach]; prim: its original index.
PBRT_DEV bool nearest_triangle(const float4* tri, const float2* tri_c, uint32_t first, uint32_t count, const F3& o,
                               const F3& d, float near, float reach, float& t_out, uint32_t& prim) {
  bool any = false;
  for (uint32_t k = first; k < first + count; ++k) {
    float4 A, B;
    load_node(&tri[2 * size_t(k)], A, B);
    const float2 C = __ldg(&tri_c[k]);
    float t;
    if (tri_hit(o, d, A, B, C.x, t) && t >= near && (any ? t < t_out : t <= reach)) {
      any = true;
      t_out = t;
      prim = __float_as_uint(C.y);
    }
  }
  return any;
}

// Whether some triangle of a leaf is hit within [near, far].
PBRT_DEV bool blocking_triangle(const float4* tri, const float2* tri_c, uint32_t first, uint32_t count, const F3& o,
                                const F3& d, float near, float far) {
  for (uint32_t k = first; k < first + count; ++k) {
    float4 A, B;
    load_node(&tri[2 * size_t(k)], A, B);
    const float2 C = __ldg(&tri_c[k]);
    float t;
    if (tri_hit(o, d, A, B, C.x, t) && t >= near && t <= far) return true;
  }
  return false;
}

// ---- one mesh's binary nodes, in the binary order --------------------------------------------
// References of this walk: a sibling pair by half its first index, or kLeafRef | a node.
PBRT_DEV uint32_t binary_ref(const float4& lo, const float4& hi, uint32_t node) {
  return __float_as_uint(hi.w) ? kLeafRef | node : __float_as_uint(lo.w) >> 1;
}

// Visits a sibling pair: the children hit with an entry below lim (any hit: up to it), the right one
// first only when strictly nearer (bvh.rs:503-506).
template <bool kAny>
PBRT_DEV uint32_t binary_step(const float4* nodes, uint32_t pair, const WRay& r, float near, float lim, WideStack& st,
                              int& sp) {
  const float4* n = nodes + 4 * size_t(pair);
  float4 l0, l1, r0, r1;
  load_node(n, l0, l1);
  load_node(n + 2, r0, r1);
  const PRay p = prepare_ray(r.o, r.d);
  const float inf = __int_as_float(0x7f800000);
  float dl, dr;
  const bool hl = box_hit(p, l0, l1, near, inf, dl);
  const bool hr = box_hit(p, r0, r1, near, inf, dr);
  const bool swap = hl && hr && dr < dl;
  const uint32_t fl = binary_ref(l0, l1, 2u * pair), fr = binary_ref(r0, r1, 2u * pair + 1u);
  const bool hn = swap ? hr : hl, hf = swap ? hl : hr;
  const float dn = swap ? dr : dl, df = swap ? dl : dr;
  const uint32_t fn = swap ? fr : fl, ff = swap ? fl : fr;
  const bool take_n = hn && (kAny ? !(lim < dn) : dn < lim), take_f = hf && (kAny ? !(lim < df) : df < lim);
  if (take_n) {
    if (take_f) wide_push(st, sp, ff, df);
    return fn;
  }
  return take_f ? ff : kAny ? wide_pop_any(st, sp) : wide_pop(st, sp, lim);
}

}  // namespace pbrt
