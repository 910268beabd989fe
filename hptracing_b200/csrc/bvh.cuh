// Closest-hit query through the 8-wide bounding volume hierarchy.
//
// The result is that of the tree walk in traverse.cuh, bit for bit: the
// minimum-t triangle over the tree leaves that pass the reference's box
// filter. A query runs in two parts:
//  1. The hierarchy's walk finds the nearest triangle of all that the
//     Moller-Trumbore test accepts in a leaf the ray crosses. Every triangle
//     is tested once (the tree lists it in every leaf it touches, ~50 times),
//     with the same FP32 arithmetic. A child's boxes hold every ray for which
//     that arithmetic can accept a triangle below it, by an error bound
//     derived in bvh_build.cpp, so the tree walk, which tests some of the same
//     triangles, finds this triangle or none as near.
//  2. bvh_certain shows that the tree walk tests this triangle in a leaf that
//     passes the reference's filter; then its answer is this one.
// A ray for which part 2 fails (mostly rays in a split plane) is walked
// through the tree instead.
//
// Part 2, from the triangle alone. The reference's builder puts a
// triangle into every leaf its bounds touch (src/hp/scene/kdtree.cpp:145-154),
// so around a hit point inside the bounds all leaves list it, except a leaf
// beyond a split just outside the bounds. Where no leaf that lists the
// triangle ends within 3 `round` of a bound (its flags say how far the first
// one is), or the hit point is not at that bound, every leaf within `round` of
// the hit point lists the triangle. [A leaf near the hit that does not list it
// was cut off by a split X beyond the bound m, m < X <= m + 3 round; the leaf
// on the split's near side that holds m lists the triangle and ends in (m, X].]
// The tree walk has to be in one of these leaves that the ray truly crosses
// (the filter rejects others). It finds its leaf by the rounded point o + t d,
// so within e = r (4 t |d| + |o + t d|) of a split, r = 2^-24, per axis, it may be on
// the wrong side, for as long as the ray takes to move away: a ray almost along
// the split stays there. Of the stretch within `round` of the hit, that is at
// most 2 e / |d| in t per axis; round is twice what the three need together.
// Besides, the leaf where the walk starts holds the origin, unrounded, and
// passes the filter by that: it is enough that it lists the triangle (a light
// that samples a point of its own plane).
// What this leaves open, and two triangles at exactly the same t, bvh_settle
// looks up in the tree.
#pragma once

#include "traverse.cuh"

namespace hpt {

HPT_HD float fma_rn(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return std::fmaf(a, b, c);
#endif
}
// a / b within 2 ulp.
HPT_HD float near_div(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fdividef(a, b);
#else
  return a / b;
#endif
}
HPT_HD uint32_t popc(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __popc(x);
#else
  return (uint32_t)__builtin_popcount(x);
#endif
}
HPT_HD int high_bit(uint32_t x) {
#ifdef __CUDA_ARCH__
  return 31 - __clz(x);
#else
  return 31 - __builtin_clz(x);
#endif
}
// Byte k of w as the float 32768 + byte (exact; one byte permute).
template <int k>
HPT_HD float plane(uint32_t w) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7604u | (k << 4)));
#else
  return as_float_u(0x47000000u | (((w >> (8 * k)) & 255u) << 8));
#endif
}
// Three-operand minimum and maximum (one instruction on sm_100).
HPT_HD float max3(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
#else
  return fmaxf(a, fmaxf(b, c));
#endif
}
HPT_HD float min3(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
#else
  return fminf(a, fminf(b, c));
#endif
}
// Two fused multiply-adds in one instruction.
struct Pair {
#ifdef __CUDA_ARCH__
  unsigned long long v;
#else
  float x, y;
#endif
};
HPT_HD Pair pair(float x, float y) {
#ifdef __CUDA_ARCH__
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(x), "f"(y));
  return p;
#else
  return Pair{x, y};
#endif
}
HPT_HD void unpair(const Pair& p, float& x, float& y) {
#ifdef __CUDA_ARCH__
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(p.v));
#else
  x = p.x;
  y = p.y;
#endif
}
HPT_HD Pair fma2(const Pair& a, const Pair& b, const Pair& c) {
#ifdef __CUDA_ARCH__
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
#else
  return Pair{fma_rn(a.x, b.x, c.x), fma_rn(a.y, b.y, c.y)};
#endif
}

// acc + the dot product of four signed bytes.
HPT_HD int dot4(uint32_t a, uint32_t b, int acc) {
#ifdef __CUDA_ARCH__
  int r;
  asm("dp4a.s32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(acc));
  return r;
#else
  for (int k = 0; k < 32; k += 8) acc += (int)(int8_t)(a >> k) * (int)(int8_t)(b >> k);
  return acc;
#endif
}
// mask << 1, with x's sign as the new bit.
HPT_HD uint32_t push_sign(uint32_t mask, int x) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l((uint32_t)x, mask, 1);
#else
  return (mask << 1) | ((uint32_t)x >> 31);
#endif
}
// Bytes 0xFF for the low four bits of m.
HPT_HD uint32_t byte_mask(uint32_t m) { return (((m & 15u) * 0x00204081u) & 0x01010101u) * 255u; }
// Bytes of b where mask is set, of a elsewhere.
HPT_HD uint32_t pick(uint32_t a, uint32_t b, uint32_t mask) { return a ^ ((a ^ b) & mask); }

// Walk state of one ray.
struct BvhRay {
  Ray ray;
  f3 inv;            // 1 / d
  uint32_t q, nq;    // d / |d| and its opposite in 127ths, bytes 0-2; byte 3 = -127
  float cull;        // boxes that start beyond it are skipped
  float best_t;      // nearest accepted t, +inf = none
  uint32_t best;     // its record in btris, kBvhNone = none; | kBvhTie when
                     // another triangle was accepted at exactly best_t,
                     // | kBvhMany when more than one was
  uint32_t node_base, node_bits;  // pending children: base; bits 0-7 = slots in
                                  // visiting order, 8-15 = imask, 16-18 =
                                  // octant (bit a: the ray runs toward +a)
  uint32_t tri_base, tri_bits;    // pending triangles
  uint32_t steps;    // bits 0-4 = stack entries, the rest counts node visits
                     // and triangle tests
};
constexpr uint32_t kBvhStep = 32u;
static_assert(kBvhStack == 32, "stack entries fit bits 0-4");
constexpr uint32_t kBvhNone = 0x3FFFFFFFu, kBvhTie = 0x40000000u, kBvhMany = 0x80000000u;

// d / |d| as bytes, for the test against a child's cone (BvhNode).
HPT_HD uint32_t direction_bytes(const f3& d, float scale127) {
  const uint32_t x = (uint32_t)(int)rintf(rn_mul(d.x, scale127)) & 255u;
  const uint32_t y = (uint32_t)(int)rintf(rn_mul(d.y, scale127)) & 255u;
  const uint32_t z = (uint32_t)(int)rintf(rn_mul(d.z, scale127)) & 255u;
  return x | (y << 8) | (z << 16) | (0x81u << 24);
}

// Starts a walk. Returns false when the ray is to be walked through the tree
// instead (non-finite rays; origins so far away that the roundings outgrow what
// the boxes and the certificate allow for; directions of a length, and scenes
// of a size, at which products of the test overflow or underflow).
HPT_HD bool bvh_init(const Ray& r, float scene_eps, BvhRay& b) {
  b.ray = r;
  b.best = kBvhNone;
  b.best_t = b.cull = as_float(0x7f800000);
  b.steps = 0;
  b.tri_bits = 0;
  b.tri_base = 0;
  const float dmax = fmaxf(fabsf(r.d.x), fmaxf(fabsf(r.d.y), fabsf(r.d.z)));
  // Reciprocals. A component below 1e-9 of the largest moves the ray by less
  // than rounding over the scene: its slab test is the origin's side of the
  // two planes, which a very large reciprocal gives (no 0 x inf).
  const float tiny = rn_mul(dmax, 1e-9f);
  const float big = rn_mul(rn_rcp(dmax), 1e9f);
  b.inv.x = fabsf(r.d.x) > tiny ? rn_rcp(r.d.x) : copysignf(big, r.d.x);
  b.inv.y = fabsf(r.d.y) > tiny ? rn_rcp(r.d.y) : copysignf(big, r.d.y);
  b.inv.z = fabsf(r.d.z) > tiny ? rn_rcp(r.d.z) : copysignf(big, r.d.z);
  // The root as the only pending child (slot 0).
  const uint32_t oct =
      (b.inv.x > 0.f ? 1u : 0u) | (b.inv.y > 0.f ? 2u : 0u) | (b.inv.z > 0.f ? 4u : 0u);
  b.node_base = 0;
  b.node_bits = (oct << 16) | (1u << 8) | (1u << oct);
  const float omax = fmaxf(fabsf(r.o.x), fmaxf(fabsf(r.o.y), fabsf(r.o.z)));
  if (!(finite3(r.o) && finite3(r.d) && dmax > 1e-9f && dmax < 1e9f && scene_eps < 2e4f &&
        omax <= rn_mul(kMaxOrigin, scene_eps)))
    return false;
  const float len127 = rn_div(127.f, length(r.d));
  b.q = direction_bytes(r.d, len127);
  b.nq = direction_bytes(r.d, -len127);
  return true;
}

// Bit k, when the ray enters the box of slot k before cull: the planes of
// four slots are the bytes of near / far words. N / F: the node's offsets of
// near and far planes.
template <int k>
HPT_HD uint32_t bvh_slot(uint32_t nx, uint32_t ny, uint32_t nz, uint32_t fx, uint32_t fy,
                         uint32_t fz, const Pair& Sxy, const Pair& Nxy, const Pair& Fxy,
                         const Pair& Szz, const Pair& NFz, float cull) {
  float x0, y0, z0, x1, y1, z1;
  unpair(fma2(pair(plane<k & 3>(nx), plane<k & 3>(ny)), Sxy, Nxy), x0, y0);
  unpair(fma2(pair(plane<k & 3>(fx), plane<k & 3>(fy)), Sxy, Fxy), x1, y1);
  unpair(fma2(pair(plane<k & 3>(nz), plane<k & 3>(fz)), Szz, NFz), z0, z1);
  const float t0 = fmaxf(max3(x0, y0, z0), 0.f), t1 = fminf(min3(x1, y1, z1), cull);
  return t0 <= t1 ? 1u << k : 0u;
}

// Visits a node: sets the pending children and triangles.
HPT_HD void bvh_node(BvhRay& b, const uint4* node) {
  const uint4 n0 = ldg(node), n1 = ldg(node + 1);
  uint4 n2 = ldg(node + 2), n3 = ldg(node + 3), n4 = ldg(node + 4);
  {
    // The slots whose wide box counts.
    const uint4 c0 = ldg(node + 8), c1 = ldg(node + 9);
    uint32_t r = 0;
    r = push_sign(r, dot4(c1.w, b.q, -1) & dot4(c1.w, b.nq, -1));
    r = push_sign(r, dot4(c1.z, b.q, -1) & dot4(c1.z, b.nq, -1));
    r = push_sign(r, dot4(c1.y, b.q, -1) & dot4(c1.y, b.nq, -1));
    r = push_sign(r, dot4(c1.x, b.q, -1) & dot4(c1.x, b.nq, -1));
    r = push_sign(r, dot4(c0.w, b.q, -1) & dot4(c0.w, b.nq, -1));
    r = push_sign(r, dot4(c0.z, b.q, -1) & dot4(c0.z, b.nq, -1));
    r = push_sign(r, dot4(c0.y, b.q, -1) & dot4(c0.y, b.nq, -1));
    r = push_sign(r, dot4(c0.x, b.q, -1) & dot4(c0.x, b.nq, -1));
    const uint4 w2 = ldg(node + 5), w3 = ldg(node + 6), w4 = ldg(node + 7);
    const uint32_t m0 = byte_mask(r), m1 = byte_mask(r >> 4);
    n2.x = pick(n2.x, w2.x, m0);
    n2.y = pick(n2.y, w2.y, m1);
    n2.z = pick(n2.z, w2.z, m0);
    n2.w = pick(n2.w, w2.w, m1);
    n3.x = pick(n3.x, w3.x, m0);
    n3.y = pick(n3.y, w3.y, m1);
    n3.z = pick(n3.z, w3.z, m0);
    n3.w = pick(n3.w, w3.w, m1);
    n4.x = pick(n4.x, w4.x, m0);
    n4.y = pick(n4.y, w4.y, m1);
    n4.z = pick(n4.z, w4.z, m0);
    n4.w = pick(n4.w, w4.w, m1);
  }
  const uint32_t e = n0.w;
  const float sx = as_float_u((e & 255u) << 23), sy = as_float_u(((e >> 8) & 255u) << 23),
              sz = as_float_u(((e >> 16) & 255u) << 23);
  const float rx = rn_sub(as_float_u(n0.x), b.ray.o.x), ry = rn_sub(as_float_u(n0.y), b.ray.o.y),
              rz = rn_sub(as_float_u(n0.z), b.ray.o.z);
  // The planes move outward by kBoxGrowth of the distance to the node's far
  // side.
  const float far_side =
      fma_rn(256.f, max3(sx, sy, sz), max3(fabsf(rx), fabsf(ry), fabsf(rz)));
  const float grow = rn_mul(kBoxGrowth, far_side);
  f3 S;
  S.x = rn_mul(sx, b.inv.x);
  S.y = rn_mul(sy, b.inv.y);
  S.z = rn_mul(sz, b.inv.z);
  const float ox = fma_rn(-32768.f, S.x, rn_mul(rx, b.inv.x));
  const float oy = fma_rn(-32768.f, S.y, rn_mul(ry, b.inv.y));
  const float oz = fma_rn(-32768.f, S.z, rn_mul(rz, b.inv.z));
  const Pair Oxy = pair(ox, oy), Axy = pair(fabsf(b.inv.x), fabsf(b.inv.y));
  const Pair Sxy = pair(S.x, S.y), Szz = pair(S.z, S.z);
  const Pair Nxy = fma2(pair(-grow, -grow), Axy, Oxy), Fxy = fma2(pair(grow, grow), Axy, Oxy);
  const Pair NFz = fma2(pair(-grow, grow), pair(fabsf(b.inv.z), fabsf(b.inv.z)), pair(oz, oz));
  const uint32_t oct = b.node_bits >> 16;
  const bool px = oct & 1u, py = oct & 2u, pz = oct & 4u;
  uint32_t h = 0;
  // Words: n2 = lo x (2), lo y (2); n3 = lo z, hi x; n4 = hi y, hi z.
  {
    const uint32_t nx = px ? n2.x : n3.z, fx = px ? n3.z : n2.x;
    const uint32_t ny = py ? n2.z : n4.x, fy = py ? n4.x : n2.z;
    const uint32_t nz = pz ? n3.x : n4.z, fz = pz ? n4.z : n3.x;
    h |= bvh_slot<0>(nx, ny, nz, fx, fy, fz, Sxy, Nxy, Fxy, Szz, NFz, b.cull);
    h |= bvh_slot<1>(nx, ny, nz, fx, fy, fz, Sxy, Nxy, Fxy, Szz, NFz, b.cull);
    h |= bvh_slot<2>(nx, ny, nz, fx, fy, fz, Sxy, Nxy, Fxy, Szz, NFz, b.cull);
    h |= bvh_slot<3>(nx, ny, nz, fx, fy, fz, Sxy, Nxy, Fxy, Szz, NFz, b.cull);
  }
  {
    const uint32_t nx = px ? n2.y : n3.w, fx = px ? n3.w : n2.y;
    const uint32_t ny = py ? n2.w : n4.y, fy = py ? n4.y : n2.w;
    const uint32_t nz = pz ? n3.y : n4.w, fz = pz ? n4.w : n3.y;
    h |= bvh_slot<4>(nx, ny, nz, fx, fy, fz, Sxy, Nxy, Fxy, Szz, NFz, b.cull);
    h |= bvh_slot<5>(nx, ny, nz, fx, fy, fz, Sxy, Nxy, Fxy, Szz, NFz, b.cull);
    h |= bvh_slot<6>(nx, ny, nz, fx, fy, fz, Sxy, Nxy, Fxy, Szz, NFz, b.cull);
    h |= bvh_slot<7>(nx, ny, nz, fx, fy, fz, Sxy, Nxy, Fxy, Szz, NFz, b.cull);
  }
  const uint32_t imask = e >> 24;
  uint32_t inner = h & imask;
  // Hits by visiting order: slot s goes to bit s ^ oct, the highest first.
  if (px) inner = ((inner & 0x55u) << 1) | ((inner >> 1) & 0x55u);
  if (py) inner = ((inner & 0x33u) << 2) | ((inner >> 2) & 0x33u);
  if (pz) inner = ((inner & 0x0Fu) << 4) | (inner >> 4);
  b.node_base = n1.x;
  b.node_bits = (oct << 16) | (imask << 8) | inner;
  b.tri_base = n1.y;
  uint32_t tri = 0;
  for (uint32_t l = h & ~imask; l; l &= l - 1) {
    const int k = high_bit(l & (0u - l));
    const uint32_t m = ((k < 4 ? n1.z : n1.w) >> (8 * (k & 3))) & 255u;
    tri |= (m >> 5) << (m & 31u);
  }
  b.tri_bits = tri;
}

// Takes the next pending child (from the stack when this node's are done)
// and visits it. Returns false when nothing is pending.
HPT_HD bool bvh_visit(const BvhNode* bvh, uint32_t num_bvh, BvhRay& b, uint2* stack,
                      DevErr* err) {
  if (!(b.node_bits & 255u)) {
    if ((b.steps & 31u) == 0) return false;
    --b.steps;
    const uint2 e = stack[b.steps & 31u];
    b.node_base = e.x;
    b.node_bits = e.y;
  }
  const int bit = high_bit(b.node_bits & 255u);
  const uint32_t slot = (uint32_t)bit ^ (b.node_bits >> 16);
  const uint32_t node = b.node_base + popc((b.node_bits >> 8) & ((1u << slot) - 1u));
  b.node_bits &= ~(1u << bit);
  if (b.node_bits & 255u) {
    HPT_DCHECK(err, (b.steps & 31u) < kBvhStack - 1, 113, b.steps, return false);
    stack[b.steps & 31u].x = b.node_base;
    stack[b.steps & 31u].y = b.node_bits;
    ++b.steps;
  }
  HPT_DCHECK(err, node < num_bvh, 114, node, return false);
  bvh_node(b, reinterpret_cast<const uint4*>(bvh + node));
  b.steps += kBvhStep;
  return true;
}

// One triangle test of the pending ones. A winning hit shrinks the cull
// distance to the tree walk's own stopping rule (1.0001 times the best t plus
// slack), or a little beyond it: what the computed t can be off by.
// tie receives the other triangle's record where best gets kBvhTie.
HPT_HD void bvh_test(const BvhTri* btris, float scene_eps, BvhRay& b, uint32_t& tie) {
  const int k = high_bit(b.tri_bits);
  b.tri_bits &= ~(1u << k);
  const int32_t i = (int32_t)b.tri_base + k;
  const float4* rec = reinterpret_cast<const float4*>(btris + i);
  b.steps += kBvhStep;
  float t, u, v;
  if (mt_test(b.ray, ldg(rec), ldg(rec + 1), ldg(rec + 2), t, u, v)) {
    if (t < b.best_t) {
      b.best_t = t;
      b.best = (uint32_t)i;
      const float per_unit =
          fminf(fabsf(b.inv.x), fminf(fabsf(b.inv.y), fabsf(b.inv.z)));  // 1 / largest |d|
      b.cull = fma_rn(t, kCullFactor, rn_mul(scene_eps, per_unit));
    } else if (t == b.best_t) {
      b.best |= b.best & kBvhTie ? kBvhMany : kBvhTie;
      tie = (uint32_t)i;
    }
  }
}

// A ray that meets nothing misses - unless it runs exactly along a triangle's
// edge e2: then the Moller-Trumbore test divides by zero, its comparisons
// pass 0 / 0, and the reference "hits" the triangle at t = +inf when there is
// no other hit. d x e2 comes out as exactly zero only if d has e2's direction
// within two roundings per component. True when the scene has no such edge.
// (A det of exactly zero with d x e2 not zero leaves the tested products +-inf
// or NaN and is rejected, but for rounded sums that cancel by chance for a ray
// in the triangle's plane.)
template <class Sc>
HPT_HD bool bvh_no_parallel_edge(const Sc& s, const f3& d) {
  const float x = fabsf(d.x), y = fabsf(d.y), z = fabsf(d.z);
  const int a = x >= y && x >= z ? 0 : (y >= z ? 1 : 2);
  const uint32_t n = (uint32_t)(a == 0 ? s.num_edge_keys[0] : (a == 1 ? s.num_edge_keys[1] : s.num_edge_keys[2]));
  if (n == 0) return true;
  const float* keys = a == 0 ? s.edge_keys[0] : (a == 1 ? s.edge_keys[1] : s.edge_keys[2]);
  const float da = a == 0 ? d.x : (a == 1 ? d.y : d.z);
  const float r1 = near_div(a == 0 ? d.y : (a == 1 ? d.z : d.x), da);
  const float r2 = near_div(a == 0 ? d.z : (a == 1 ? d.x : d.y), da);
  const uint32_t c1 = edge_cell(r1), c2 = edge_cell(r2), tag = edge_tag(c1, c2);
  // Entries of a bucket are filled from the first; the table is not full.
  const uint32_t buckets = n >> 2;
  for (uint32_t b = edge_bucket(c1, c2, buckets), left = buckets; left != 0; --left) {
    const uint4 k = ldg(reinterpret_cast<const uint4*>(keys) + b);
    if (k.x == tag || k.y == tag || k.z == tag || k.w == tag) return false;
    if (k.w == 0) break;
    b = b + 1 < buckets ? b + 1 : 0;
  }
  return true;
}

// At least this far from a triangle's bound (face 2a: lower on axis a, 2a + 1:
// upper) ends the first leaf that lists it and ends beyond (BvhTri::flags).
HPT_HD float leaf_gap(uint32_t flags, int face, float scene_eps) {
  const uint32_t c = (flags >> (8 + 4 * face)) & 15u;
  return c == 0 ? 0.f : rn_mul(rn_mul(kGapUnit, scene_eps), as_float_u((126u + c) << 23));
}

// True when the tree walk's answer for ray r is (best, best_t), the result
// of its hierarchy walk (see the file comment); kBvhNone alone: a miss.
template <class Sc>
HPT_HD bool bvh_certain(const Sc& s, const Ray& r, uint32_t best, float best_t, DevErr* err) {
  if (best & (kBvhTie | kBvhMany)) return false;
  const bool axes = r.d.x != 0.f && r.d.y != 0.f && r.d.z != 0.f;
  if (best == kBvhNone) return bvh_no_parallel_edge(s, r.d);
  HPT_DCHECK(err, best < (uint32_t)s.num_btris, 115, best, return false);
  const float4* rec = reinterpret_cast<const float4*>(s.btris + best);
  const float4 A = ldg(rec), E1 = ldg(rec + 1), E2 = ldg(rec + 2);
  const uint32_t flags = (uint32_t)as_int(E2.w);
  if (flags & kTriIrregular) return false;
  const float o[3] = {r.o.x, r.o.y, r.o.z}, d[3] = {r.d.x, r.d.y, r.d.z};
  const float p[3] = {rn_add(r.o.x, rn_mul(best_t, r.d.x)), rn_add(r.o.y, rn_mul(best_t, r.d.y)),
                      rn_add(r.o.z, rn_mul(best_t, r.d.z))};
  const float a[3] = {A.x, A.y, A.z}, e1[3] = {E1.x, E1.y, E1.z}, e2[3] = {E2.x, E2.y, E2.z};
  const float along = fma_rn(1.5e-6f, best_t,
                             rn_mul(1.2e-7f, rn_add(fabsf(near_div(p[0], d[0])),
                                                    rn_add(fabsf(near_div(p[1], d[1])),
                                                           fabsf(near_div(p[2], d[2]))))));
  float lo[3], hi[3], below[3], above[3], exact[3];
  bool ok = axes;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float v1 = rn_add(a[k], e1[k]), v2 = rn_add(a[k], e2[k]);
    lo[k] = min3(a[k], v1, v2);
    hi[k] = max3(a[k], v1, v2);
    exact[k] = rn_mul(2.4e-7f, fmaxf(fabsf(lo[k]), fabsf(hi[k])));
    below[k] = leaf_gap(flags, 2 * k, s.scene_eps);
    above[k] = leaf_gap(flags, 2 * k + 1, s.scene_eps);
    const float round = fma_rn(along, fabsf(d[k]), exact[k]);
    ok = ok && p[k] > rn_add(lo[k], 3.f * round <= below[k] ? -2.f * round : round) &&
         p[k] < rn_sub(hi[k], 3.f * round <= above[k] ? -2.f * round : round);
  }
  if (ok) return true;
  ok = true;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    ok = ok && o[k] >= s.root_lo[k] && o[k] <= s.root_hi[k] &&
         o[k] > rn_add(rn_sub(lo[k], below[k]), exact[k]) &&
         o[k] < rn_sub(rn_add(hi[k], above[k]), exact[k]);
  return ok;
}

// Looks up in the tree a hit that bvh_certain leaves open: goes through the
// leaves that list the triangle - of two at the same t, both - along the ray.
// kLookupHit: the tree walk tests it in a leaf that counts, and `winner` is
// the record it would report: of two triangles at one t the reference keeps
// the one it meets first, the lowest position in the leaf lists over the
// leaves that count for either. kLookupNone: no leaf that lists it counts.
// kLookupOpen: a leaf may count or not (the ray crosses it by no more than
// rounding, or it lies at the walk's end), or the tree is irregular there.
enum Lookup : int { kLookupOpen = 0, kLookupHit = 1, kLookupNone = 2 };
// Not inlined (two call sites: its code is mostly run cold).
template <class Sc>
__host__ __device__ __noinline__ Lookup bvh_lookup(const Sc& s, const Ray& r, uint32_t best, uint32_t tie, float best_t,
                         uint32_t& winner, DevErr* err) {
  const bool two = best & kBvhTie;
  const uint32_t first = best & kBvhNone;
  if ((best & kBvhMany) || first == kBvhNone || !(best_t < as_float(0x7f800000)))
    return kLookupOpen;
  const float o[3] = {r.o.x, r.o.y, r.o.z};
  // 1 / d; zero stands for a zero component.
  const float inv[3] = {r.d.x != 0.f ? rn_rcp(r.d.x) : 0.f, r.d.y != 0.f ? rn_rcp(r.d.y) : 0.f,
                        r.d.z != 0.f ? rn_rcp(r.d.z) : 0.f};
  const float dmax = fmaxf(fabsf(r.d.x), fmaxf(fabsf(r.d.y), fabsf(r.d.z)));
  const float slack = rn_div(s.scene_eps, dmax);
  // A face's distance is off by a few 1e-7 of the scene's size and of itself.
  const float tol = fma_rn(best_t, 1e-6f, rn_mul(0.1f, slack));
  // The walk visits the leaves that begin before this.
  const float stop = fma_rn(best_t, 1.0001f, slack);
  // A ray that stays within rounding of its place on some axis all the way up
  // to the hit: no leaf holds it by more.
  if (!two)
    for (int a = 0; a < 3; ++a)
      if (rn_mul(2.4e-7f, rn_mul(fabsf(o[a]), fabsf(inv[a]))) > best_t) return kLookupOpen;
  // The bounds of the triangle, or of both, and the tree node that holds all
  // their leaves.
  float lo[3], hi[3];
  int32_t id[2] = {-1, -1};
  int node = 0;
  for (int k = 0; k < (two ? 2 : 1); ++k) {
    const uint32_t cand = k ? tie : first;
    HPT_DCHECK(err, cand < (uint32_t)s.num_btris, 116, cand, return kLookupOpen);
    const float4* rec = reinterpret_cast<const float4*>(s.btris + cand);
    const float4 A = ldg(rec), E1 = ldg(rec + 1), E2 = ldg(rec + 2);
    if ((uint32_t)as_int(E2.w) & kTriIrregular) return kLookupOpen;
    id[k] = as_int(A.w);
    if (!two) node = as_int(E1.w);
    const float grow = rn_mul(0.1f, s.scene_eps);
    const float v0[3] = {A.x, A.y, A.z}, e1[3] = {E1.x, E1.y, E1.z}, e2[3] = {E2.x, E2.y, E2.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float v1 = rn_add(v0[a], e1[a]), v2 = rn_add(v0[a], e2[a]);
      const float l = rn_sub(fminf(v0[a], fminf(v1, v2)), grow);
      const float h = rn_add(fmaxf(v0[a], fmaxf(v1, v2)), grow);
      lo[a] = k ? fminf(lo[a], l) : l;
      hi[a] = k ? fmaxf(hi[a], h) : h;
    }
  }
  // Depth-first over the nodes that the bounds and the ray touch: of two
  // triangles up to the walk's end, of one all along the ray (until a leaf
  // counts the walk has no end there).
  constexpr int kDepth = 64;
  int node_stack[kDepth];
  float t0_stack[kDepth], t1_stack[kDepth];
  int sp = 0, rank = 0x7FFFFFFF;
  bool reached = false;  // a leaf that counts and begins before the hit
  // Leaves that may count: the lowest entry of each triangle in them.
  int open_first = 0x7FFFFFFF, open_tie = 0x7FFFFFFF;
  float t0 = 0.f, t1 = two ? rn_add(stop, tol) : as_float(0x7f800000);
  winner = kBvhNone;
  while (true) {
    HPT_DCHECK(err, node >= 0 && node < s.num_nodes, 110, node, return kLookupOpen);
    const uint2 nd = ldg(reinterpret_cast<const uint2*>(s.nodes) + node);
    const uint32_t axis = nd.x >> 30;
    if (axis != kLeafKind) {
      const float split = as_float_u(nd.y);
      const float iv = axis == 0 ? inv[0] : (axis == 1 ? inv[1] : inv[2]);
      const float oa = axis == 0 ? o[0] : (axis == 1 ? o[1] : o[2]);
      const float la = axis == 0 ? lo[0] : (axis == 1 ? lo[1] : lo[2]);
      const float ha = axis == 0 ? hi[0] : (axis == 1 ? hi[1] : hi[2]);
      // The side the ray is on before the split, and the one after it. Along
      // a zero component it stays on the origin's side, in the split plane
      // itself it touches both.
      const bool up = iv > 0.f || (iv == 0.f && oa <= split);
      const bool flat = iv == 0.f;
      const float ts = flat ? as_float(0x7f800000) : rn_mul(rn_sub(split, oa), iv);
      const bool before = (up ? la <= split : ha >= split) && t0 <= rn_add(ts, tol);
      const bool after = (up ? ha >= split : la <= split) &&
                         (flat ? oa == split : t1 >= rn_sub(ts, tol));
      const int child = (int)(nd.x & kIndexMask);
      const int near = child + (up ? 0 : 1), far = child + (up ? 1 : 0);
      const float far_t0 = flat ? t0 : fmaxf(t0, rn_sub(ts, tol));
      if (before && after) {
        if (sp >= kDepth) return kLookupOpen;
        node_stack[sp] = far;
        t0_stack[sp] = far_t0;
        t1_stack[sp] = t1;
        ++sp;
      }
      if (before) {
        node = near;
        t1 = fminf(t1, rn_add(ts, tol));
        continue;
      }
      if (after) {
        node = far;
        t0 = far_t0;
        continue;
      }
    } else {
      HPT_DCHECK(err, (int)(nd.x & kIndexMask) < s.num_leaves, 111, nd.x & kIndexMask,
                 return kLookupOpen);
      const float4* L = reinterpret_cast<const float4*>(s.leaves + (nd.x & kIndexMask));
      const float4 bl = ldg(L), bh = ldg(L + 1);
      const int begin = as_int(bl.w), count = as_int(bh.w);
      HPT_DCHECK(err, begin >= 0 && count >= 0 && (long long)begin + count <= s.num_leaf_tris,
                 112, begin, return kLookupOpen);
      int at = -1;  // the first entry of either
      uint32_t which = first;
#pragma unroll 4
      for (int k = count - 1; k >= 0; --k) {
        const int32_t entry = ldg(s.leaf_refs + begin + k);
        if (entry == id[0] || entry == id[1]) {
          at = begin + k;
          which = entry == id[0] ? first : tie;
        }
      }
      if (at >= 0) {
        const float l[3] = {bl.x, bl.y, bl.z}, h[3] = {bh.x, bh.y, bh.z};
        // The stretch of the ray that is in the leaf by more than the walk's
        // rounding (see part 2), and the one that is not outside by more.
        float f0 = 0.f, f1 = as_float(0x7f800000), g0 = 0.f, g1 = as_float(0x7f800000);
        bool inside = true, face = false;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          inside = inside && o[a] >= l[a] && o[a] <= h[a];
          if (inv[a] == 0.f) {
            if (!(o[a] >= l[a] && o[a] <= h[a])) f1 = g1 = -as_float(0x7f800000);
            face = face || o[a] == l[a] || o[a] == h[a];
            continue;
          }
          const float x0 = rn_mul(rn_sub(l[a], o[a]), inv[a]);
          const float x1 = rn_mul(rn_sub(h[a], o[a]), inv[a]);
          const float off =
              fma_rn(rn_mul(1.2e-7f, fmaxf(fabsf(l[a]), fabsf(h[a]))), fabsf(inv[a]), tol);
          f0 = fmaxf(f0, rn_add(fminf(x0, x1), off));
          f1 = fminf(f1, rn_sub(fmaxf(x0, x1), off));
          g0 = fmaxf(g0, rn_sub(fminf(x0, x1), off));
          g1 = fminf(g1, rn_add(fmaxf(x0, x1), off));
        }
        if (face && !inside) {
          // The filter's slab of the face the ray lies in is 0 / 0: rejected
          // (see tie_goes_right).
        } else if (face) {
          return kLookupOpen;  // the origin's own leaves: left to the walk
        } else if (f0 < f1 && f0 < rn_sub(stop, tol)) {
          // The ray crosses the leaf and the walk comes to it.
          if (at < rank) {
            rank = at;
            winner = which;
          }
          reached = reached || f0 < best_t;
          if (!two && reached) return kLookupHit;
        } else if (g0 <= g1 && !(two && g0 > rn_add(stop, tol))) {
          if (ref_box_test(r, bl, bh)) {
            if (which == first) open_first = at < open_first ? at : open_first;
            else open_tie = at < open_tie ? at : open_tie;
          }
        }
      }
    }
    if (sp == 0) break;
    --sp;
    node = node_stack[sp];
    t0 = t0_stack[sp];
    t1 = t1_stack[sp];
  }
  // They matter when they could bring in the other triangle, or any.
  if (reached) return (winner == first ? open_tie : open_first) < rank ? kLookupOpen : kLookupHit;
  return winner == kBvhNone && open_first == 0x7FFFFFFF && open_tie == 0x7FFFFFFF ? kLookupNone
                                                                                  : kLookupOpen;
}

// The tree walk for one triangle, or two at the same t, known to be nearest of
// all that are accepted: the same leaves in the same order, but only those
// entries of their lists are looked at, with the known t. True with the record
// of the one the walk reports, false when it passes the hit without one (the
// walk may then report another triangle).
template <class Sc>
__host__ __device__ __noinline__ bool walk_for(const Sc& s, const Ray& r, uint32_t first,
                                               uint32_t tie, float best_t, uint32_t& winner,
                                               DevErr* err) {
  TravState st;
  TravCold tc;
  trav_init(s, r, st, tc);
  if (tc.ties) return false;  // zero components: walks on several sides
  const int32_t id0 = as_int(ldg(reinterpret_cast<const float4*>(s.btris + first)).w);
  const int32_t id1 =
      tie == kBvhNone ? -1 : as_int(ldg(reinterpret_cast<const float4*>(s.btris + tie)).w);
  const float stop = rn_add(best_t, rn_add(rn_mul(best_t, 1e-4f), tc.slack));
  int rank = 0x7FFFFFFF;
  while (st.node >= 0) {
    const float px = rn_add(r.o.x, rn_mul(st.t_entry, r.d.x));
    const float py = rn_add(r.o.y, rn_mul(st.t_entry, r.d.y));
    const float pz = rn_add(r.o.z, rn_mul(st.t_entry, r.d.z));
    int node = st.node;
    uint2 nd = ldg(reinterpret_cast<const uint2*>(s.nodes) + node);
    while ((nd.x >> 30) != kLeafKind) {
      const uint32_t axis = nd.x >> 30;
      const float split = as_float_u(nd.y);
      const float p = axis == 0 ? px : (axis == 1 ? py : pz);
      const float dd = axis == 0 ? r.d.x : (axis == 1 ? r.d.y : r.d.z);
      node = (int)(nd.x & kIndexMask) + (p > split || (p == split && dd > 0.f) ? 1 : 0);
      HPT_DCHECK(err, node < s.num_nodes, 106, node, return false);
      nd = ldg(reinterpret_cast<const uint2*>(s.nodes) + node);
      if (++st.steps > s.max_steps) return false;
    }
    HPT_DCHECK(err, (int)(nd.x & kIndexMask) < s.num_leaves, 102, nd.x & kIndexMask,
               return false);
    const DevLeaf* L = s.leaves + (nd.x & kIndexMask);
    const float4 L0 = ldg(reinterpret_cast<const float4*>(L));
    const float4 L1 = ldg(reinterpret_cast<const float4*>(L) + 1);
    const int4 R03 = ldg(reinterpret_cast<const int4*>(L) + 2);
    const int2 R45 = ldg(reinterpret_cast<const int2*>(L) + 6);
    const int begin = as_int(L0.w), count = as_int(L1.w);
    HPT_DCHECK(err, begin >= 0 && count >= 0 && (long long)begin + count <= s.num_leaf_tris, 103,
               begin, return false);
    int at = -1;
    uint32_t which = first;
#pragma unroll 4
    for (int k = count - 1; k >= 0; --k) {
      const int32_t entry = ldg(s.leaf_refs + begin + k);
      if (entry == id0 || entry == id1) {
        at = begin + k;
        which = entry == id0 ? first : tie;
      }
    }
    if (at >= 0 && at < rank && ref_box_test(r, L0, L1)) {
      // A t before the first leaf that has the triangle (a ray in its plane):
      // the hierarchy left out what begins behind that t, the walk does not.
      if (st.t_entry > stop) return false;
      rank = at;
      winner = which;
    }
    float t_exit = as_float(0x7f800000);
    int rope = -1;
    const float tx = rn_mul(rn_sub(r.d.x > 0.f ? L1.x : L0.x, r.o.x), tc.inv_d.x);
    const float ty = rn_mul(rn_sub(r.d.y > 0.f ? L1.y : L0.y, r.o.y), tc.inv_d.y);
    const float tz = rn_mul(rn_sub(r.d.z > 0.f ? L1.z : L0.z, r.o.z), tc.inv_d.z);
    if (tx < t_exit) {
      t_exit = tx;
      rope = r.d.x > 0.f ? R03.y : R03.x;
    }
    if (ty < t_exit) {
      t_exit = ty;
      rope = r.d.y > 0.f ? R03.w : R03.z;
    }
    if (tz < t_exit) {
      t_exit = tz;
      rope = r.d.z > 0.f ? R45.y : R45.x;
    }
    // Before the hit is found the walk goes on at least this far, after it no
    // further.
    if (!(t_exit < tc.t_end) || rope < 0 || t_exit > stop) break;
    HPT_DCHECK(err, rope < s.num_nodes, 105, rope, return false);
    if (++st.steps > s.max_steps) return false;
    st.node = rope;
    st.t_entry = fmaxf(st.t_entry, t_exit);
  }
  return rank != 0x7FFFFFFF;
}

// Settles an open hit: sets the triangle's record (kBvhNone: a miss) and t of
// the tree walk's answer and returns true, or returns false when the tree has
// to be walked. A hit in leaves that do not count (the ray lies in a split
// plane) makes it search the hierarchy again for the nearest one that does.
template <class Sc>
HPT_HD bool bvh_settle(const Sc& s, const Ray& r, uint32_t& best, uint32_t tie, float& t,
                       DevErr* err) {
  uint32_t winner;
  const Lookup l = bvh_lookup(s, r, best, tie, t, winner, err);
  if (l == kLookupHit) {
    best = winner;
    return true;
  }
  if (l == kLookupOpen) {
    if ((best & kBvhMany) || (best & kBvhNone) == kBvhNone || !(t < as_float(0x7f800000)) ||
        !walk_for(s, r, best & kBvhNone, best & kBvhTie ? tie : kBvhNone, t, winner, err))
      return false;
    best = winner;
    return true;
  }
  BvhRay b;
  if (!bvh_init(r, s.scene_eps, b)) return false;
  uint2 stack[kBvhStack];
  while (true) {
    while (b.tri_bits) {
      const uint32_t before = b.best;
      const float before_t = b.best_t, before_cull = b.cull;
      uint32_t other = 0;
      bvh_test(s.btris, s.scene_eps, b, other);
      if (b.best == before) continue;
      if (b.best & (kBvhTie | kBvhMany)) return false;
      const Lookup c = bvh_lookup(s, r, b.best, 0u, b.best_t, winner, err);
      if (c == kLookupOpen) return false;
      if (c == kLookupNone) {
        b.best = before;
        b.best_t = before_t;
        b.cull = before_cull;
      }
    }
    if (!bvh_visit(s.bvh, (uint32_t)s.num_bvh, b, stack, err)) break;
  }
  best = b.best;
  t = b.best_t;
  return best != kBvhNone || bvh_no_parallel_edge(s, r.d);
}

// Of two triangles at the same t (best with kBvhTie, second), the record of the one the tree walk reports
// wherever it accepts it: when one's bounds hold the other's, every leaf that
// lists the inner one lists the outer one too, and with the smaller id the
// outer one stands before it there. kBvhNone when that does not settle it.
template <class Sc>
HPT_HD uint32_t bvh_outer(const Sc& s, uint32_t best, uint32_t second, DevErr* err) {
  const uint32_t first = best & kBvhNone;
  if ((best & kBvhMany) || first == kBvhNone) return kBvhNone;
  HPT_DCHECK(err, first < (uint32_t)s.num_btris && second < (uint32_t)s.num_btris, 117, second,
             return kBvhNone);
  float lo[2][3], hi[2][3];
  int32_t id[2];
  for (int k = 0; k < 2; ++k) {
    const float4* rec = reinterpret_cast<const float4*>(s.btris + (k ? second : first));
    const float4 A = ldg(rec), E1 = ldg(rec + 1), E2 = ldg(rec + 2);
    if ((uint32_t)as_int(E2.w) & (kTriIrregular | kTriUnordered)) return kBvhNone;
    id[k] = as_int(A.w);
    const float a[3] = {A.x, A.y, A.z}, e1[3] = {E1.x, E1.y, E1.z}, e2[3] = {E2.x, E2.y, E2.z};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float v1 = rn_add(a[c], e1[c]), v2 = rn_add(a[c], e2[c]);
      lo[k][c] = fminf(a[c], fminf(v1, v2));
      hi[k][c] = fmaxf(a[c], fmaxf(v1, v2));
    }
  }
  bool first_holds = id[0] < id[1], second_holds = id[1] < id[0];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    first_holds = first_holds && lo[0][c] <= lo[1][c] && hi[0][c] >= hi[1][c];
    second_holds = second_holds && lo[1][c] <= lo[0][c] && hi[1][c] >= hi[0][c];
  }
  return first_holds ? first : (second_holds ? second : kBvhNone);
}

// The whole query of one ray; the tree walk's answer (t and triangle id).
// The work of both walks is added to cnt (leaves: the tree walk's).
template <class Sc>
HPT_HD void bvh_query(const Sc& s, const Ray& r, int32_t& tri, float& t, DevErr* err,
                      TravCount& cnt, int* how = nullptr) {
  BvhRay b;
  bool ok = bvh_init(r, s.scene_eps, b);
  if (ok) {
    uint2 stack[kBvhStack];
    uint32_t tie = 0;
    while (true) {
      for (; b.tri_bits; ++cnt.tris) bvh_test(s.btris, s.scene_eps, b, tie);
      if (b.steps / kBvhStep > (uint32_t)s.max_steps) {
        hpt_atomic_or(&err->flags, 1u);
        break;
      }
      if (!bvh_visit(s.bvh, (uint32_t)s.num_bvh, b, stack, err)) break;
      ++cnt.nodes;
    }
    ok = bvh_certain(s, r, b.best, b.best_t, err);
    if (b.best & kBvhTie) {
      const uint32_t outer = bvh_outer(s, b.best, tie, err);
      if (outer != kBvhNone && bvh_certain(s, r, outer, b.best_t, err)) {
        b.best = outer;
        ok = true;
      }
    }
    if (!ok) ok = bvh_settle(s, r, b.best, tie, b.best_t, err);
  }
  if (how) *how = ok;
  if (ok) {
    tri = b.best == kBvhNone ? -1 : as_int(ldg(reinterpret_cast<const float4*>(s.btris + b.best)).w);
    t = b.best == kBvhNone ? 0.f : b.best_t;
    return;
  }
  TravState st;
  TravCold tc;
  trav_init(s, r, st, tc);
  while (!trav_leaf(s, st, tc, nullptr, 0, err, cnt)) {
  }
  tri = st.best.tri;
  t = st.best.rec >= 0 ? st.best.t : 0.f;
}

}  // namespace hpt
