// Closest-hit query through the 8-wide bounding volume hierarchy.
//
// The result is that of the tree walk in traverse.cuh, bit for bit: the
// minimum-t triangle over the tree leaves that pass the reference's box
// filter. A query runs in two parts:
//  1. The hierarchy's walk finds the nearest triangle of all the
//     Moller-Trumbore test accepts. Every triangle is tested once (the tree
//     lists it in every leaf it touches, ~50 times), with the same FP32
//     arithmetic. The boxes are grown by what that arithmetic can be off by
//     (build_bvh), so the tree walk, which tests some of the same triangles,
//     finds this triangle or none as near.
//  2. bvh_certain looks the hit up in the tree: it descends to the leaf that
//     holds the hit point and checks that the leaf lists the triangle and
//     that the ray runs through the leaf by more than rounding. Then the
//     leaf passes the reference's filter, and the tree walk, whose leaves
//     cover the ray up to its best hit, visits it: its answer is this one.
// A ray for which part 2 fails (hits at a leaf's corner, rays in a split
// plane) and one with two triangles at exactly the same t are walked through
// the tree instead.
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

// Walk state of one ray.
struct BvhRay {
  Ray ray;
  f3 inv;            // 1 / d
  float cull;        // boxes that start beyond it are skipped
  float slack;       // rounding slack in t units
  float best_t;      // nearest accepted t, +inf = none
  uint32_t best;     // its record in btris, kBvhNone = none; | kBvhTie when
                     // another triangle was accepted at exactly best_t
  uint32_t oct;      // bit a: the ray runs toward +a (slot order)
  uint32_t node_base, node_bits;  // pending children: base, imask << 8 | hits
  uint32_t tri_base, tri_bits;    // pending triangles
  int32_t sp;        // entries on the stack
};
constexpr uint32_t kBvhNone = 0x3FFFFFFFu, kBvhTie = 0x40000000u;

// Starts a walk. Returns false when the ray is to be walked through the tree
// instead (non-finite rays, directions of extreme length).
HPT_HD bool bvh_init(float scene_eps, const Ray& r, BvhRay& b) {
  b.ray = r;
  b.best = kBvhNone;
  b.best_t = b.cull = as_float(0x7f800000);
  b.sp = 0;
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
  b.oct = (b.inv.x > 0.f ? 1u : 0u) | (b.inv.y > 0.f ? 2u : 0u) | (b.inv.z > 0.f ? 4u : 0u);
  b.node_base = 0;
  b.node_bits = (1u << 8) | (1u << b.oct);
  b.slack = rn_div(scene_eps, dmax);
  return finite3(r.o) && finite3(r.d) && dmax > 1e-15f && dmax < 1e15f;
}

// The slots of a node whose boxes the ray enters before b.cull.
template <int k>
HPT_HD uint32_t bvh_slot(uint32_t nx, uint32_t ny, uint32_t nz, uint32_t fx, uint32_t fy,
                         uint32_t fz, const f3& S, const f3& O, float cull) {
  const float t0 = fmaxf(fmaxf(fma_rn(plane<k & 3>(nx), S.x, O.x), fma_rn(plane<k & 3>(ny), S.y, O.y)),
                         fmaxf(fma_rn(plane<k & 3>(nz), S.z, O.z), 0.f));
  const float t1 = fminf(fminf(fma_rn(plane<k & 3>(fx), S.x, O.x), fma_rn(plane<k & 3>(fy), S.y, O.y)),
                         fminf(fma_rn(plane<k & 3>(fz), S.z, O.z), cull));
  return t0 <= t1 ? 1u << k : 0u;
}

// Visits a node: sets the pending children and triangles.
HPT_HD void bvh_node(BvhRay& b, const uint4& n0, const uint4& n1, const uint4& n2,
                     const uint4& n3, const uint4& n4) {
  const uint32_t e = n0.w;
  f3 S, O;
  S.x = rn_mul(as_float_u((e & 255u) << 23), b.inv.x);
  S.y = rn_mul(as_float_u(((e >> 8) & 255u) << 23), b.inv.y);
  S.z = rn_mul(as_float_u(((e >> 16) & 255u) << 23), b.inv.z);
  O.x = fma_rn(-32768.f, S.x, rn_mul(rn_sub(as_float_u(n0.x), b.ray.o.x), b.inv.x));
  O.y = fma_rn(-32768.f, S.y, rn_mul(rn_sub(as_float_u(n0.y), b.ray.o.y), b.inv.y));
  O.z = fma_rn(-32768.f, S.z, rn_mul(rn_sub(as_float_u(n0.z), b.ray.o.z), b.inv.z));
  const bool px = b.oct & 1u, py = b.oct & 2u, pz = b.oct & 4u;
  uint32_t h = 0;
  // Words: n2 = lo x (2), lo y (2); n3 = lo z, hi x; n4 = hi y, hi z.
  {
    const uint32_t nx = px ? n2.x : n3.z, fx = px ? n3.z : n2.x;
    const uint32_t ny = py ? n2.z : n4.x, fy = py ? n4.x : n2.z;
    const uint32_t nz = pz ? n3.x : n4.z, fz = pz ? n4.z : n3.x;
    h |= bvh_slot<0>(nx, ny, nz, fx, fy, fz, S, O, b.cull);
    h |= bvh_slot<1>(nx, ny, nz, fx, fy, fz, S, O, b.cull);
    h |= bvh_slot<2>(nx, ny, nz, fx, fy, fz, S, O, b.cull);
    h |= bvh_slot<3>(nx, ny, nz, fx, fy, fz, S, O, b.cull);
  }
  {
    const uint32_t nx = px ? n2.y : n3.w, fx = px ? n3.w : n2.y;
    const uint32_t ny = py ? n2.w : n4.y, fy = py ? n4.y : n2.w;
    const uint32_t nz = pz ? n3.y : n4.w, fz = pz ? n4.w : n3.y;
    h |= bvh_slot<4>(nx, ny, nz, fx, fy, fz, S, O, b.cull);
    h |= bvh_slot<5>(nx, ny, nz, fx, fy, fz, S, O, b.cull);
    h |= bvh_slot<6>(nx, ny, nz, fx, fy, fz, S, O, b.cull);
    h |= bvh_slot<7>(nx, ny, nz, fx, fy, fz, S, O, b.cull);
  }
  const uint32_t imask = e >> 24;
  uint32_t inner = h & imask;
  // Hits by visiting order: slot s goes to bit s ^ oct, the highest first.
  if (b.oct & 1u) inner = ((inner & 0x55u) << 1) | ((inner >> 1) & 0x55u);
  if (b.oct & 2u) inner = ((inner & 0x33u) << 2) | ((inner >> 2) & 0x33u);
  if (b.oct & 4u) inner = ((inner & 0x0Fu) << 4) | (inner >> 4);
  b.node_base = n1.x;
  b.node_bits = (imask << 8) | inner;
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
    if (b.sp == 0) return false;
    const uint2 e = stack[--b.sp];
    b.node_base = e.x;
    b.node_bits = e.y;
  }
  const int bit = high_bit(b.node_bits & 255u);
  const uint32_t slot = (uint32_t)bit ^ b.oct;
  const uint32_t node = b.node_base + popc((b.node_bits >> 8) & ((1u << slot) - 1u));
  b.node_bits &= ~(1u << bit);
  if (b.node_bits & 255u) {
    HPT_DCHECK(err, b.sp < kBvhStack, 113, b.sp, return false);
    stack[b.sp].x = b.node_base;
    stack[b.sp].y = b.node_bits;
    ++b.sp;
  }
  HPT_DCHECK(err, node < num_bvh, 114, node, return false);
  const uint4* n = reinterpret_cast<const uint4*>(bvh + node);
  bvh_node(b, ldg(n), ldg(n + 1), ldg(n + 2), ldg(n + 3), ldg(n + 4));
  return true;
}

// One triangle test of the pending ones. A winning hit shrinks the cull
// distance to the tree walk's own stopping rule (best t plus slack).
HPT_HD void bvh_test(const BvhTri* btris, BvhRay& b) {
  const int k = high_bit(b.tri_bits);
  b.tri_bits &= ~(1u << k);
  const int32_t i = (int32_t)b.tri_base + k;
  const float4* rec = reinterpret_cast<const float4*>(btris + i);
  float t, u, v;
  if (mt_test(b.ray, ldg(rec), ldg(rec + 1), ldg(rec + 2), t, u, v)) {
    if (t < b.best_t) {
      b.best_t = t;
      b.best = (uint32_t)i;
      b.cull = fma_rn(t, 1.0001f, b.slack);
    } else if (t == b.best_t) {
      b.best |= kBvhTie;
    }
  }
}

// True when the tree walk's answer for ray r is (best, best_t), the result
// of its hierarchy walk (see the file comment); kBvhNone without kBvhTie: a
// miss.
template <class Sc>
HPT_HD bool bvh_certain(const Sc& s, const Ray& r, uint32_t best, float best_t, DevErr* err) {
  if (best & kBvhTie) return false;
  // Nothing accepted: a miss. Along a zero component a triangle with an edge
  // parallel to the ray can be "hit" at t = +inf (0 / 0 passes the tests),
  // which the reference reports when there is no other hit.
  if (best == kBvhNone) return r.d.x != 0.f && r.d.y != 0.f && r.d.z != 0.f;
  HPT_DCHECK(err, best < (uint32_t)s.num_btris, 115, best, return false);
  const float4* rec = reinterpret_cast<const float4*>(s.btris + best);
  const int32_t id = as_int(ldg(rec).w);
  int node = as_int(ldg(rec + 1).w);
  const float px = rn_add(r.o.x, rn_mul(best_t, r.d.x));
  const float py = rn_add(r.o.y, rn_mul(best_t, r.d.y));
  const float pz = rn_add(r.o.z, rn_mul(best_t, r.d.z));
  uint2 nd;
  while (true) {
    HPT_DCHECK(err, node >= 0 && node < s.num_nodes, 110, node, return false);
    nd = ldg(reinterpret_cast<const uint2*>(s.nodes) + node);
    const uint32_t axis = nd.x >> 30;
    if (axis == kLeafKind) break;
    const float split = as_float_u(nd.y);
    const float p = axis == 0 ? px : (axis == 1 ? py : pz);
    const float dd = axis == 0 ? r.d.x : (axis == 1 ? r.d.y : r.d.z);
    // In a split plane of a zero component the tree walk takes both sides.
    if (p == split && dd == 0.f) return false;
    node = (int)(nd.x & kIndexMask) + (p > split || (p == split && dd > 0.f) ? 1 : 0);
  }
  HPT_DCHECK(err, (int)(nd.x & kIndexMask) < s.num_leaves, 111, nd.x & kIndexMask, return false);
  const float4* L = reinterpret_cast<const float4*>(s.leaves + (nd.x & kIndexMask));
  const float4 lo = ldg(L), hi = ldg(L + 1);
  // Along a zero component the reference's filter wants the origin strictly
  // between the leaf's faces (0 / 0 on a face).
  if ((r.d.x == 0.f && !(r.o.x > lo.x && r.o.x < hi.x)) ||
      (r.d.y == 0.f && !(r.o.y > lo.y && r.o.y < hi.y)) ||
      (r.d.z == 0.f && !(r.o.z > lo.z && r.o.z < hi.z)))
    return false;
  // The ray's interval in the leaf, against rounding: 2e-6 of the scene's
  // size and 1e-6 of the distance (a face's distance is off by a few 1e-7).
  float t0 = 0.f, t1 = as_float(0x7f800000);
  const float o[3] = {r.o.x, r.o.y, r.o.z}, d[3] = {r.d.x, r.d.y, r.d.z};
  const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
#pragma unroll
  for (int a = 0; a < 3; ++a)
    if (d[a] != 0.f) {
      const float inv = rn_rcp(d[a]);
      const float x0 = rn_mul(rn_sub(l[a], o[a]), inv), x1 = rn_mul(rn_sub(h[a], o[a]), inv);
      t0 = fmaxf(t0, fminf(x0, x1));
      t1 = fminf(t1, fmaxf(x0, x1));
    }
  const float dmax = fmaxf(fabsf(r.d.x), fmaxf(fabsf(r.d.y), fabsf(r.d.z)));
  const float tol = fma_rn(best_t, 1e-6f, rn_mul(0.1f, rn_div(s.scene_eps, dmax)));
  if (!(rn_sub(t1, t0) > tol) || !(best_t > rn_sub(t0, tol)) || !(best_t < rn_add(t1, tol)))
    return false;
  const int begin = as_int(lo.w), count = as_int(hi.w);
  HPT_DCHECK(err, begin >= 0 && count >= 0 && (long long)begin + count <= s.num_leaf_tris, 112,
             begin, return false);
  for (int k = 0; k < count; ++k)
    if (ldg(s.leaf_refs + begin + k) == id) return true;
  return false;
}

// The whole query of one ray; the tree walk's answer (t and triangle id).
// The nodes, leaf groups and tests of both walks are added to cnt.
template <class Sc>
HPT_HD void bvh_query(const Sc& s, const Ray& r, int32_t& tri, float& t, DevErr* err,
                      TravCount& cnt, int* how = nullptr) {
  BvhRay b;
  bool ok = bvh_init(s.scene_eps, r, b);
  int steps = 0;
  if (ok) {
    uint2 stack[kBvhStack];
    while (true) {
      for (; b.tri_bits; ++cnt.tris, ++steps) bvh_test(s.btris, b);
      if (steps > s.max_steps) {
        hpt_atomic_or(&err->flags, 1u);
        break;
      }
      if (!bvh_visit(s.bvh, (uint32_t)s.num_bvh, b, stack, err)) break;
      ++cnt.nodes;
      ++steps;
      if (b.tri_bits) ++cnt.leaves;
    }
    ok = bvh_certain(s, r, b.best, b.best_t, err);
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
