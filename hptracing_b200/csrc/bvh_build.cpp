// Builder of the 8-wide hierarchy of the closest-hit kernels.
//
// Boxes. A ray has to visit every triangle that the tree walk (traverse.cuh)
// would accept, and the FP32 Moller-Trumbore test accepts rays that pass
// beside the triangle. How far beside? With r = 2^-24, T = o - a, n = e1 x e2,
// S = |e1||e2|, det = -n.d = -c |n||d| (c: sine of the angle between ray and
// plane), the computed T.(d x e2) and d.(T x e1) are off by at most 7 r
// |T||d||e|, the computed det by 6 r |d| S, the reciprocal and the products by
// 2 r more. Let X = a + u e1 + v e2 for the computed u, v: an accepted X is a
// point of the triangle, and
//     (o - X) det = -d (n.T) + E,   |E| <= r |d| S (14 |T| + 8 max|e|).
// (1) So X is within W = r (14 |T| + 8 max|e|) / (c s) of the ray's line, s =
//     |n| / S, the sine of the angle at vertex a, and by the same steps the
//     computed t is off by no more than r (15 |T| + 8 max|e|) / (c s |d|). If c
//     s >= kGrazing, the ray meets a box around the triangle that is grown by
//     r (36 max-norm |T| + 40 max|e|) / kGrazing (the rest beyond W: where the
//     line's nearest point lies behind the origin). The walk grows boxes by the
//     first term (kBoxGrowth), the second is part of the box; kCullFactor
//     covers the error of t. [The first term is what makes origins far away
//     and triangles of any size come out right.]
// (2) If c s < kGrazing, the ray runs almost in the plane, and W is no bound.
//     But |n.(x - X)| <= |n| c |x - X| + |E| / |d| for every point x of the
//     ray: it stays within a thin slab around the plane, of height h = c |x -
//     X| + r (14 |T| + 8 max|e|) / s, and the tree walk only tests the triangle
//     in a leaf that lists it. So the ray meets the part of such a leaf that
//     lies in the slab. The wide box of a triangle holds these parts; it is
//     used for rays that are within kGrazing of the plane (a cone per child,
//     device_types.h). If s < kGrazing (slivers, no area), the leaves count
//     whole, for all rays.
//     A triangle with e1 and e2 exactly zero on one axis needs no wide box:
//     every rounded term of the test then carries d's component on that axis
//     or the distance along it, and (1) holds without c.
// A box kept in a node also covers the walk's own rounding (8 r of its largest
// coordinate; the leaf it is in is found by the rounded o + t d).
// What it costs: 14.6 node visits and 6.6 tests a ray on the 61k-triangle
// spheres and 19 and 7 on an 842k-triangle terrain, against 11.7 and 6.4, and
// 12.6 and 5.3 with boxes grown by a fiftieth of a triangle, which lost hits.
// (Wide boxes for all rays: 20 and 18, and 30 and 37. kGrazing 0.003 / 0.004 /
// 0.006 / 0.008: 18.4 / 18.4 / 19.3 / 20.5 visits and 7.3 / 7.2 / 7.2 / 7.3
// tests for the terrain's bounces, 7.2 / 5.4 / 4.5 / 4.2 for its camera rays.)
// Not covered: an accepted t = +inf (the answer where nothing else is hit),
// which takes a computed det of exactly zero: see bvh_no_parallel_edge.
//
// Tree. A binary tree by binned SAH (16 bins on three axes, object median
// where bins fail or the tree gets deep), opened greedily by surface area
// into nodes of up to eight children; children are placed in slots so that
// visiting slots in the order of the ray's octant runs roughly front to back.
// Splits are chosen for boxes 0.6 of the way from the triangle to its wide
// box. (Own bounds / 0.6 / wide boxes: 15.6 / 14.0 / 15.6 visits on the spheres,
// 18.1 / 17.8 / 19.0 on a terrain.)
#include "bvh_build.h"

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <mutex>
#include <thread>

#include "parallel.h"

namespace hpt {

namespace {

// f(i) for i below count, on up to `threads` threads.
template <class F>
void for_all(int threads, size_t count, F&& f) {
  const size_t step = std::max<size_t>(1, std::min<size_t>(256, count / (4 * (size_t)threads)));
  std::atomic<size_t> cursor{0};
  run_threads((int)std::min<size_t>(threads, count), [&] {
    for (size_t i = cursor.fetch_add(step); i < count; i = cursor.fetch_add(step))
      for (size_t k = i; k < std::min(count, i + step); ++k) f(k);
  });
}

struct Box {
  float lo[3], hi[3];
  void reset() {
    for (int a = 0; a < 3; ++a) {
      lo[a] = FLT_MAX;
      hi[a] = -FLT_MAX;
    }
  }
  void add(const Box& b) {
    for (int a = 0; a < 3; ++a) {
      lo[a] = std::min(lo[a], b.lo[a]);
      hi[a] = std::max(hi[a], b.hi[a]);
    }
  }
  bool holds(const Box& b) const {
    for (int a = 0; a < 3; ++a)
      if (b.lo[a] < lo[a] || b.hi[a] > hi[a]) return false;
    return true;
  }
  float half_area() const {
    if (!(lo[0] <= hi[0])) return 0.f;
    const float x = hi[0] - lo[0], y = hi[1] - lo[1], z = hi[2] - lo[2];
    return x * y + y * z + z * x;
  }
};

struct Prim {
  Box b;
  int32_t tri;
};

// A triangle's boxes (see the file comment).
struct TriBoxes {
  Box own, wide;
  float normal[3];   // unit, zero without area
  float graze;       // sine below which a ray counts as in the plane; >= 1: all
};

// What a child of a wide node stores.
struct ChildBoxes {
  Box own, wide;
  int8_t cone[4];
};

struct Node2 {
  Box b;
  int32_t left = -1, right = -1;  // -1: leaf
  int32_t begin = 0, count = 0;
};

constexpr int kBins = 16;
constexpr int kLeafTris = 3;
// Cost of a binary split over a triangle test: a visit of an eight-child node
// stands for up to seven splits. (0.25 / 0.5 / 1 / 2: 14.9 visits and 6.2 tests
// / 14.6, 6.6 / 14.4, 7.5 / 14.3, 8.0 a ray on the spheres.)
constexpr float kNodeCost = 0.5f;
constexpr int kMedianDepth = 40;
constexpr float kSplitBlend = 0.6f;
constexpr double kUlp = 1.0 / (1 << 24);
// Leaf entries and triangles per thread (about 2 ms of work).
constexpr size_t kWorkPerThread = 32768;
// Subtrees above this size take their wide box for all rays.
constexpr int32_t kMaxCone = 32768;

class Builder2 {
 public:
  std::vector<Prim>& prims;
  std::vector<Node2> nodes;
  std::atomic<int32_t> used{0};
  bool median;

  Builder2(std::vector<Prim>& p, bool median_only) : prims(p), median(median_only) {
    nodes.resize(2 * p.size());
  }

  void run(int threads) {
    used = 1;
    {
      std::lock_guard<std::mutex> lk(mu);
      queue.push_back({0, 0, (int32_t)prims.size(), 0});
      outstanding = 1;
    }
    run_threads(threads, [this] {
      try {
        worker();
      } catch (...) {  // the other workers must not wait for this one's task
        std::lock_guard<std::mutex> lk(mu);
        failed = true;
        cv.notify_all();
        throw;
      }
    });
    nodes.resize((size_t)used.load());
  }

 private:
  struct Task {
    int32_t node, begin, end, depth;
  };
  std::mutex mu;
  std::condition_variable cv;
  std::deque<Task> queue;
  int outstanding = 0;
  bool failed = false;
  static constexpr int32_t kTaskMin = 4096;

  void worker() {
    std::unique_lock<std::mutex> lk(mu);
    while (true) {
      cv.wait(lk, [&] { return failed || !queue.empty() || outstanding == 0; });
      if (failed || queue.empty()) return;
      const Task t = queue.front();
      queue.pop_front();
      lk.unlock();
      split(t);
      lk.lock();
      if (--outstanding == 0) cv.notify_all();
    }
  }

  void child(const Task& t) {
    if (t.end - t.begin > kTaskMin) {
      std::lock_guard<std::mutex> lk(mu);
      queue.push_back(t);
      ++outstanding;
      cv.notify_one();
    } else {
      split(t);
    }
  }

  void split(const Task& t) {
    Node2& n = nodes[t.node];
    Box b, c;
    b.reset();
    c.reset();
    for (int32_t i = t.begin; i < t.end; ++i) {
      const Box& p = prims[i].b;
      b.add(p);
      for (int a = 0; a < 3; ++a) {
        const float m = p.lo[a] + p.hi[a];
        c.lo[a] = std::min(c.lo[a], m);
        c.hi[a] = std::max(c.hi[a], m);
      }
    }
    n.b = b;
    n.begin = t.begin;
    n.count = t.end - t.begin;
    if (n.count == 1) return;
    int32_t mid = -1;
    if (!median && t.depth < kMedianDepth) {
      float cost = 0.f;
      mid = sah(t, c, cost);
      if (mid >= 0 && n.count <= kLeafTris &&
          n.count * b.half_area() <= kNodeCost * b.half_area() + cost)
        return;
    }
    if (mid <= t.begin || mid >= t.end) {
      if (n.count <= kLeafTris) return;
      mid = (t.begin + t.end) / 2;
      int axis = 0;
      for (int a = 1; a < 3; ++a)
        if (c.hi[a] - c.lo[a] > c.hi[axis] - c.lo[axis]) axis = a;
      std::nth_element(prims.begin() + t.begin, prims.begin() + mid, prims.begin() + t.end,
                       [axis](const Prim& x, const Prim& y) {
                         const float mx = x.b.lo[axis] + x.b.hi[axis];
                         const float my = y.b.lo[axis] + y.b.hi[axis];
                         return mx != my ? mx < my : x.tri < y.tri;
                       });
    }
    const int32_t l = used.fetch_add(2);
    n.left = l;
    n.right = l + 1;
    child({l, t.begin, mid, t.depth + 1});
    child({l + 1, mid, t.end, t.depth + 1});
  }

  // Partitions [begin, end) at the cheapest of the binned splits of all three
  // axes; returns the middle, or -1 when the centroids coincide. cost: the
  // split's summed area x count.
  int32_t sah(const Task& t, const Box& c, float& cost) {
    Box bins[3][kBins];
    int32_t cnt[3][kBins];
    float k[3];
    for (int a = 0; a < 3; ++a) {
      const float w = c.hi[a] - c.lo[a];
      k[a] = w > 0.f ? (kBins * 0.9999f) / w : 0.f;
      if (!(k[a] < FLT_MAX)) k[a] = 0.f;
      for (int i = 0; i < kBins; ++i) {
        bins[a][i].reset();
        cnt[a][i] = 0;
      }
    }
    auto bin = [&](const Box& p, int a) {
      const int i = (int)((p.lo[a] + p.hi[a] - c.lo[a]) * k[a]);
      return std::min(std::max(i, 0), kBins - 1);
    };
    for (int32_t i = t.begin; i < t.end; ++i)
      for (int a = 0; a < 3; ++a) {
        const int x = bin(prims[i].b, a);
        bins[a][x].add(prims[i].b);
        ++cnt[a][x];
      }
    float best = FLT_MAX;
    int axis = -1, at = 0;
    for (int a = 0; a < 3; ++a) {
      if (k[a] == 0.f) continue;
      float right[kBins];
      Box r;
      r.reset();
      int32_t rc = 0;
      for (int i = kBins - 1; i > 0; --i) {
        r.add(bins[a][i]);
        rc += cnt[a][i];
        right[i] = rc ? r.half_area() * rc : 0.f;
      }
      Box l;
      l.reset();
      int32_t lc = 0;
      for (int i = 1; i < kBins; ++i) {
        l.add(bins[a][i - 1]);
        lc += cnt[a][i - 1];
        if (lc == 0 || lc == t.end - t.begin) continue;
        const float v = l.half_area() * lc + right[i];
        if (v < best) {
          best = v;
          axis = a;
          at = i;
        }
      }
    }
    if (axis < 0) return -1;
    cost = best;
    auto m = std::partition(prims.begin() + t.begin, prims.begin() + t.end,
                            [&](const Prim& p) { return bin(p.b, axis) < at; });
    return (int32_t)(m - prims.begin());
  }
};

// Opens the binary tree into wide nodes.
struct Collapser {
  const std::vector<Node2>& in;
  const std::vector<Prim>& prims;
  const PackedScene& scene;
  const std::vector<std::atomic<uint32_t>>& flags;
  const std::vector<TriBoxes>& boxes;
  PackedBvh& out;
  struct Kids {
    int32_t slot[8];   // binary node of each slot, -1: free
  };
  std::vector<Kids> kids_of;

  struct Item {
    int32_t src;    // binary node
    uint32_t dst;   // wide node
    int depth;
  };

  // The nodes' structure in a fixed order, then their boxes on all threads.
  void run(int threads) {
    out.nodes.clear();
    out.nodes.reserve(prims.size() / 3 + 16);
    out.tris.clear();
    out.tris.reserve(prims.size());
    out.max_depth = 0;
    kids_of.clear();
    out.nodes.push_back(BvhNode());
    kids_of.push_back(Kids());
    std::vector<Item> todo{{0, 0, 0}};
    while (!todo.empty()) {
      const Item it = todo.back();
      todo.pop_back();
      emit(it, todo);
    }
    for_all(threads, out.nodes.size(), [&](size_t i) { fill(i); });
  }

  bool leaf(int32_t n) const { return in[n].left < 0; }

  void emit(const Item& it, std::vector<Item>& todo) {
    out.max_depth = std::max(out.max_depth, it.depth);
    int32_t kids[8];
    int n = 0;
    kids[n++] = it.src;
    // Open the inner child of the largest area until eight children are there.
    while (n < 8) {
      int best = -1;
      for (int i = 0; i < n; ++i)
        if (!leaf(kids[i]) &&
            (best < 0 || in[kids[i]].b.half_area() > in[kids[best]].b.half_area()))
          best = i;
      if (best < 0) break;
      const Node2& o = in[kids[best]];
      kids[best] = o.left;
      kids[n++] = o.right;
    }
    const Box& nb = in[it.src].b;
    // Slots: bit a of a slot set = far side along axis a. Greedy assignment
    // of the child whose centre lies furthest out in some free slot's
    // direction.
    Kids& w = kids_of[it.dst];
    std::fill(w.slot, w.slot + 8, -1);
    bool placed[8] = {};
    for (int k = 0; k < n; ++k) {
      float best = -FLT_MAX;
      int bc = -1, bs = -1;
      for (int c = 0; c < n; ++c) {
        if (placed[c]) continue;
        const Box& b = in[kids[c]].b;
        float d[3];
        for (int a = 0; a < 3; ++a) d[a] = (b.lo[a] + b.hi[a]) - (nb.lo[a] + nb.hi[a]);
        for (int s = 0; s < 8; ++s) {
          if (w.slot[s] >= 0) continue;
          float v = 0.f;
          for (int a = 0; a < 3; ++a) v += (s >> a & 1) ? d[a] : -d[a];
          if (v > best) {
            best = v;
            bc = c;
            bs = s;
          }
        }
      }
      if (bc < 0) break;  // not reached: a free slot and child remain
      w.slot[bs] = kids[bc];
      placed[bc] = true;
    }
    BvhNode node;
    memset(&node, 0, sizeof node);
    node.child_base = (uint32_t)out.nodes.size();
    node.tri_base = (uint32_t)out.tris.size();
    int inner = 0, tris = 0;
    uint32_t next = node.child_base;
    for (int s = 0; s < 8; ++s) {
      const int32_t src = w.slot[s];
      if (src < 0) continue;
      const Node2& c = in[src];
      if (!leaf(src)) {
        node.imask |= (uint8_t)(1u << s);
        ++inner;
        todo.push_back({src, next++, it.depth + 1});
        continue;
      }
      node.meta[s] = (uint8_t)((((1u << c.count) - 1u) << 5) | (uint32_t)tris);
      for (int32_t i = 0; i < c.count; ++i) out.tris.push_back(record(prims[c.begin + i].tri));
      tris += c.count;
    }
    out.nodes[it.dst] = node;
    out.nodes.resize(out.nodes.size() + inner);
    kids_of.resize(out.nodes.size());
  }

  // The boxes and planes of wide node i.
  void fill(size_t i) {
    ChildBoxes kids[8];
    Box all;
    all.reset();
    for (int s = 0; s < 8; ++s) {
      if (kids_of[i].slot[s] < 0) continue;
      kids[s] = child_boxes(in[kids_of[i].slot[s]]);
      all.add(kids[s].wide);
    }
    quantise(all, kids_of[i].slot, kids, out.nodes[i]);
  }

  // A subtree's box may be grown so that it holds the wide boxes of some of
  // its triangles; the others' wide boxes, and the cone around their normals,
  // make up the child's wide box. Of a few growths, the one with the smallest
  // expected area.
  ChildBoxes child_boxes(const Node2& c) const {
    ChildBoxes r;
    Box own, wide;
    own.reset();
    wide.reset();
    for (int32_t i = c.begin; i < c.begin + c.count; ++i) {
      own.add(boxes[(size_t)prims[i].tri].own);
      wide.add(boxes[(size_t)prims[i].tri].wide);
    }
    const int8_t never[4] = {0, 0, 0, -1};
    r.own = wide;
    r.wide = wide;
    memcpy(r.cone, never, 4);
    if (c.count > kMaxCone) return r;
    float extent = 0.f, best = wide.half_area();
    for (int a = 0; a < 3; ++a) extent = std::max(extent, own.hi[a] - own.lo[a]);
    for (const float g : {0.f, 0.02f, 0.07f, 0.2f}) {
      Box b;
      for (int a = 0; a < 3; ++a) {
        const float by = g * std::max(0.3f * extent, own.hi[a] - own.lo[a]);
        b.lo[a] = std::max(wide.lo[a], own.lo[a] - by);
        b.hi[a] = std::min(wide.hi[a], own.hi[a] + by);
      }
      Box w = b;
      int8_t around[4];
      const float part = cone(c, b, w, around);
      const float cost = b.half_area() + part * (w.half_area() - b.half_area());
      if (cost < best) {
        best = cost;
        r.own = b;
        r.wide = w;
        memcpy(r.cone, around, 4);
      }
      if (part == 0.f) break;  // b holds all: the larger ones cost more
    }
    return r;
  }

  // The cone for those of c's triangles whose wide boxes b does not hold;
  // adds these boxes to w. Returns the share of all directions it takes.
  float cone(const Node2& c, const Box& b, Box& w, int8_t around[4]) const {
    double axis[3] = {0, 0, 0}, length = 0;
    bool any = false, all = false;
    for (int32_t i = c.begin; i < c.begin + c.count; ++i) {
      const TriBoxes& t = boxes[(size_t)prims[i].tri];
      if (b.holds(t.wide)) continue;
      any = true;
      w.add(t.wide);
      all = all || t.graze >= 1.f;
      const double side =
          axis[0] * t.normal[0] + axis[1] * t.normal[1] + axis[2] * t.normal[2] < 0 ? -1 : 1;
      for (int a = 0; a < 3; ++a) axis[a] += side * t.normal[a];
    }
    const int8_t never[4] = {0, 0, 0, -1}, always[4] = {0, 0, 0, 1};
    memcpy(around, any ? always : never, 4);
    if (!any) return 0.f;
    for (int a = 0; a < 3; ++a) length += axis[a] * axis[a];
    length = std::sqrt(length);
    if (all || !(length > 1e-6)) return 1.f;
    // The axis in 127ths, and the largest |axis . d| of a direction within
    // some triangle's grazing angle of its plane; d's own bytes are off by up
    // to half a 127th.
    double q[3], norm = 0, off = 0, sine = 0;
    for (int a = 0; a < 3; ++a) {
      q[a] = std::nearbyint(127 * axis[a] / length);
      norm += q[a] * q[a];
      off += 0.501 * std::fabs(q[a]);
    }
    norm = std::sqrt(norm);
    for (int32_t i = c.begin; i < c.begin + c.count && sine < 1; ++i) {
      const TriBoxes& t = boxes[(size_t)prims[i].tri];
      if (b.holds(t.wide)) continue;
      const double dot = std::min(
          1.0, std::fabs(q[0] * t.normal[0] + q[1] * t.normal[1] + q[2] * t.normal[2]) / norm);
      // asin(graze) + the angle between normal and axis.
      const double angle = std::asin((double)t.graze) + std::acos(dot);
      sine = angle < 1.570 ? std::max(sine, std::sin(angle)) : 1;
    }
    const double s = std::ceil((127 * norm * sine + off) / 127 + 1e-3);
    if (sine >= 1 || s >= 127) return 1.f;
    for (int a = 0; a < 3; ++a) around[a] = (int8_t)q[a];
    around[3] = (int8_t)s;
    return (float)(s / 127);
  }

  BvhTri record(int32_t id) const {
    const DevTri& t = scene.tris[id];
    BvhTri r;
    memset(&r, 0, sizeof r);
    for (int a = 0; a < 3; ++a) {
      r.a[a] = t.a[a];
      r.e1[a] = t.e1[a];
      r.e2[a] = t.e2[a];
    }
    r.tri_id = id;
    r.flags = flags[(size_t)id].load(std::memory_order_relaxed);
    return r;
  }

  // Child planes rounded outward by at least 1/64 of a step, which covers the
  // walk's decoding error (1/512 of a step).
  static void quantise(const Box& nb, const int32_t slot[8], const ChildBoxes kids[8],
                       BvhNode& w) {
    for (int k = 0; k < 8; ++k) {
      const int8_t never[4] = {0, 0, 0, -1};
      memcpy(w.cone[k], slot[k] < 0 ? never : kids[k].cone, 4);
    }
    for (int a = 0; a < 3; ++a) {
      int e = -100;
      const double ext = (double)nb.hi[a] - nb.lo[a];
      double s = 0, p = 0;
      // Smallest step 2^e for which the margins fit 0..255.
      if (ext > 0) e = std::max(-100, std::ilogb(ext) - 8);
      for (;; ++e) {
        s = std::ldexp(1.0, e);
        float pf = (float)((double)nb.lo[a] - s / 32);
        while ((double)pf > (double)nb.lo[a] - s / 64) pf = std::nextafterf(pf, -INFINITY);
        p = pf;
        w.p[a] = pf;
        if (((double)nb.hi[a] - p) / s + 1.0 / 64 <= 255.0) break;
      }
      w.e[a] = (uint8_t)(e + 127);
      auto low = [&](double x) {
        return (uint8_t)std::min(255.0, std::max(0.0, std::floor((x - p) / s - 1.0 / 64)));
      };
      auto high = [&](double x) {
        return (uint8_t)std::min(255.0, std::max(0.0, std::ceil((x - p) / s + 1.0 / 64)));
      };
      for (int k = 0; k < 8; ++k) {
        if (slot[k] < 0) {
          // An empty slot: lower plane above the upper one (and a hit of it
          // adds no child).
          w.qlo[a][k] = w.wlo[a][k] = 255;
          w.qhi[a][k] = w.whi[a][k] = 0;
          continue;
        }
        w.qlo[a][k] = low(kids[k].own.lo[a]);
        w.qhi[a][k] = high(kids[k].own.hi[a]);
        w.wlo[a][k] = low(kids[k].wide.lo[a]);
        w.whi[a][k] = high(kids[k].wide.hi[a]);
      }
    }
  }
};

}  // namespace

namespace {

// Leaves whose closed box the closed box b touches.
int64_t touched_leaves(const PackedScene& scene, const Box& b) {
  int64_t count = 0;
  static thread_local std::vector<uint32_t> stack;
  stack.assign(1, 0u);
  while (!stack.empty()) {
    const DevNode& d = scene.nodes[stack.back()];
    stack.pop_back();
    const uint32_t axis = d.meta >> 30, child = d.meta & kIndexMask;
    if (axis == kLeafKind) {
      ++count;
      continue;
    }
    if (b.lo[axis] <= d.split) stack.push_back(child);
    if (b.hi[axis] >= d.split) stack.push_back(child + 1);
  }
  return count;
}

// DevScene::edge_keys of axis a, at most half full.
void edge_table(const std::vector<DevTri>& tris, int a, std::vector<float>& keys) {
  const int b = (a + 1) % 3, c = (a + 2) % 3;
  auto largest = [&](const DevTri& t) {
    // Within rounding: a direction as good as the edge's may have another
    // largest component.
    const double x = 1.000001 * std::fabs((double)t.e2[a]);
    return x > 0 && x >= std::fabs(t.e2[b]) && x >= std::fabs(t.e2[c]);
  };
  auto cell = [](double r) { return edge_cell((float)std::min(1.0, std::max(-1.0, r))); };
  size_t count = 0;
  for (const DevTri& t : tris) count += largest(t);
  keys.clear();
  if (count == 0) return;
  // (A regular mesh has far fewer directions than edges: grown as it fills.)
  std::vector<uint32_t> table;
  uint32_t buckets = 1;
  while (buckets < 1024 && buckets < count) buckets *= 2;
  for (;; buckets *= 4) {
    size_t used = 0;
    table.assign(4 * (size_t)buckets, 0u);
    for (const DevTri& t : tris) {
      if (!largest(t)) continue;
      const double r1 = (double)t.e2[b] / t.e2[a], r2 = (double)t.e2[c] / t.e2[a];
      for (uint32_t i = cell(r1 - kEdgeTolerance); i <= cell(r1 + kEdgeTolerance); ++i)
        for (uint32_t j = cell(r2 - kEdgeTolerance); j <= cell(r2 + kEdgeTolerance); ++j) {
          const uint32_t tag = edge_tag(i, j);
          size_t k = 4 * (size_t)edge_bucket(i, j, buckets);
          while (table[k] != 0 && table[k] != tag) k = k + 1 < table.size() ? k + 1 : 0;
          used += table[k] == 0;
          table[k] = tag;
        }
      if (used > table.size() / 2) break;
    }
    if (used <= table.size() / 2) break;
  }
  keys.resize(table.size());
  memcpy(keys.data(), table.data(), table.size() * sizeof(uint32_t));
}

// The codes of BvhTri::flags (bits 8-31) with face's at most that of a leaf that
// ends `gap` beyond it (gap <= 0: it does not).
uint32_t with_gap(uint32_t codes, int face, float gap, float unit) {
  if (!(gap > 0.f)) return codes;
  const int at = 8 + 4 * face;
  uint32_t c = 0;
  for (float x = unit; c < 15 && x <= gap; x *= 2) ++c;
  const uint32_t have = (codes >> at) & 15u;
  return c < have ? (codes & ~(15u << at)) | (c << at) : codes;
}
// Sets f's bits and takes the smaller code of each face.
void merge_flags(std::atomic<uint32_t>& flags, uint32_t f, uint32_t codes) {
  for (uint32_t have = flags.load(std::memory_order_relaxed);;) {
    uint32_t want = (have & 255u) | f;
    for (int at = 8; at < 32; at += 4)
      want |= std::min((have >> at) & 15u, (codes >> at) & 15u) << at;
    if (want == have || flags.compare_exchange_weak(have, want, std::memory_order_relaxed)) return;
  }
}

// Bounds that several threads grow.
struct SharedBox {
  std::atomic<float> lo[3], hi[3];
  void set(const Box& b) {
    for (int a = 0; a < 3; ++a) {
      lo[a].store(b.lo[a], std::memory_order_relaxed);
      hi[a].store(b.hi[a], std::memory_order_relaxed);
    }
  }
  Box get() const {
    Box b;
    for (int a = 0; a < 3; ++a) {
      b.lo[a] = lo[a].load(std::memory_order_relaxed);
      b.hi[a] = hi[a].load(std::memory_order_relaxed);
    }
    return b;
  }
  void add(const Box& b) {
    for (int a = 0; a < 3; ++a) {
      for (float x = lo[a].load(std::memory_order_relaxed);
           b.lo[a] < x && !lo[a].compare_exchange_weak(x, b.lo[a], std::memory_order_relaxed);) {
      }
      for (float x = hi[a].load(std::memory_order_relaxed);
           b.hi[a] > x && !hi[a].compare_exchange_weak(x, b.hi[a], std::memory_order_relaxed);) {
      }
    }
  }
};

// What the wide boxes need to know of a triangle.
struct Plane {
  double n[3];       // unit normal
  double graze;      // TriBoxes::graze
  double thickness;  // the slab's, beside graze times the distance
  bool wide;         // has a wide box
};
Plane plane_of(const DevTri& t, double scene_size) {
  Plane p;
  memset(&p, 0, sizeof p);
  double l1 = 0, l2 = 0, l = 0;
  bool flat = false;
  for (int a = 0; a < 3; ++a) {
    const int b = (a + 1) % 3, c = (a + 2) % 3;
    p.n[a] = (double)t.e1[b] * t.e2[c] - (double)t.e1[c] * t.e2[b];
    l1 += (double)t.e1[a] * t.e1[a];
    l2 += (double)t.e2[a] * t.e2[a];
    l += p.n[a] * p.n[a];
    flat = flat || (t.e1[a] == 0.f && t.e2[a] == 0.f);
  }
  l = std::sqrt(l);
  // (Of so small a triangle the test's products underflow: its error is not
  // relative any more. As one without area.)
  const double s = l1 * l2 > 1e-52 ? l / std::sqrt(l1 * l2) : 0;
  for (int a = 0; a < 3; ++a) p.n[a] = l > 0 ? p.n[a] / l : 0;
  p.graze = s > kGrazing ? kGrazing / s : 1;
  // (|T| is at most kMaxDistance sizes, an edge sqrt 3.)
  p.thickness = s > kGrazing ? 14 * kUlp * (kMaxDistance + 1) * scene_size / s : 0;
  p.wide = p.graze >= 1 || !flat;
  return p;
}

// Narrows leaf box b to where the slab of triangle t (bounds tb, plane p)
// passes. False when it does not.
bool clip_to_slab(const DevTri& t, const Box& tb, const Plane& p, Box& b) {
  if (p.graze >= 1) return true;
  double lo[3], hi[3], reach = 0, round = 0;
  for (int a = 0; a < 3; ++a) {
    const double x = p.n[a] * ((double)b.lo[a] - t.a[a]), y = p.n[a] * ((double)b.hi[a] - t.a[a]);
    lo[a] = std::min(x, y);
    hi[a] = std::max(x, y);
    const double far_off =
        std::max((double)b.hi[a] - tb.lo[a], (double)tb.hi[a] - b.lo[a]);
    reach += far_off * far_off;
    round = std::max({round, std::fabs((double)b.lo[a]), std::fabs((double)b.hi[a])});
  }
  // n.(x - a) within [-h, h] (the floats of a box are rounded outward).
  const double h = p.graze * std::sqrt(reach) + p.thickness + 4 * kUlp * round;
  for (int a = 0; a < 3; ++a) {
    const int c = (a + 1) % 3, d = (a + 2) % 3;
    const double l = -h - hi[c] - hi[d], m = h - lo[c] - lo[d];
    if (std::max(l, lo[a]) > std::min(m, hi[a])) return false;
    if (std::fabs(p.n[a]) < 1e-9) continue;
    const double x = t.a[a] + l / p.n[a], y = t.a[a] + m / p.n[a];
    b.lo[a] = std::max(b.lo[a], std::nextafterf((float)std::min(x, y), -INFINITY));
    b.hi[a] = std::min(b.hi[a], std::nextafterf((float)std::max(x, y), INFINITY));
  }
  return true;
}

}  // namespace

void build_bvh(const float* points, const int32_t* triangles, const PackedScene& scene,
               float scene_eps, int num_threads, PackedBvh& out) {
  const size_t n = scene.tris.size();
  // The work goes with the leaves' entries; a small scene builds in less than
  // it takes to start a thread.
  const size_t cores =
      num_threads > 0 ? (size_t)num_threads : std::max(1u, std::thread::hardware_concurrency());
  const int threads =
      (int)std::max<size_t>(1, std::min(cores, (n + scene.refs.size()) / kWorkPerThread));
  // Per triangle: its bounds and plane, the union of the leaves that list it,
  // how many do, its flags and its wide box.
  std::vector<Box> bounds(n);
  std::vector<Plane> planes(n);
  std::vector<SharedBox> wide(n), leaves(n);
  std::vector<std::atomic<int32_t>> listed(n);
  std::vector<std::atomic<uint32_t>> flags(n);
  // (scene_eps is 2e-5 of the scene's size.)
  const double scene_size = scene_eps / 2e-5;
  for_all(threads, n, [&](size_t i) {
    Box none;
    none.reset();
    leaves[i].set(none);
    listed[i].store(0, std::memory_order_relaxed);
    flags[i].store(~255u, std::memory_order_relaxed);
    bounds[i].reset();
    for (int k = 0; k < 3; ++k) {
      const float* v = points + 4 * (size_t)triangles[4 * i + k];
      for (int a = 0; a < 3; ++a) {
        bounds[i].lo[a] = std::min(bounds[i].lo[a], v[a]);
        bounds[i].hi[a] = std::max(bounds[i].hi[a], v[a]);
      }
    }
    planes[i] = plane_of(scene.tris[i], scene_size);
    wide[i].set(bounds[i]);
  });
  const float unit = kGapUnit * scene_eps;
  for_all(threads, scene.leaves.size(), [&](size_t l) {
    const DevLeaf& L = scene.leaves[l];
    Box b;
    for (int a = 0; a < 3; ++a) {
      b.lo[a] = L.lo[a];
      b.hi[a] = L.hi[a];
    }
    const int32_t* ids = scene.refs.data() + L.tri_begin;
    int32_t count = L.tri_count;
    bool ascending = true;
    for (int32_t k = 1; k < count; ++k) ascending = ascending && ids[k - 1] < ids[k];
    std::vector<int32_t> unique;
    if (!ascending) {  // a triangle may be there twice: it counts once
      unique.assign(ids, ids + count);
      std::sort(unique.begin(), unique.end());
      unique.erase(std::unique(unique.begin(), unique.end()), unique.end());
      ids = unique.data();
      count = (int32_t)unique.size();
    }
    for (int32_t k = 0; k < count; ++k) {
      const size_t id = (size_t)ids[k];
      leaves[id].add(b);
      listed[id].fetch_add(1, std::memory_order_relaxed);
      const Box& t = bounds[id];
      uint32_t f = ascending ? 0u : kTriUnordered, codes = ~0u;
      for (int a = 0; a < 3; ++a) {
        codes = with_gap(codes, 2 * a, t.lo[a] - b.lo[a], unit);
        codes = with_gap(codes, 2 * a + 1, b.hi[a] - t.hi[a], unit);
        if (b.lo[a] > t.hi[a] || b.hi[a] < t.lo[a]) f |= kTriIrregular;
      }
      merge_flags(flags[id], f, codes);
      Box part = b;
      if (planes[id].wide && !wide[id].get().holds(b) &&
          clip_to_slab(scene.tris[id], t, planes[id], part))
        wide[id].add(part);
    }
  });
  for_all(threads, n, [&](size_t i) {
    if (listed[i].load(std::memory_order_relaxed) != touched_leaves(scene, bounds[i]))
      flags[i].fetch_or(kTriIrregular, std::memory_order_relaxed);
  });
  for_all(threads, 3, [&](size_t a) { edge_table(scene.tris, (int)a, out.edge_keys[a]); });
  std::vector<TriBoxes> boxes(n);
  std::vector<Prim> prims;
  prims.reserve(n);
  for (size_t i = 0; i < n; ++i) {
    if (listed[i].load() == 0) continue;  // no leaf lists it: never tested
    TriBoxes& t = boxes[i];
    t.own = bounds[i];
    t.wide = wide[i].get();
    t.graze = (float)planes[i].graze;
    double edge = 0, coordinate = 0;
    for (int a = 0; a < 3; ++a) {
      t.normal[a] = (float)planes[i].n[a];
      edge = std::max({edge, std::fabs((double)scene.tris[i].e1[a]),
                       std::fabs((double)scene.tris[i].e2[a])});
      coordinate = std::max({coordinate, std::fabs((double)t.wide.lo[a]),
                             std::fabs((double)t.wide.hi[a])});
    }
    // (max|e| is at most sqrt 3 times the largest component.)
    const double pad = kUlp * (8 * coordinate + 70 * edge / kGrazing);
    Prim p;
    p.tri = (int32_t)i;
    for (int a = 0; a < 3; ++a) {
      t.own.lo[a] = std::nextafterf((float)(t.own.lo[a] - pad), -INFINITY);
      t.own.hi[a] = std::nextafterf((float)(t.own.hi[a] + pad), INFINITY);
      t.wide.lo[a] = std::nextafterf((float)(t.wide.lo[a] - pad), -INFINITY);
      t.wide.hi[a] = std::nextafterf((float)(t.wide.hi[a] + pad), INFINITY);
      p.b.lo[a] = t.own.lo[a] + kSplitBlend * (t.wide.lo[a] - t.own.lo[a]);
      p.b.hi[a] = t.own.hi[a] + kSplitBlend * (t.wide.hi[a] - t.own.hi[a]);
    }
    prims.push_back(p);
  }
  for (const bool median : {false, true}) {
    out.nodes.clear();
    if (prims.empty()) {
      out.nodes.assign(1, BvhNode());
      memset(&out.nodes[0], 0, sizeof(BvhNode));
      memset(out.nodes[0].qlo, 255, sizeof out.nodes[0].qlo);
      memset(out.nodes[0].wlo, 255, sizeof out.nodes[0].wlo);
      break;
    }
    Builder2 b2(prims, median);
    b2.run(threads);
    Collapser c{b2.nodes, prims, scene, flags, boxes, out, {}};
    c.run(threads);
    if (out.max_depth < kBvhStack - 1) break;
  }
  // Where the certificate's descent starts: the lowest tree node that holds
  // every leaf listing the triangle.
  for_all(threads, out.tris.size(), [&](size_t i) {
    BvhTri& t = out.tris[i];
    const Box b = leaves[(size_t)t.tri_id].get();
    uint32_t node = 0;
    while (true) {
      const DevNode& d = scene.nodes[node];
      const uint32_t axis = d.meta >> 30;
      if (axis == kLeafKind) break;
      if (b.hi[axis] <= d.split) node = d.meta & kIndexMask;
      else if (b.lo[axis] >= d.split) node = (d.meta & kIndexMask) + 1;
      else break;
    }
    t.start_node = (int32_t)node;
  });
}

}  // namespace hpt
