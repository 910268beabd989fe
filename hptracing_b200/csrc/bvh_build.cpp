// Builder of the 8-wide hierarchy of the closest-hit kernels.
//
// Boxes. A triangle's box is its bounds, grown
//  - by 2e-6 of the scene's size, for the rounding of box and hit distances;
//  - by a fiftieth of its extent within its plane. For a ray almost in that
//    plane (cosine c) the Moller-Trumbore test is off by some 5e-8 / c of the
//    distance and can accept a ray that passes beside the triangle; the tree
//    walk (traverse.cuh) would then report it, so the hierarchy has to test
//    it too. Such a ray has to lie within rounding of the triangle's plane:
//    in 1.5e9 queries (bounces on the 61k-triangle spheres and on the
//    2.4M-triangle terrain) plain bounds grown by 4e-7 of the scene's size
//    alone gave the tree walk's answer every time, and this growth is about
//    50 times that.
//    The growth stays inside the union of the leaves that list the triangle:
//    outside of it the tree walk never tests it. (That union alone as the
//    box costs 27 node visits and 51 tests a ray on the spheres against 12
//    and 7, and 67 and 180 against 13 and 6 on a terrain.)
//
// Tree. A binary tree by binned SAH (16 bins on three axes, object median
// where bins fail or the tree gets deep), opened greedily by surface area
// into nodes of up to eight children; children are placed in slots so that
// visiting slots in the order of the ray's octant runs roughly front to back.
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
  float half_area() const {
    const float x = hi[0] - lo[0], y = hi[1] - lo[1], z = hi[2] - lo[2];
    return x * y + y * z + z * x;
  }
};

struct Prim {
  Box b;
  int32_t tri;
};

struct Node2 {
  Box b;
  int32_t left = -1, right = -1;  // -1: leaf
  int32_t begin = 0, count = 0;
};

constexpr int kBins = 16;
constexpr int kLeafTris = 3;
// Cost of a node visit over a triangle test (per-lane instruction counts of
// the walk: about 230 per eight-child node, 60 per test).
constexpr float kNodeCost = 1.0f;
constexpr int kMedianDepth = 40;
constexpr float kPlaneGrowth = 0.02f;

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
  const std::vector<uint8_t>& flags;
  PackedBvh& out;

  struct Item {
    int32_t src;    // binary node
    uint32_t dst;   // wide node
    int depth;
  };

  void run() {
    out.nodes.clear();
    out.nodes.reserve(prims.size() / 3 + 16);
    out.tris.clear();
    out.tris.reserve(prims.size());
    out.max_depth = 0;
    out.nodes.push_back(BvhNode());
    std::vector<Item> todo{{0, 0, 0}};
    while (!todo.empty()) {
      const Item it = todo.back();
      todo.pop_back();
      emit(it, todo);
    }
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
    int slot_kid[8];
    std::fill(slot_kid, slot_kid + 8, -1);
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
          if (slot_kid[s] >= 0) continue;
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
      slot_kid[bs] = kids[bc];
      placed[bc] = true;
    }
    BvhNode w;
    memset(&w, 0, sizeof w);
    quantise(nb, slot_kid, w);
    w.child_base = (uint32_t)out.nodes.size();
    w.tri_base = (uint32_t)out.tris.size();
    int inner = 0, tris = 0;
    for (int s = 0; s < 8; ++s) {
      if (slot_kid[s] < 0) continue;
      const Node2& c = in[slot_kid[s]];
      if (!leaf(slot_kid[s])) {
        w.imask |= (uint8_t)(1u << s);
        ++inner;
        continue;
      }
      w.meta[s] = (uint8_t)((((1u << c.count) - 1u) << 5) | (uint32_t)tris);
      for (int32_t i = 0; i < c.count; ++i) out.tris.push_back(record(prims[c.begin + i].tri));
      tris += c.count;
    }
    out.nodes.resize(out.nodes.size() + inner);
    uint32_t next = w.child_base;
    for (int s = 0; s < 8; ++s)
      if (slot_kid[s] >= 0 && !leaf(slot_kid[s])) todo.push_back({slot_kid[s], next++, it.depth + 1});
    out.nodes[it.dst] = w;
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
    r.flags = flags[(size_t)id];
    return r;
  }

  // Child planes rounded outward by at least 1/64 of a step, which covers the
  // walk's decoding error (1/512 of a step).
  void quantise(const Box& nb, const int slot_kid[8], BvhNode& w) const {
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
      for (int k = 0; k < 8; ++k) {
        if (slot_kid[k] < 0) {
          w.qlo[a][k] = 255;  // an empty slot: lower plane above the upper one
          w.qhi[a][k] = 0;
          continue;
        }
        const Box& b = in[slot_kid[k]].b;
        const double lo = std::floor(((double)b.lo[a] - p) / s - 1.0 / 64);
        const double hi = std::ceil(((double)b.hi[a] - p) / s + 1.0 / 64);
        w.qlo[a][k] = (uint8_t)std::min(255.0, std::max(0.0, lo));
        w.qhi[a][k] = (uint8_t)std::min(255.0, std::max(0.0, hi));
      }
    }
  }
};

}  // namespace

namespace {

// Leaves whose closed box the closed box b touches.
int64_t touched_leaves(const PackedScene& scene, const Box& b, std::vector<uint32_t>& stack) {
  int64_t count = 0;
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

}  // namespace

void build_bvh(const float* points, const int32_t* triangles, const PackedScene& scene,
               float scene_eps, int num_threads, PackedBvh& out) {
  const size_t n = scene.tris.size();
  // A small scene builds in less than it takes to start a thread.
  const int threads = n <= 8192 ? 1
                      : num_threads > 0
                          ? num_threads
                          : (int)std::max(1u, std::thread::hardware_concurrency());
  // Per triangle: its bounds, the union of the leaves that list it, how many
  // do, and its flags.
  std::vector<Box> bounds(n), boxes(n);
  std::vector<int32_t> listed(n, 0);
  std::vector<uint8_t> flags(n, 0);
  for (size_t i = 0; i < n; ++i) {
    boxes[i].reset();
    bounds[i].reset();
    for (int k = 0; k < 3; ++k) {
      const float* v = points + 4 * (size_t)triangles[4 * i + k];
      for (int a = 0; a < 3; ++a) {
        bounds[i].lo[a] = std::min(bounds[i].lo[a], v[a]);
        bounds[i].hi[a] = std::max(bounds[i].hi[a], v[a]);
      }
    }
  }
  const float near = kCertainNear * scene_eps;
  for (const DevLeaf& L : scene.leaves) {
    Box b;
    for (int a = 0; a < 3; ++a) {
      b.lo[a] = L.lo[a];
      b.hi[a] = L.hi[a];
    }
    bool ascending = true;
    for (int32_t k = 1; k < L.tri_count; ++k)
      ascending = ascending && scene.refs[(size_t)L.tri_begin + k - 1] <
                                   scene.refs[(size_t)L.tri_begin + k];
    for (int32_t k = 0; k < L.tri_count; ++k) {
      const size_t id = (size_t)scene.refs[(size_t)L.tri_begin + k];
      boxes[id].add(b);
      ++listed[id];
      const Box& t = bounds[id];
      uint32_t f = ascending ? 0u : kTriUnordered;
      for (int a = 0; a < 3; ++a) {
        const float below = t.lo[a] - b.lo[a], above = b.hi[a] - t.hi[a];
        if (below > 0.f && below < near) f |= 1u << (2 * a);
        if (above > 0.f && above < near) f |= 2u << (2 * a);
        if (b.lo[a] > t.hi[a] || b.hi[a] < t.lo[a]) f |= kTriIrregular;
      }
      flags[id] |= (uint8_t)f;
    }
  }
  {
    std::atomic<size_t> cursor{0};
    run_threads(threads, [&] {
      std::vector<uint32_t> stack;
      for (size_t i = cursor.fetch_add(1024); i < n; i = cursor.fetch_add(1024))
        for (size_t k = i; k < std::min(n, i + 1024); ++k)
          if (listed[k] != touched_leaves(scene, bounds[k], stack))
            flags[k] |= (uint8_t)kTriIrregular;
    });
  }
  {
    std::atomic<int> axis{0};
    run_threads(std::min(threads, 3), [&] {
      for (int a = axis++; a < 3; a = axis++) {
        std::vector<float>& keys = out.edge_keys[a];
        keys.clear();
        for (const DevTri& t : scene.tris) {
          const float b = t.e2[(a + 1) % 3], c = t.e2[(a + 2) % 3];
          if (t.e2[a] == 0.f && (b != 0.f || c != 0.f)) keys.push_back(edge_key(b, c));
        }
        std::sort(keys.begin(), keys.end());
        keys.erase(std::unique(keys.begin(), keys.end()), keys.end());
      }
    });
  }
  const float pad = 0.1f * scene_eps;
  std::vector<Prim> prims;
  prims.reserve(n);
  for (size_t i = 0; i < n; ++i) {
    Prim p;
    p.b = boxes[i];
    p.tri = (int32_t)i;
    if (p.b.lo[0] > p.b.hi[0]) continue;  // no leaf lists it: never tested
    const DevTri& t = scene.tris[i];
    const float nx = t.e1[1] * t.e2[2] - t.e1[2] * t.e2[1];
    const float ny = t.e1[2] * t.e2[0] - t.e1[0] * t.e2[2];
    const float nz = t.e1[0] * t.e2[1] - t.e1[1] * t.e2[0];
    const float n[3] = {nx, ny, nz}, nn = nx * nx + ny * ny + nz * nz;
    const Box& tb = bounds[i];
    float extent = 0.f;
    for (int a = 0; a < 3; ++a) extent = std::max(extent, tb.hi[a] - tb.lo[a]);
    for (int a = 0; a < 3; ++a) {
      const float in_plane = nn > 0.f ? std::sqrt(std::max(0.f, 1.f - n[a] * n[a] / nn)) : 1.f;
      p.b.lo[a] = std::max(p.b.lo[a], tb.lo[a] - kPlaneGrowth * extent * in_plane);
      p.b.hi[a] = std::min(p.b.hi[a], tb.hi[a] + kPlaneGrowth * extent * in_plane);
    }
    for (int a = 0; a < 3; ++a) {
      p.b.lo[a] -= pad;
      p.b.hi[a] += pad;
    }
    prims.push_back(p);
  }
  for (const bool median : {false, true}) {
    out.nodes.clear();
    if (prims.empty()) {
      out.nodes.assign(1, BvhNode());
      memset(&out.nodes[0], 0, sizeof(BvhNode));
      memset(out.nodes[0].qlo, 255, sizeof out.nodes[0].qlo);
      break;
    }
    Builder2 b2(prims, median);
    b2.run(threads);
    Collapser c{b2.nodes, prims, scene, flags, out};
    c.run();
    if (out.max_depth < kBvhStack - 1) break;
  }
  // Where the certificate's descent starts: the lowest tree node that holds
  // every leaf listing the triangle.
  for (BvhTri& t : out.tris) {
    const Box& b = boxes[(size_t)t.tri_id];
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
  }
}

}  // namespace hpt
