// Host build of the closest-hit query through the hierarchy (bvh.cuh over
// build_bvh) beside the tree walk it must agree with (test infrastructure).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "../../hptracing_b200/csrc/bvh.cuh"
#include "../../hptracing_b200/csrc/bvh_build.h"
#include "../../hptracing_b200/csrc/scene_pack.h"

using namespace hpt;

namespace {
struct Emu {
  PackedScene pk;
  PackedBvh bvh;
  DevScene dev;
};
}  // namespace

extern "C" {

void* bvhemu_create(const hpt_scene_desc* d) {
  Emu* e = new Emu();
  if (pack_scene(*d, 8192, e->pk) != HPT_OK) {
    delete e;
    return nullptr;
  }
  DevScene& s = e->dev;
  memset(&s, 0, sizeof s);
  float scale = 0.f;
  for (int a = 0; a < 3; ++a) {
    s.root_lo[a] = e->pk.root_lo[a];
    s.root_hi[a] = e->pk.root_hi[a];
    scale = std::max({scale, std::fabs(s.root_lo[a]), std::fabs(s.root_hi[a]),
                      s.root_hi[a] - s.root_lo[a]});
  }
  s.scene_eps = 2e-5f * scale;
  s.max_steps = 1 << 30;
  build_bvh(d->points, d->triangles, e->pk, s.scene_eps, 0, e->bvh);
  s.nodes = e->pk.nodes.data();
  s.leaves = e->pk.leaves.data();
  s.leaf_refs = e->pk.refs.data();
  s.tris = e->pk.tris.data();
  s.num_nodes = (int32_t)e->pk.nodes.size();
  s.num_leaves = (int32_t)e->pk.leaves.size();
  s.num_leaf_tris = (int32_t)e->pk.refs.size();
  s.num_triangles = d->num_triangles;
  s.bvh = e->bvh.nodes.data();
  s.btris = e->bvh.tris.data();
  s.num_bvh = (int32_t)e->bvh.nodes.size();
  s.num_btris = (int32_t)e->bvh.tris.size();
  for (int a = 0; a < 3; ++a) {
    s.edge_keys[a] = e->bvh.edge_keys[a].data();
    s.num_edge_keys[a] = (int32_t)e->bvh.edge_keys[a].size();
  }
  return e;
}

void bvhemu_destroy(void* h) { delete static_cast<Emu*>(h); }

// counts: nodes, triangles, depth.
void bvhemu_shape(void* h, int32_t* counts) {
  const Emu* e = static_cast<Emu*>(h);
  counts[0] = (int32_t)e->bvh.nodes.size();
  counts[1] = (int32_t)e->bvh.tris.size();
  counts[2] = e->bvh.max_depth;
}

// Both walks per ray; certain: the hierarchy's answer was certified. Returns
// the error flags.
int bvhemu_query(void* h, int n, const float* o, const float* d, int32_t* tri, float* t,
                 int32_t* walk_tri, float* walk_t, int32_t* certain) {
  const DevScene& s = static_cast<Emu*>(h)->dev;
  DevErr err;
  memset(&err, 0, sizeof err);
  TravCount cnt{};
  for (int i = 0; i < n; ++i) {
    const Ray r{mk(o[3 * i], o[3 * i + 1], o[3 * i + 2]), mk(d[3 * i], d[3 * i + 1], d[3 * i + 2])};
    bvh_query(s, r, tri[i], t[i], &err, cnt, certain + i);
    TravState st;
    TravCold tc;
    trav_init(s, r, st, tc);
    while (!trav_leaf(s, st, tc, nullptr, 0, &err, cnt)) {
    }
    walk_tri[i] = st.best.tri;
    walk_t[i] = st.best.rec >= 0 ? st.best.t : 0.f;
  }
  return (int)err.flags;
}

}  // extern "C"
