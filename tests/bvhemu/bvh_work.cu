// What the hierarchy's query and the tree walk do for a set of rays (test
// infrastructure; the scene is bvh_emu.cu's).
#include "bvh_emu.cu"

// work: per ray, node visits and triangle tests of the query, then node steps,
// leaves and triangle tests of the tree walk.
extern "C" void bvhemu_work(void* h, int n, const float* o, const float* d, double* work) {
  const DevScene& s = static_cast<Emu*>(h)->dev;
  DevErr err;
  memset(&err, 0, sizeof err);
  TravCount query{}, walk{};
  for (int i = 0; i < n; ++i) {
    const Ray r{mk(o[3 * i], o[3 * i + 1], o[3 * i + 2]), mk(d[3 * i], d[3 * i + 1], d[3 * i + 2])};
    int32_t tri;
    float t;
    bvh_query(s, r, tri, t, &err, query);
    TravState st;
    TravCold tc;
    trav_init(s, r, st, tc);
    while (!trav_leaf(s, st, tc, nullptr, 0, &err, walk)) {
    }
  }
  work[0] = (double)query.nodes / n;
  work[1] = (double)query.tris / n;
  work[2] = (double)walk.nodes / n;
  work[3] = (double)walk.leaves / n;
  work[4] = (double)walk.tris / n;
}
