// Wavefront path-tracing engine for sm_100a.
//
// Reference control flow (src/hp/trace_runner.cpp:116-356): primary rays are
// generated and intersected once per frame (misses write background *
// sample); then, per sample, every primary hit is shaded, branched and
// re-intersected up to `depth` shading passes, with blocking host reads of
// the stage sizes after every stage.
//
// Here the same per-path arithmetic runs as a regenerating wavefront over
// job slots (one job = one frame of one scene):
//   k_trace    - closest hit for the queue's rays, or for the camera rays of
//                newly admitted jobs, or both, with persistent warps that
//                refill idle lanes (ballot + one atomic per warp). A queue
//                ray's hit goes to the hit list, its miss adds background *
//                strength; camera hits go to a per-job cache, misses add
//                background * sample.
//   k_shade    - for each hit: self-emission, normal / UV / texture, branch
//                choice and next direction (s1_run + s2_*_run fused); new
//                (primary hit, sample) paths are started in the same pass
//                from the grants. Survivors are compacted (warp ballot +
//                block scan, one atomic per block) into the other queue;
//                finished paths flush their radiance. Hits that k_trace
//                leaves open are settled here first.
//                The last block advances queue counters and path cursors,
//                sets new jobs' path counts and grants the free wavefront
//                capacity to the active jobs in priority order (the host never
//                reads stage sizes).
//   k_resolve  - fixed-point accumulators -> get_image's tone map.
// Every random number is drawn from a stream keyed by (job, ray, sample,
// bounce) and radiance is summed in 2^-32 fixed point, so a job's image does
// not depend on how its paths are scheduled, batched or interleaved.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstring>
#include <numeric>

#include "bvh.cuh"
#include "engine.h"
#include "shading.cuh"
#include "traverse.cuh"

namespace hpt {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

struct EngineParams {
  DevJob* jobs;
  DevSlot* slots;
  int num_slots;
  DevCtrl* ctrl;
  const int32_t* order;
  int32_t* quota_slot;
  int32_t* quota_prefix;
  const int32_t* prim_slot;
  const int64_t* prim_prefix;
  // Primary passes over part of a job's rays (null: every entry covers its
  // job from ray 0 and completes its primary pass): entry e covers rays
  // [prim_first[e], prim_first[e] + its count); prim_final[e] != 0 marks
  // the part that completes the job's primary pass.
  const int64_t* prim_first;
  const int32_t* prim_final;
  int prim_n;
  // The queue of paths, double-buffered: k_shade reads queue c->parity and
  // writes the survivors to the other one, whose rays k_trace then traces.
  float4* Q_o[2];       // origin, ray index
  float4* Q_d[2];       // direction, sample << 8 | bounce
  float4* Q_s[2];       // strength, job slot
  float4* Q_r[2];       // radiance so far
  uint4* hits;          // rays that hit: (item, triangle, t bits, -)
  // Rays whose hits k_trace leaves open: (item, best, tie, t bits) as
  // bvh_settle takes them; the next k_shade settles them.
  uint4* open;
  int capacity;
  int refill;           // idle lanes that make a warp refill
  int rounds;           // warp rounds between refills
  // When every job of the launch renders the same scene (a frame, or a
  // batch over one scene): a copy of its DevScene in the kernel's parameter
  // space, whose pointers the walk then reads as constant operands. With
  // several scenes each lane keeps its own in registers.
  int uniform_scene;
  DevScene uscene;
};

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Index of the last prefix entry <= g (prefix[0] = 0, n entries).
template <typename T>
__device__ __forceinline__ int find_prefix(const T* prefix, int n, int64_t g) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((int64_t)prefix[mid] <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ int64_t job_rays(const DevJob& J) { return (int64_t)J.nx * J.ny; }

// Adds a path's radiance to its ray's fixed-point accumulator. Non-finite
// or out-of-range values set a marker so the resolve reproduces the float
// semantics (NaN stays NaN, +-inf saturates).
__device__ __forceinline__ void flush_radiance(const DevJob& J, int64_t ray, f3 rad) {
  const float v[3] = {rad.x, rad.y, rad.z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (v[c] == 0.f) continue;
    if (isnan(v[c])) {
      atomicOr(J.flags + ray, 1u << (4 * c));
    } else if (!(fabsf(v[c]) < 1073741824.0f)) {
      atomicOr(J.flags + ray, 1u << (4 * c + (v[c] > 0.f ? 1 : 2)));
    } else {
      const long long q = __double2ll_rn((double)v[c] * kAccumScale);
      atomicAdd(J.accum + 3 * ray + c, (unsigned long long)q);
    }
  }
}

// Counts finished paths per slot with one atomic per (warp, slot).
__device__ __forceinline__ void count_done(DevSlot* slots, bool done, int slot) {
  const unsigned m = __ballot_sync(kFull, done);
  if (!m) return;
  const unsigned same = __match_any_sync(kFull, done ? slot : -1);
  if (done && (__ffs(same & m) - 1) == (int)(threadIdx.x & 31))
    atomicAdd(&slots[slot].done, (unsigned long long)__popc(same & m));
}

// Counts the paths each slot sends on to be traced (one atomic per
// (warp, slot)).
__device__ __forceinline__ void count_queries(DevSlot* slots, bool alive, int slot) {
  const unsigned m = __ballot_sync(kFull, alive);
  if (!m) return;
  const unsigned same = __match_any_sync(kFull, alive ? slot : -1);
  if (alive && (__ffs(same & m) - 1) == (int)(threadIdx.x & 31))
    atomicAdd(&slots[slot].queries, (unsigned long long)__popc(same & m));
}

// A warp's counts for one slot, kept in shared memory by its lane 0 and added
// to the slot when another slot comes up and at the end of the kernel: one
// atomic on a slot's counter per 32 paths is what the warps would queue for
// when all paths are of one job.
struct Tally {
  int slot;
  uint32_t done, queries;
};

__device__ __forceinline__ void flush_tally(DevSlot* slots, Tally& w) {
  if ((threadIdx.x & 31) == 0) {
    if (w.done) atomicAdd(&slots[w.slot].done, (unsigned long long)w.done);
    if (w.queries) atomicAdd(&slots[w.slot].queries, (unsigned long long)w.queries);
    w.slot = 0;
    w.done = w.queries = 0;
  }
}

// Counts finished and surviving paths of the warp's lanes by slot.
__device__ __forceinline__ void count_paths(DevSlot* slots, Tally& w, bool done, bool alive,
                                            int slot) {
  const unsigned dm = __ballot_sync(kFull, done), am = __ballot_sync(kFull, alive);
  if (!(dm | am)) return;
  const int s = __shfl_sync(kFull, slot, __ffs(dm | am) - 1);
  if (__ballot_sync(kFull, (done || alive) && slot != s) == 0) {
    if ((threadIdx.x & 31) == 0) {
      if (w.slot != s) flush_tally(slots, w);
      w.slot = s;
      w.done += __popc(dm);
      w.queries += __popc(am);
    }
  } else {
    count_done(slots, done, slot);
    count_queries(slots, alive, slot);
  }
}

// Adds a warp's query and work counts to the control block (lane 0 calls).
__device__ __forceinline__ void add_counts(DevCtrl* c, uint32_t queries, uint32_t nodes,
                                           uint32_t leaves, uint32_t tests) {
#ifdef HPT_DEVICE_CHECKS
  if (queries) atomicAdd(&c->chk_isect_done, (int)queries);
#endif
  if (queries) atomicAdd(&c->isect_queries, (unsigned long long)queries);
  if (nodes) atomicAdd(&c->nodes_visited, (unsigned long long)nodes);
  if (leaves) atomicAdd(&c->leaves_visited, (unsigned long long)leaves);
  if (tests) atomicAdd(&c->tri_tests, (unsigned long long)tests);
}

// Grants the free wavefront capacity to active slots in priority order
// (one thread). A slot with nothing left to issue no longer needs grants.
__device__ void schedule(const EngineParams& P) {
  DevCtrl* c = P.ctrl;
  // Counts that other blocks of this launch added to are read past L1.
  const int budget =
      P.capacity - (__ldcg(&c->n_hit[c->parity]) + __ldcg(&c->n_open[c->parity]));
  int n_new = 0, nq = 0;
  bool remaining = false;
  // Paths the capped slots hold now, against their shared budget.
  int64_t capped = 0;
  if (c->capped_budget > 0)
    for (int k = 0; k < c->n_order; ++k) {
      const int s = P.order[k];
      if (s < 0 || s >= P.num_slots) continue;
      const DevSlot& S = P.slots[s];
      if (S.active && S.max_inflight > 0) capped += S.cursor - (int64_t)__ldcg(&S.done);
    }
  for (int k = 0; k < c->n_order; ++k) {
    const int s = P.order[k];
    HPT_DCHECK(&c->err, s >= 0 && s < P.num_slots, 231, s, continue);
    DevSlot& S = P.slots[s];
    S.alloc = 0;
    if (!S.active) continue;
    const int64_t rem = S.num_paths - S.cursor;
    if (rem <= 0) continue;
    remaining = true;
    int64_t grant = min(rem, (int64_t)(budget - n_new));
    // A capped job (e.g. a large request that must not crowd out the
    // latency-sensitive ones behind it) keeps at most max_inflight paths
    // started and unfinished.
    if (S.max_inflight > 0) {
      grant = min(grant, S.max_inflight - (S.cursor - (int64_t)__ldcg(&S.done)));
      if (c->capped_budget > 0) grant = min(grant, c->capped_budget - capped);
    }
    const int a = (int)grant;
    if (a <= 0) continue;
    if (S.max_inflight > 0) capped += a;
    S.alloc = a;
    P.quota_slot[nq] = s;
    P.quota_prefix[nq] = n_new;
    n_new += a;
    ++nq;
  }
  P.quota_prefix[nq] = n_new;
  c->n_quota = nq;
  c->n_new = n_new;
  c->done = (budget == P.capacity && !remaining) ? 1 : 0;
}

// ---------------------------------------------------------------------------
// Closest hits: queue rays and camera rays, persistent warps with lane refill.
// ---------------------------------------------------------------------------

// --- Camera rays of a launch's primary-pass entries (P.prim_*).
// Entry g: its slot and ray index within the job.
__device__ __forceinline__ bool prim_locate(const EngineParams& P, int64_t g, int& slot,
                                            int64_t& ray) {
  const int e = find_prefix(P.prim_prefix, P.prim_n, g);
  slot = P.prim_slot[e];
  ray = g - P.prim_prefix[e] + (P.prim_first ? P.prim_first[e] : 0);
  bool ok = true;
  HPT_DCHECK(&P.ctrl->err, slot >= 0 && slot < P.num_slots, 201, slot, ok = false);
  HPT_DCHECK(&P.ctrl->err, !ok || (ray >= 0 && ray < job_rays(P.jobs[slot])), 202, ray,
             ok = false);
  return ok;
}

// The job's camera ray (set_viewdirs / set_viewdirs_vr, kernel.cl:559-613).
__device__ __forceinline__ Ray prim_ray(const DevJob& J, int64_t ray) {
  const int x = (int)(ray % J.nx), y = (int)(ray / J.nx);
  const f3 d = J.pano ? pano_dir(x, y, J.vr_x_shift, J.ny)
                      : pinhole_dir(J.top, J.right, J.width, J.height, x, y, J.nx, J.ny);
  return Ray{mk(J.view_p[0], J.view_p[1], J.view_p[2]), d};
}

// Rays a warp has finished walking, waiting to be certified and written out
// 32 at a time with every lane busy (a lane that finishes takes its next ray
// at once). item: index in the queue, or -1 - ray for a camera ray of job slot
// `slot` (launches with camera rays). The lists are as short as their use
// allows: what they take of the SM's 256 KB, L1 does not have for nodes.
template <bool kPrim>
struct HitList {
  int32_t item[64];
  uint32_t best[64], tie[64];
  float t[64];
  int32_t slot[kPrim ? 64 : 1];
};
// Camera rays of a warp whose hits bvh_certain leaves open. Queue rays go to
// P.open for the next k_shade instead: a call in the walk's loop that settles
// them costs its registers (1.84 against 1.30 ms for the first bounce of 4M
// paths on the spheres scene), and one ray's tree walk at the end of a launch
// takes up to 0.65 ms, which k_shade has other work to hide behind. (The kernels
// that make the call have 1.4 to 1.8 KB of stack a thread and 280 to 400 bytes of
// spills, the queue form 272 and 12.)
struct OpenList {
  int32_t item[32], slot[32];
  uint32_t best[32], tie[32];
  float t[32];
};

// An open hit: looked up in the tree, and by the tree walk where that does not
// settle it. tri: -1 for a miss. Not inlined: few rays need it, and its
// registers must not weigh on the callers.
__device__ __noinline__ void settle(const DevScene& s, const Ray& r, uint32_t best, uint32_t tie,
                                    DevCtrl* c, int& tri, float& t) {
  if (bvh_settle(s, r, best, tie, t, &c->err)) {
    tri = best == kBvhNone
              ? -1
              : __float_as_int(__ldg(reinterpret_cast<const float4*>(s.btris + best)).w);
    return;
  }
  TravState st;
  TravCold tc;
  TravCount cnt{};
  trav_init(s, r, st, tc);
  while (!trav_leaf(s, st, tc, nullptr, 0, &c->err, cnt)) {
  }
  tri = st.best.rec >= 0 ? st.best.tri : -1;
  t = st.best.t;
  add_counts(c, 0, cnt.nodes, cnt.leaves, cnt.tris);
  if (cnt.repeats) atomicAdd(&c->tri_repeats, (unsigned long long)cnt.repeats);
}

// Writes out one camera ray per lane (`have`): a hit goes to its job's
// primary-hit cache; a miss adds the background (kernel.cl:193-206: the first
// pass assigns background * strength * sample_n with strength (1,1,1)). Every
// lane of the warp calls it.
__device__ __forceinline__ void write_camera(const EngineParams& P, bool have, int ray, int slot,
                                             const f3& dir, int tri, float t) {
  const int lane = threadIdx.x & 31;
  const bool hit = have && tri >= 0;
  const unsigned hm = __ballot_sync(kFull, hit);
  if (hm) {
    const unsigned same = __match_any_sync(kFull, hit ? slot : -1) & hm;
    const int leader = hit ? __ffs(same) - 1 : 0;
    int base = 0;
    if (hit && lane == leader) base = atomicAdd(P.jobs[slot].prim_count, __popc(same));
    base = __shfl_sync(kFull, base, leader);
    if (hit) {
      const DevJob& J = P.jobs[slot];
      int k = base + __popc(same & lanemask_lt());
      HPT_DCHECK(&P.ctrl->err, k < job_rays(J), 203, k, k = -1);
      if (k >= 0) {
        float4* dst = reinterpret_cast<float4*>(J.prim) + 2 * (size_t)k;
        dst[0] = make_float4(dir.x, dir.y, dir.z, __int_as_float(ray));
        dst[1] = make_float4(__int_as_float(tri), t, 0.f, 0.f);
      }
    }
  }
  if (have && !hit) {
    const DevJob& J = P.jobs[slot];
    const f3 val = scale((float)J.spp, mul(mk(J.bg[0], J.bg[1], J.bg[2]), mk(1.f, 1.f, 1.f)));
    flush_radiance(J, ray, val);
  }
}

__device__ __noinline__ void settle_camera(const EngineParams& P, const OpenList& W, int n) {
  const int lane = threadIdx.x & 31;
  const bool have = lane < n;
  int ray = 0, slot = 0, tri = -1;
  float t = 0.f;
  Ray r{};
  if (have) {
    ray = -1 - W.item[lane];
    slot = W.slot[lane];
    t = W.t[lane];
    const DevJob& J = P.jobs[slot];
    r = prim_ray(J, ray);
    settle(J.scene, r, W.best[lane], W.tie[lane], P.ctrl, tri, t);
  }
  __syncwarp();
  write_camera(P, have, ray, slot, r.d, tri, t);
}

// Hands over one open ray per lane (`want`); W / n: the warp's list of camera
// rays, worked off when it has no room. Returns its new length.
template <bool kQueue, bool kPrim>
__device__ __forceinline__ int push_open(const EngineParams& P, OpenList* W, int n, bool want,
                                         int item, int slot, uint32_t best, uint32_t tie,
                                         float t) {
  unsigned m = __ballot_sync(kFull, want);
  if (m == 0) return n;
  if constexpr (kQueue) {
    const bool queued = want && (!kPrim || item >= 0);
    const unsigned qm = __ballot_sync(kFull, queued);
    if (qm) {
      int base = 0;
      const int leader = __ffs(qm) - 1;
      if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(&P.ctrl->n_open[P.ctrl->parity ^ 1], __popc(qm));
      base = __shfl_sync(kFull, base, leader) + __popc(qm & lanemask_lt());
      bool ok = queued;
      HPT_DCHECK(&P.ctrl->err, !queued || base < P.capacity, 225, base, ok = false);
      if (ok) P.open[base] = make_uint4((uint32_t)item, best, tie, __float_as_uint(t));
    }
    m &= ~qm;
    want = want && !queued;
  }
  if constexpr (kPrim) {
    if (m) {
      if (n + __popc(m) > 32) {
        settle_camera(P, *W, n);
        n = 0;
        __syncwarp();
      }
      if (want) {
        const int k = n + __popc(m & lanemask_lt());
        W->item[k] = item;
        W->slot[k] = slot;
        W->best[k] = best;
        W->tie[k] = tie;
        W->t[k] = t;
      }
      __syncwarp();
      n += __popc(m);
    }
  }
  return n;
}

// True when the ray's strength is zero and its answer, whichever it is, adds
// zero to its path and ends it (a light sampled along the surface it lies in:
// the ray runs in a split plane, where a certain hit would take a look at the
// tree). The answer may be a miss: 0 times an infinite background is not zero.
// `s`: its scene.
__device__ __forceinline__ bool no_strength(const EngineParams& P, const DevScene& s, const Ray& r,
                                            int item) {
  const float4 w = P.Q_s[P.ctrl->parity ^ 1][item];
  if (w.x != 0.f || w.y != 0.f || w.z != 0.f || !s.finite_shading) return false;
  const int slot = __float_as_int(w.w);
  HPT_DCHECK(&P.ctrl->err, slot >= 0 && slot < P.num_slots, 222, slot, return false);
  const float* bg = P.jobs[slot].bg;
  return isfinite(bg[0]) && isfinite(bg[1]) && isfinite(bg[2]) && bvh_no_parallel_edge(s, r.d);
}

// Writes out one ray of the queue per lane (`have`): a hit goes to the hit
// list, a miss adds background * strength (kernel.cl:195-200, sample_n = 1)
// and ends its path. Every lane of the warp calls it.
__device__ __forceinline__ void write_queue(const EngineParams& P, bool have, int item, int tri,
                                            float t) {
  DevCtrl* c = P.ctrl;
  const int lane = threadIdx.x & 31;
  const int q = c->parity ^ 1;
  const bool hit = have && tri >= 0;
  const unsigned hm = __ballot_sync(kFull, hit);
  if (hm) {
    int base = 0;
    const int leader = __ffs(hm) - 1;
    if (lane == leader) base = atomicAdd(&c->n_hit[q], __popc(hm));
    base = __shfl_sync(kFull, base, leader) + __popc(hm & lanemask_lt());
    bool ok = hit;
    HPT_DCHECK(&c->err, !hit || base < P.capacity, 223, base, ok = false);
    if (ok) P.hits[base] = make_uint4((uint32_t)item, (uint32_t)tri, __float_as_uint(t), 0u);
  }
  const bool missed = have && tri < 0;
  int slot = 0;
  if (missed) {
    const float4 s4 = P.Q_s[q][item], r4 = P.Q_r[q][item];
    const int64_t ray = __float_as_int(P.Q_o[q][item].w);
    slot = __float_as_int(s4.w);
    bool ok = true;
    HPT_DCHECK(&c->err, slot >= 0 && slot < P.num_slots, 222, slot, ok = false);
    HPT_DCHECK(&c->err, !ok || (ray >= 0 && ray < job_rays(P.jobs[slot])), 224, ray, ok = false);
    if (ok) {
      const DevJob& J = P.jobs[slot];
      const f3 rad = mk(r4.x, r4.y, r4.z);
      flush_radiance(J, ray, add(rad, mul(mk(J.bg[0], J.bg[1], J.bg[2]), mk(s4.x, s4.y, s4.z))));
    }
  }
  count_done(P.slots, missed, slot);
}

// Certifies the finished rays [first, first + n) of the list, n <= 32, and
// writes them out, or hands them over as open. Returns W's new length.
template <bool kUniform, bool kQueue, bool kPrim>
__device__ __noinline__ int finish_rays(const EngineParams& P, const HitList<kPrim>& L, int first,
                                        int n, OpenList* W, int n_open) {
  DevCtrl* c = P.ctrl;
  const int lane = threadIdx.x & 31;
  const bool have = lane < n;
  int item = 0, slot = 0, tri = -1;
  uint32_t best = kBvhNone, tie = 0;
  float t = 0.f;
  bool certain = false, camera = false;
  Ray r{};
  if (have) {
    item = L.item[first + lane];
    best = L.best[first + lane];
    t = L.t[first + lane];
    camera = kPrim && (!kQueue || item < 0);
    if (camera) {
      slot = L.slot[kPrim ? first + lane : 0];
      r = prim_ray(P.jobs[slot], -1 - (int64_t)item);
    } else {
      const int q = c->parity ^ 1;
      const float4 o4 = P.Q_o[q][item], d4 = P.Q_d[q][item];
      r = Ray{mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z)};
      if (!kUniform) slot = __float_as_int(P.Q_s[q][item].w);
    }
    const DevScene& s = kUniform ? P.uscene : P.jobs[slot].scene;
    if (best & kBvhTie) {
      tie = L.tie[first + lane];
      const uint32_t outer = bvh_outer(s, best, tie, &c->err);
      if (outer != kBvhNone) best = outer;
    }
    certain = bvh_certain(s, r, best, t, &c->err);
    if (!certain && kQueue && !camera && best < kBvhNone && no_strength(P, s, r, item))
      certain = true;
    if (certain && best != kBvhNone)
      tri = __float_as_int(__ldg(reinterpret_cast<const float4*>(s.btris + best)).w);
  }
  __syncwarp();
  if (kQueue) write_queue(P, have && certain && !camera, item, tri, t);
  if (kPrim)
    write_camera(P, have && certain && camera, -1 - item, slot, r.d, tri, t);
  return push_open<kQueue, kPrim>(P, W, n_open, have && !certain, item, slot, best, tie, t);
}

// Sets the path count of primary-pass entry e's slot when the entry
// completes its job's primary pass. A slot whose primary pass is still
// partial stays as it was: inactive, or finished with nothing left to issue.
__device__ void activate_slot(const EngineParams& P, int e) {
  const int s = P.prim_slot[e];
  HPT_DCHECK(&P.ctrl->err, s >= 0 && s < P.num_slots, 232, s, return);
  if (P.prim_final && !P.prim_final[e]) return;
  DevSlot& S = P.slots[s];
  S.num_paths = (int64_t)__ldcg(P.jobs[s].prim_count) * P.jobs[s].spp;
  S.cursor = 0;
  S.done = 0;
  S.queries = 0;
  S.max_inflight = P.jobs[s].max_inflight;
  S.alloc = 0;
  S.active = 1;
}

// After a pass of camera rays: starts the paths of the slots whose primary
// pass completed and grants paths (one thread).
__device__ void admit(const EngineParams& P) {
#ifdef HPT_DEVICE_CHECKS
  HPT_DCHECK(&P.ctrl->err, __ldcg(&P.ctrl->chk_isect_done) == P.prim_prefix[P.prim_n], 243,
             P.ctrl->chk_isect_done, (void)0);
  P.ctrl->chk_isect_done = 0;
#endif
  for (int e = 0; e < P.prim_n; ++e) activate_slot(P, e);
  P.ctrl->prim_head = 0;
  schedule(P);
}

// Advances the queues and the path cursors, then grants paths (one thread).
__device__ void control(const EngineParams& P) {
  DevCtrl* c = P.ctrl;
#ifdef HPT_DEVICE_CHECKS
  HPT_DCHECK(&c->err, c->chk_shade_done == c->chk_shade_items, 241,
             (long long)c->chk_shade_items * 1000000 + c->chk_shade_done, (void)0);
  const int traced = __ldcg(&c->chk_isect_done);
  HPT_DCHECK(&c->err, traced == c->nR + (P.prim_n ? P.prim_prefix[P.prim_n] : 0), 242,
             (long long)c->nR * 1000000 + traced, (void)0);
  c->chk_shade_items = 0;
  c->chk_shade_done = 0;
  c->chk_isect_done = 0;
#endif
  for (int k = 0; k < c->n_quota; ++k) {
    DevSlot& S = P.slots[P.quota_slot[k]];
    S.cursor += S.alloc;
    S.alloc = 0;
  }
  c->nQ = c->nR;
  c->nR = 0;
  c->shade_head = 0;
  c->isect_head = 0;
  c->n_open[c->parity] = 0;
  c->n_hit[c->parity] = 0;
  c->parity ^= 1;
  c->iterations += 1;
  // Jobs whose primary pass the iteration's k_trace completed (kPrim).
  for (int e = 0; e < P.prim_n; ++e) activate_slot(P, e);
  schedule(P);
}

// The end of a launch's last block (one thread of it, after every block is
// done): a launch that ends with it needs none of its own for it.
__device__ __forceinline__ bool last_block(DevCtrl* c) {
  // What this block wrote happens before the last block's reads.
  __threadfence();
  __syncthreads();
  if (threadIdx.x != 0 || atomicAdd(&c->ticket, 1) != (int)gridDim.x - 1) return false;
  __threadfence();
  c->ticket = 0;
  return true;
}

// An iteration's control without a trace (the run's last).
__global__ void k_ctrl(EngineParams P) { control(P); }

// Test rounds run when at least this share (in eighths) of the warp's live
// lanes hold pending triangles.
#ifndef HPT_TEST_EIGHTHS
#define HPT_TEST_EIGHTHS 3
#endif

// kUniform: every job of the launch renders P.uscene. kQueue: traces the
// queue; kPrim: traces the camera rays of the launch's primary-pass
// entries (P.prim_*), after the queue's. The last block to finish advances the
// queues, starts the paths of the jobs whose primary pass completed and grants
// paths. A serving loop admits requests with both, with no launch of its own.
//
// A round of the warp runs one code path: a node visit for the lanes without
// pending triangles, or one triangle test for those with some.
template <int BS, int MINB, bool kUniform, bool kQueue, bool kPrim>
__global__ void __launch_bounds__(BS, MINB) k_trace(const __grid_constant__ EngineParams P) {
  __shared__ HitList<kPrim> hit_lists[BS / 32];
  __shared__ OpenList open_lists[kPrim ? BS / 32 : 1];
  HitList<kPrim>& L = hit_lists[threadIdx.x >> 5];
  OpenList* W = open_lists + (kPrim ? threadIdx.x >> 5 : 0);
  DevCtrl* c = P.ctrl;
  const int q = c->parity ^ 1;
  const int n = kQueue ? c->nR : 0;
  const int64_t total = kPrim ? (int64_t)n + P.prim_prefix[P.prim_n] : (int64_t)n;
  unsigned long long* head = kQueue ? &c->isect_head : &c->prim_head;
  const int lane = threadIdx.x & 31;
  bool active = false;
  BvhRay b;
  b.tri_bits = 0;
  // The node stack (at most kBvhStack - 1 entries); its last word holds the
  // other triangle of a tie.
  uint2 stack[kBvhStack];
  // The lane's ray (as HitList), read when it finishes: kept out of the
  // registers the walk needs.
  __shared__ int item_sh[BS], slot_sh[kPrim ? BS : 1];
  int& my_item = item_sh[threadIdx.x];
  int& my_slot = slot_sh[kPrim ? threadIdx.x : 0];
  const BvhNode* bvh = P.uscene.bvh;
  const BvhTri* btris = P.uscene.btris;
  uint32_t num_bvh = (uint32_t)P.uscene.num_bvh;
  float eps = P.uscene.scene_eps;
  uint32_t max_steps = (uint32_t)P.uscene.max_steps;
  // The warp's counts and list lengths (the same value in every lane).
  uint32_t queries = 0, nodes = 0, tests = 0;
  int n_hits = 0, n_open = 0;
  // Once a refill finds the rays exhausted the warp stops asking, so the
  // cursor overshoots by at most one grab per warp.
  bool drained = false;
  while (true) {
    const unsigned idle = __ballot_sync(kFull, !active);
    if (!drained && __popc(idle) >= P.refill) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(head, (unsigned long long)__popc(idle));
      base = __shfl_sync(kFull, base, 0);
      drained = (int64_t)base + __popc(idle) >= total;
      bool started = false, walk = false;
      int item = 0, slot = 0;
      if (!active) {
        const int64_t i = (int64_t)base + __popc(idle & lanemask_lt());
        Ray r{};
        if (kPrim && i >= n && i < total) {
          int64_t ray = 0;
          if (prim_locate(P, i - n, slot, ray)) {
            r = prim_ray(P.jobs[slot], ray);
            item = -1 - (int)ray;
            started = true;
          }
        }
        if (kQueue && i < n) {
          bool ok = true;
          HPT_DCHECK(&c->err, i < P.capacity, 221, i, ok = false);
          if (ok) {
            const float4 o4 = P.Q_o[q][i], d4 = P.Q_d[q][i];
            if (!kUniform) {
              slot = __float_as_int(P.Q_s[q][i].w);
              HPT_DCHECK(&c->err, slot >= 0 && slot < P.num_slots, 222, slot, ok = false);
            }
            r = Ray{mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z)};
            item = (int)i;
            started = ok;
          }
        }
        if (started) {
          my_item = item;
          if (kPrim) my_slot = slot;
          if (!kUniform) {
            const DevScene& s = P.jobs[slot].scene;
            bvh = s.bvh;
            btris = s.btris;
            num_bvh = (uint32_t)s.num_bvh;
            max_steps = (uint32_t)s.max_steps;
            eps = s.scene_eps;
          }
          active = bvh_init(r, eps, b);
          walk = !active;
        }
      }
      queries += __popc(__ballot_sync(kFull, started));
      // kBvhMany: straight to the tree walk.
      n_open = push_open<kQueue, kPrim>(P, W, n_open, walk, item, slot, kBvhMany, 0, 0.f);
    }
    if (__ballot_sync(kFull, active) == 0) {
      if (drained) break;
      continue;
    }
    bool finished = false;
    for (int u = 0; u < P.rounds; ++u) {
      const bool go = active && !finished;
      const unsigned lm = __ballot_sync(kFull, go);
      if (lm == 0) break;
      const bool testing = go && b.tri_bits != 0;
      const unsigned tm = __ballot_sync(kFull, testing);
      // Every round moves a lane on: a test round needs a testing lane, a
      // visit round one that is not.
      if (tm != 0 && 8 * __popc(tm) >= HPT_TEST_EIGHTHS * __popc(lm)) {
        if (testing) bvh_test(btris, eps, b, stack[kBvhStack - 1].x);
        tests += __popc(tm);
      } else {
        if (go && !testing) finished = !bvh_visit(bvh, num_bvh, b, stack, &c->err);
        nodes += __popc(lm & ~tm);
      }
      if (go) {
        if (((b.node_bits & 255u) | b.tri_bits | (b.steps & 31u)) == 0) finished = true;
        if (b.steps / kBvhStep > max_steps) {
          atomicOr(&c->err.flags, 1u);
          finished = true;
        }
      }
    }
    const unsigned fm = __ballot_sync(kFull, finished);
    if (finished) {
      const int k = n_hits + __popc(fm & lanemask_lt());
      L.item[k] = my_item;
      L.best[k] = b.best;
      if (b.best & kBvhTie) L.tie[k] = stack[kBvhStack - 1].x;
      L.t[k] = b.best_t;
      if (kPrim) L.slot[kPrim ? k : 0] = my_slot;
      active = false;
    }
    n_hits += __popc(fm);
    __syncwarp();
    if (n_hits >= 32) {
      n_hits -= 32;
      n_open = finish_rays<kUniform, kQueue, kPrim>(P, L, n_hits, 32, W, n_open);
      __syncwarp();
    }
  }
  if (n_hits) n_open = finish_rays<kUniform, kQueue, kPrim>(P, L, 0, n_hits, W, n_open);
  if constexpr (kPrim) {
    if (n_open) settle_camera(P, *W, n_open);
  }
  if (lane == 0) add_counts(c, queries, nodes, 0, tests);
  if (last_block(c)) {
    if (kQueue) control(P);
    else admit(P);
  }
}

// Settles open ray i of the queue of nQ paths with parity par: its hit as
// P.hits would hold it, with triangle -1 for a miss. Called before anything of
// the item is loaded: what is live across the call is spilled.
__device__ __noinline__ void settle_queued(const EngineParams& P, int i, int par, int nQ,
                                           uint4& hit) {
  const uint4 e = P.open[i];
  const int item = (int)e.x;
  hit = make_uint4(e.x, 0xFFFFFFFFu, 0u, 0u);
  if (item < 0 || item >= nQ) return;  // the caller's check 211
  const float4 o = P.Q_o[par][item], d = P.Q_d[par][item];
  const int slot = __float_as_int(P.Q_s[par][item].w);
  HPT_DCHECK(&P.ctrl->err, slot >= 0 && slot < P.num_slots, 212, slot, return);
  int tri = -1;
  float t = __uint_as_float(e.w);
  settle(P.jobs[slot].scene, Ray{mk(o.x, o.y, o.z), mk(d.x, d.y, d.z)}, e.y, e.z, P.ctrl, tri, t);
  hit.y = (uint32_t)tri;
  hit.z = __float_as_uint(t);
}

// ---------------------------------------------------------------------------
// Shade + next direction (+ new paths), compacting survivors into R.
// ---------------------------------------------------------------------------
// Bound by gather latency with half of its lanes idle (the four kinds of next
// ray; DRAM at 18 % of its rate): hence the one copy of the random direction
// for two of them (shading.cuh), no atomic that all warps queue for (count_paths,
// the block's one cursor step and one queue step for BS items - one of each per
// warp costs 5 % more), and 32 warps per SM against spills (400 bytes, around the
// call that settles open hits). Over the 58 M paths of 512x512x64 on 61,476
// triangles: 6.94 ms before these three, 6.26 with them.
// MINB: blocks of BS threads per SM the register budget must fit (1 leaves the
// compiler's natural allocation of ~150); the tuning chooses.
// kUniform: every job renders P.uscene, whose pointers are constant operands.
template <int BS, int MINB, bool kUniform>
__global__ void __launch_bounds__(BS, MINB) k_shade(const __grid_constant__ EngineParams P) {
  __shared__ int warp_counts[BS / 32];
  __shared__ int block_base;
  __shared__ Tally tallies[BS / 32];
  DevCtrl* c = P.ctrl;
  const int par = c->parity;
  const int n_open = c->n_open[par], n_hit = c->n_hit[par], nQ = c->nQ;
  const int n_new = c->n_new, n_quota = c->n_quota;
  const int n_items = n_open + n_hit + n_new;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Tally& tally = tallies[warp];
  if (lane == 0) tally = Tally{0, 0, 0};
  unsigned long long shades = 0;
#ifdef HPT_DEVICE_CHECKS
  if (blockIdx.x == 0 && threadIdx.x == 0) c->chk_shade_items = n_items;
  int chk_items = 0;
#endif
  // The open hits come first (one may take a tree walk), and blocks take their
  // next items from a cursor, so the others go on meanwhile.
  while (true) {
    if (threadIdx.x == 0) block_base = atomicAdd(&c->shade_head, BS);
    __syncthreads();
    const int base = block_base;
    if (base >= n_items) break;
    const int i = base + threadIdx.x;
#ifdef HPT_DEVICE_CHECKS
    if (i < n_items) ++chk_items;
#endif
    bool alive = false, ended = false;
    int slot = 0;
    float4 oo, dd, ss, rr;
    if (i < n_items) {
      int sample = 0, bounce = 0, tri = -1;
      int64_t ray = -1;
      f3 o, d, strength, rad;
      float t = 0.f;
      bool ok = true;
      if (i < n_open + n_hit) {
        uint4 h;
        if (i < n_open) settle_queued(P, i, par, nQ, h);
        else h = P.hits[i - n_open];
        const int item = (int)h.x;
        HPT_DCHECK(&c->err, item >= 0 && item < nQ, 211, item, ok = false);
        if (ok) {
          const float4 qo = P.Q_o[par][item], qd = P.Q_d[par][item], qs = P.Q_s[par][item],
                       qr = P.Q_r[par][item];
          tri = (int)h.y;
          t = __uint_as_float(h.z);
          o = mk(qo.x, qo.y, qo.z);
          ray = __float_as_int(qo.w);
          d = mk(qd.x, qd.y, qd.z);
          const uint32_t meta = __float_as_uint(qd.w);
          sample = (int)(meta >> 8);
          bounce = (int)(meta & 0xFF);
          strength = mk(qs.x, qs.y, qs.z);
          slot = __float_as_int(qs.w);
          rad = mk(qr.x, qr.y, qr.z);
          HPT_DCHECK(&c->err, slot >= 0 && slot < P.num_slots, 212, slot, ok = false);
          if (ok && tri < 0) {
            // kernel.cl:195-200: miss adds background * strength (sample_n = 1).
            const DevJob& J = P.jobs[slot];
            HPT_DCHECK(&c->err, ray >= 0 && ray < job_rays(J), 224, ray, ok = false);
            if (ok) flush_radiance(J, ray, add(rad, mul(mk(J.bg[0], J.bg[1], J.bg[2]), strength)));
            ended = ok;
            ok = false;
          }
        }
      } else {
        const int off = i - n_open - n_hit;
        const int e = find_prefix(P.quota_prefix, n_quota, off);
        slot = P.quota_slot[e];
        HPT_DCHECK(&c->err, slot >= 0 && slot < P.num_slots, 212, slot, ok = false);
        if (ok) {
          const DevJob& J = P.jobs[slot];
          const int64_t q = P.slots[slot].cursor + (off - P.quota_prefix[e]);
          const int nh = *J.prim_count;
          HPT_DCHECK(&c->err, nh > 0 && q < (int64_t)nh * J.spp, 213, q, ok = false);
          HPT_DCHECK(&c->err, !ok || nh <= job_rays(J), 217, nh, ok = false);
          if (ok) {
            sample = q <= 0xFFFFFFFFll ? (int)((uint32_t)q / (uint32_t)nh) : (int)(q / nh);
            const int64_t k = q - (int64_t)sample * nh;
            bounce = 0;
            const float4* src = reinterpret_cast<const float4*>(J.prim) + 2 * k;
            const float4 p0 = src[0], p1 = src[1];
            o = mk(J.view_p[0], J.view_p[1], J.view_p[2]);
            d = mk(p0.x, p0.y, p0.z);
            ray = __float_as_int(p0.w);
            tri = __float_as_int(p1.x);
            t = p1.y;
            strength = mk(1.f, 1.f, 1.f);
            rad = mk(0.f, 0.f, 0.f);
          }
        }
      }
      HPT_DCHECK(&c->err, !ok || (slot >= 0 && slot < P.num_slots), 212, slot, ok = false);
      HPT_DCHECK(&c->err, !ok || (tri >= 0 && tri < P.jobs[slot].scene.num_triangles), 214, tri,
                 ok = false);
      HPT_DCHECK(&c->err, !ok || (ray >= 0 && ray < job_rays(P.jobs[slot])), 215, ray, ok = false);
      if (ok) {
        const DevJob& J = P.jobs[slot];
        const DevScene& sc = kUniform ? P.uscene : J.scene;
        // The frame's sample index keys the random stream, so a render of
        // samples [first_sample, first_sample + spp) traces the same paths
        // as those samples of one whole-frame render.
        uint64_t seed = path_seed(J.seed, (uint32_t)ray, (uint32_t)(J.first_sample + sample),
                                  (uint32_t)bounce);
        const Ray r{o, d};
        const ShadeOut so = shade_hit(sc, r, strength, tri, t, J.disable_diffuse, seed,
                                      &c->err);
        ++shades;
        rad = add(rad, so.contrib);
        if (so.branch != kDead && bounce + 1 < J.depth) {
          const NextOut no = next_direction(sc, so.branch, d, so.hit_p, so.normal,
                                            so.strength, so.param, seed, &c->err);
          if (no.alive) {
            alive = true;
            oo = make_float4(no.o.x, no.o.y, no.o.z, __int_as_float((int)ray));
            dd = make_float4(no.d.x, no.d.y, no.d.z,
                             __uint_as_float(((uint32_t)sample << 8) | (uint32_t)(bounce + 1)));
            ss = make_float4(no.strength.x, no.strength.y, no.strength.z, __int_as_float(slot));
            rr = make_float4(rad.x, rad.y, rad.z, 0.f);
          }
        }
        if (!alive) {
          flush_radiance(J, ray, rad);
          ended = true;
        }
      }
    }
    count_paths(P.slots, tally, ended, alive, slot);
    // Block-level stable compaction: ballot per warp, scan over warps.
    const unsigned m = __ballot_sync(kFull, alive);
    if (lane == 0) warp_counts[warp] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
      int sum = 0;
      for (int w = 0; w < BS / 32; ++w) {
        const int v = warp_counts[w];
        warp_counts[w] = sum;
        sum += v;
      }
      block_base = sum ? atomicAdd(&c->nR, sum) : 0;
    }
    __syncthreads();
    if (alive) {
      const int pos = block_base + warp_counts[warp] + __popc(m & lanemask_lt());
      bool ok = true;
      HPT_DCHECK(&c->err, pos < P.capacity, 216, pos, ok = false);
      if (ok) {
        P.Q_o[par ^ 1][pos] = oo;
        P.Q_d[par ^ 1][pos] = dd;
        P.Q_s[par ^ 1][pos] = ss;
        P.Q_r[par ^ 1][pos] = rr;
      }
    }
    __syncthreads();
  }
  flush_tally(P.slots, tally);
  for (int o = 16; o > 0; o >>= 1) shades += __shfl_down_sync(kFull, shades, o);
  if (lane == 0 && shades) atomicAdd(&c->shades, shades);
#ifdef HPT_DEVICE_CHECKS
  for (int o = 16; o > 0; o >>= 1) chk_items += __shfl_down_sync(kFull, chk_items, o);
  if (lane == 0 && chk_items) atomicAdd(&c->chk_shade_done, chk_items);
#endif
}

// Register budgets of the closest-hit kernels: (threads per block, blocks per
// SM the compiler must fit); more resident warps against spills. Chosen by
// the tuning.
struct IsectVariant {
  int block, min_blocks;
  // [uniform scene]: queue rays, camera rays, both in one launch.
  void (*isect[2])(EngineParams);
  void (*primary[2])(EngineParams);
  void (*both[2])(EngineParams);
};
#define HPT_ISECT_VARIANT(B, M)                                                   \
  {B, M, {k_trace<B, M, false, true, false>, k_trace<B, M, true, true, false>},   \
   {k_trace<B, M, false, false, true>, k_trace<B, M, true, false, true>},         \
   {k_trace<B, M, false, true, true>, k_trace<B, M, true, true, true>}}
const IsectVariant kIsectVariants[] = {
    HPT_ISECT_VARIANT(128, 6), HPT_ISECT_VARIANT(128, 7), HPT_ISECT_VARIANT(128, 8),
    HPT_ISECT_VARIANT(128, 9), HPT_ISECT_VARIANT(128, 10),
    HPT_ISECT_VARIANT(256, 3), HPT_ISECT_VARIANT(256, 4),
};
#undef HPT_ISECT_VARIANT
constexpr int kNumIsectVariants = sizeof(kIsectVariants) / sizeof(kIsectVariants[0]);

// The shading kernel for a tuning's register budget (shade_min_blocks 3 or
// 4 blocks of 256 per SM; anything else: the natural allocation).
void (*shade_kernel(const hpt_tuning& t, bool uniform))(EngineParams) {
  if (t.shade_min_blocks == 3) return uniform ? k_shade<256, 3, true> : k_shade<256, 3, false>;
  if (t.shade_min_blocks == 4) return uniform ? k_shade<256, 4, true> : k_shade<256, 4, false>;
  return uniform ? k_shade<256, 1, true> : k_shade<256, 1, false>;
}

__device__ __forceinline__ float ray_value(const unsigned long long* acc, const uint32_t* flags,
                                           int64_t ray, int ch) {
  const uint32_t f = (flags[ray] >> (4 * ch)) & 0xF;
  if (f & 1u) return __int_as_float(0x7fc00000);
  if ((f & 6u) == 6u) return __int_as_float(0x7fc00000);
  if (f & 2u) return __int_as_float(0x7f800000);
  if (f & 4u) return __int_as_float(0xff800000);
  const long long v = (long long)acc[3 * ray + ch];
  return __double2float_rn(__ll2double_rn(v) * (1.0 / kAccumScale));
}

// write_imagef to an RGBA UNORM_INT8 image: convert_uchar_sat_rte(x * 255).
__device__ __forceinline__ uint8_t to_unorm8(float x) {
  const float v = __fmul_rn(x, 255.0f);
  if (!(v >= 0.f)) return 0;
  if (v >= 255.f) return 255;
  return (uint8_t)__float2int_rn(v);
}

// get_image (kernel.cl:615-652) from the fixed-point accumulators.
// samples is the divisor: the full sample count for the final image, or the
// samples completed so far for a progressive preview.
__global__ void k_resolve(const DevJob* jp, int W, int H, int ssx, int ssy, float samples,
                          float brightness, uint8_t* rgba, float* accum_f) {
  const int gx = blockIdx.x * blockDim.x + threadIdx.x;
  const int gy = blockIdx.y * blockDim.y + threadIdx.y;
  if (gx >= W || gy >= H) return;
  const DevJob& J = *jp;
  float px = 0.f, py = 0.f, pz = 0.f;
  for (int i = 0; i < ssx; ++i)
    for (int j = 0; j < ssy; ++j) {
      const int row = gy * ssy + j, col = gx * ssx + i;
      const int64_t idx = (int64_t)row * W * ssx + col;
      const float vx = ray_value(J.accum, J.flags, idx, 0);
      const float vy = ray_value(J.accum, J.flags, idx, 1);
      const float vz = ray_value(J.accum, J.flags, idx, 2);
      if (accum_f) {
        accum_f[3 * idx] = vx;
        accum_f[3 * idx + 1] = vy;
        accum_f[3 * idx + 2] = vz;
      }
      px = __fadd_rn(px, vx);
      py = __fadd_rn(py, vy);
      pz = __fadd_rn(pz, vz);
    }
  const float nss = (float)(ssx * ssy), ns = samples;
  px = __fmul_rn(__fdiv_rn(__fdiv_rn(px, nss), ns), brightness);
  py = __fmul_rn(__fdiv_rn(__fdiv_rn(py, nss), ns), brightness);
  pz = __fmul_rn(__fdiv_rn(__fdiv_rn(pz, nss), ns), brightness);
  uint8_t* o = rgba + 4 * ((int64_t)gy * W + gx);
  o[0] = to_unorm8(__fsub_rn(1.f, expf(-px)));
  o[1] = to_unorm8(__fsub_rn(1.f, expf(-py)));
  o[2] = to_unorm8(__fsub_rn(1.f, expf(-pz)));
  o[3] = 0;
}

}  // namespace

// ===========================================================================
// Host side
// ===========================================================================

hpt_status cuda_fail(cudaError_t e, const char* what) {
  return fail(e == cudaErrorMemoryAllocation ? HPT_ERR_OUT_OF_MEMORY : HPT_ERR_CUDA, "%s: %s",
              what, cudaGetErrorString(e));
}

void cuda_soft_fail(cudaError_t e, const char* what) {
  (void)cudaGetLastError();
#ifdef HPT_DEVICE_CHECKS
  fprintf(stderr, "hpt: best-effort call failed: %s: %s\n", what, cudaGetErrorString(e));
#else
  (void)e;
  (void)what;
#endif
}

hpt_tuning default_tuning() {
  hpt_tuning t;
  memset(&t, 0, sizeof t);
  // From one sweep on the 512x512, 64 spp spheres frame, the 1920x1080, 4 spp
  // terrain frame and the 256x256, 16 spp box room (device time): 8 blocks of
  // 128 per SM (64 registers; 6 / 7 / 8 / 9 blocks: spheres 40.1 / 37.8 / 36.8 /
  // 40.2 ms, terrain 14.3 / 13.7 / 13.9 / 14.7 ms, room 0.88 / 0.86 / 0.87 /
  // 0.90 ms), 16 rounds between refills (8 / 16 / 24 / 32: spheres 36.9 / 36.8 /
  // 37.8 / 39.5 ms, terrain 14.0 / 13.9 / 13.7 / 13.9 ms), a wavefront of 2^24
  // paths (2.7 GB of queues, allocated only up to the paths a run has).
  t.capacity = 1 << 24;
  t.isect_block = 128;
  t.isect_min_blocks = 8;
  t.shade_block = 256;
  t.refill_chunk = 4;
  t.smem_nodes = 0;
  t.use_graph = 0;
  t.trav_steps = 16;
  // Shading at 4 blocks of 256 per SM (64 registers, the settling calls' spills
  // included): 6.4 ms of a spheres frame, 7.2 at 3 blocks, 14.2 at the natural
  // allocation.
  t.shade_min_blocks = 4;
  return t;
}

// The scene as a job sees it: the tuning's step cap, when set, replaces the
// scene's own (only ever lowering it).
DevScene capped_scene(const DevScene& s, const hpt_tuning& t) {
  DevScene out = s;
  if (t.max_steps > 0) out.max_steps = std::min(out.max_steps, t.max_steps);
  return out;
}

hpt_status check_render_params(const hpt_camera* cam, const hpt_render_params* p) {
  if (!cam || !p) return fail(HPT_ERR_INVALID_ARGUMENT, "camera/params is NULL");
  if (p->sample_x <= 0 || p->sample_y <= 0 || p->supersample_x <= 0 || p->supersample_y <= 0 ||
      p->sample <= 0 || p->depth <= 0)
    return fail(HPT_ERR_INVALID_ARGUMENT, "sizes, sample and depth must be positive");
  const int64_t rays = (int64_t)p->sample_x * p->supersample_x * p->sample_y * p->supersample_y;
  if (rays > (1ll << 30)) return fail(HPT_ERR_INVALID_ARGUMENT, "too many rays per frame");
  if (p->sample >= (1 << 24)) return fail(HPT_ERR_INVALID_ARGUMENT, "sample must be < 2^24");
  if (p->first_sample < 0 || p->first_sample > INT32_MAX - p->sample)
    return fail(HPT_ERR_INVALID_ARGUMENT, "first_sample must be >= 0 and first_sample + sample < 2^31");
  if (p->depth > 255) return fail(HPT_ERR_INVALID_ARGUMENT, "depth must be <= 255");
  if (cam->height < 0 && p->supersample_x != p->supersample_y)
    return fail(HPT_ERR_INVALID_ARGUMENT,
                "panorama needs supersample_x == supersample_y (the reference indexes rays with "
                "sample_x * supersample_y)");
  return HPT_OK;
}

int64_t job_footprint(const hpt_render_params& p, bool want_accum) {
  const int64_t rays = (int64_t)p.sample_x * p.supersample_x * p.sample_y * p.supersample_y;
  return rays * (24 + 4 + 32 + (want_accum ? 12 : 0)) + (int64_t)p.sample_x * p.sample_y * 4 + 64;
}

Engine::Engine(int dev) : device(dev) {
  tuning = default_tuning();
  for (auto& e : ev_) e = nullptr;
  init_status_ = init();
}

// Device resources every run needs; a failure is reported by run().
hpt_status Engine::init() {
  HPT_CUDA(cudaSetDevice(device));
  HPT_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  HPT_CUDA(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, device));
  HPT_CUDA(cudaMalloc(&ctrl_, sizeof(DevCtrl)));
  HPT_CUDA(cudaMallocHost(&ctrl_host_, sizeof(DevCtrl)));
  for (auto& e : ev_) HPT_CUDA(cudaEventCreate(&e));
  for (auto& e : ev_done_) HPT_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  HPT_CUDA(cudaMallocHost(&done_host_, 2 * sizeof(int32_t)));
  // Per-job buffers come from the engine's own stream-ordered pool, which
  // keeps up to 4 GiB of freed memory mapped between renders instead of
  // returning it to the driver at every synchronisation.
  cudaMemPoolProps props;
  memset(&props, 0, sizeof props);
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = device;
  HPT_CUDA(cudaMemPoolCreate(&pool_, &props));
  uint64_t keep = 4ull << 30;
  HPT_CUDA(cudaMemPoolSetAttribute(pool_, cudaMemPoolAttrReleaseThreshold, &keep));
  return HPT_OK;
}

Engine::~Engine() {
  HPT_SOFT(cudaSetDevice(device));
  if (stream) HPT_SOFT(cudaStreamSynchronize(stream));
  free_queues();
  HPT_SOFT(cudaFree(ctrl_));
  HPT_SOFT(cudaFree(jobs_));
  HPT_SOFT(cudaFree(slot_state_));
  HPT_SOFT(cudaFree(order_));
  HPT_SOFT(cudaFree(quota_slot_));
  HPT_SOFT(cudaFree(quota_prefix_));
  HPT_SOFT(cudaFree(prim_slot_));
  HPT_SOFT(cudaFree(prim_prefix_));
  HPT_SOFT(cudaFree(prim_first_));
  HPT_SOFT(cudaFree(prim_final_));
  HPT_SOFT(cudaFreeHost(ctrl_host_));
  HPT_SOFT(cudaFreeHost(host_i32_));
  HPT_SOFT(cudaFreeHost(host_i64_));
  HPT_SOFT(cudaFreeHost(host_jobs_));
  HPT_SOFT(cudaFreeHost(slots_host_));
  for (auto& e : ev_)
    if (e) HPT_SOFT(cudaEventDestroy(e));
  for (auto& e : ev_done_)
    if (e) HPT_SOFT(cudaEventDestroy(e));
  for (auto& e : pev_) HPT_SOFT(cudaEventDestroy(e));
  if (done_host_) HPT_SOFT(cudaFreeHost(done_host_));
  if (pool_) HPT_SOFT(cudaMemPoolDestroy(pool_));
  if (graph_exec_) HPT_SOFT(cudaGraphExecDestroy(graph_exec_));
  for (StagingSet& st : staging_) {
    HPT_SOFT(cudaFreeHost(st.jobs));
    HPT_SOFT(cudaFreeHost(st.i32));
    HPT_SOFT(cudaFreeHost(st.i64));
    if (st.ev) HPT_SOFT(cudaEventDestroy(st.ev));
  }
  if (stream) HPT_SOFT(cudaStreamDestroy(stream));
}

void Engine::free_queues() {
  for (int p = 0; p < 2; ++p) {
    HPT_SOFT(cudaFree(Q_o_[p]));
    HPT_SOFT(cudaFree(Q_d_[p]));
    HPT_SOFT(cudaFree(Q_s_[p]));
    HPT_SOFT(cudaFree(Q_r_[p]));
    Q_o_[p] = Q_d_[p] = Q_s_[p] = Q_r_[p] = nullptr;
  }
  HPT_SOFT(cudaFree(hits_));
  HPT_SOFT(cudaFree(open_));
  hits_ = nullptr;
  open_ = nullptr;
  capacity_ = 0;
}

hpt_status Engine::ensure_capacity(int capacity) {
  if (capacity <= capacity_) return HPT_OK;
  HPT_SOFT(cudaStreamSynchronize(stream));
  free_queues();
  const size_t n = (size_t)capacity;
  for (int p = 0; p < 2; ++p) {
    HPT_CUDA(cudaMalloc(&Q_o_[p], n * sizeof(float4)));
    HPT_CUDA(cudaMalloc(&Q_d_[p], n * sizeof(float4)));
    HPT_CUDA(cudaMalloc(&Q_s_[p], n * sizeof(float4)));
    HPT_CUDA(cudaMalloc(&Q_r_[p], n * sizeof(float4)));
  }
  HPT_CUDA(cudaMalloc(&hits_, n * sizeof(uint4)));
  HPT_CUDA(cudaMalloc(&open_, n * sizeof(uint4)));
  capacity_ = capacity;
  return HPT_OK;
}

hpt_status Engine::ensure_slots(int slots) {
  if (slots <= slots_) return HPT_OK;
  HPT_SOFT(cudaStreamSynchronize(stream));
  HPT_SOFT(cudaFree(jobs_));
  HPT_SOFT(cudaFree(slot_state_));
  HPT_SOFT(cudaFree(order_));
  HPT_SOFT(cudaFree(quota_slot_));
  HPT_SOFT(cudaFree(quota_prefix_));
  HPT_SOFT(cudaFree(prim_slot_));
  HPT_SOFT(cudaFree(prim_prefix_));
  HPT_SOFT(cudaFree(prim_first_));
  HPT_SOFT(cudaFree(prim_final_));
  HPT_SOFT(cudaFreeHost(host_i32_));
  HPT_SOFT(cudaFreeHost(host_i64_));
  HPT_SOFT(cudaFreeHost(host_jobs_));
  HPT_SOFT(cudaFreeHost(slots_host_));
  slots_host_ = nullptr;
  jobs_ = nullptr;
  slot_state_ = nullptr;
  order_ = quota_slot_ = quota_prefix_ = prim_slot_ = prim_final_ = nullptr;
  prim_prefix_ = prim_first_ = nullptr;
  host_i32_ = nullptr;
  host_i64_ = nullptr;
  host_jobs_ = nullptr;
  slots_ = 0;
  const size_t n = (size_t)slots;
  HPT_CUDA(cudaMalloc(&jobs_, n * sizeof(DevJob)));
  HPT_CUDA(cudaMalloc(&slot_state_, n * sizeof(DevSlot)));
  HPT_CUDA(cudaMalloc(&order_, n * sizeof(int32_t)));
  HPT_CUDA(cudaMalloc(&quota_slot_, n * sizeof(int32_t)));
  HPT_CUDA(cudaMalloc(&quota_prefix_, (n + 1) * sizeof(int32_t)));
  HPT_CUDA(cudaMalloc(&prim_slot_, n * sizeof(int32_t)));
  HPT_CUDA(cudaMalloc(&prim_prefix_, (n + 1) * sizeof(int64_t)));
  HPT_CUDA(cudaMalloc(&prim_first_, n * sizeof(int64_t)));
  HPT_CUDA(cudaMalloc(&prim_final_, n * sizeof(int32_t)));
  HPT_CUDA(cudaMallocHost(&host_i32_, (2 * n + 3) * sizeof(int32_t)));
  HPT_CUDA(cudaMallocHost(&host_i64_, (n + 1) * sizeof(int64_t)));
  HPT_CUDA(cudaMallocHost(&host_jobs_, n * sizeof(DevJob)));
  HPT_CUDA(cudaMallocHost(&slots_host_, n * sizeof(DevSlot)));
  HPT_CUDA(cudaMemsetAsync(jobs_, 0, n * sizeof(DevJob), stream));
  HPT_CUDA(cudaMemsetAsync(slot_state_, 0, n * sizeof(DevSlot), stream));
  HPT_CUDA(cudaMemsetAsync(quota_prefix_, 0, (n + 1) * sizeof(int32_t), stream));
  HPT_CUDA(cudaMemsetAsync(prim_prefix_, 0, (n + 1) * sizeof(int64_t), stream));
  slots_ = slots;
  return HPT_OK;
}

// The compiled variant with the tuning's block size and blocks-per-SM
// budget; without an exact match, the first one with that block size.
int Engine::isect_variant() const {
  for (int i = 0; i < kNumIsectVariants; ++i)
    if (kIsectVariants[i].block == tuning.isect_block &&
        kIsectVariants[i].min_blocks == tuning.isect_min_blocks)
      return i;
  for (int i = 0; i < kNumIsectVariants; ++i)
    if (kIsectVariants[i].block == tuning.isect_block) return i;
  return 0;
}

hpt_status Engine::query_occupancy() {
  if (occ_done_) return HPT_OK;
  const IsectVariant& v = kIsectVariants[isect_variant()];
  int b = 0;
  HPT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &b, v.isect[1], v.block, 0));
  occ_isect_ = std::max(1, b);
  HPT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, shade_kernel(tuning, false), 256, 0));
  occ_shade_ = std::max(1, b);
  occ_done_ = true;
  return HPT_OK;
}

hpt_status Engine::alloc_job(const JobSpec& js, bool want_accum, JobBuffers& b) {
  const hpt_render_params& p = js.params;
  const int64_t nx = (int64_t)p.sample_x * p.supersample_x, ny = (int64_t)p.sample_y * p.supersample_y;
  b.rays = nx * ny;
  // One allocation and one clear: accumulators, flags and hit count first.
  size_t size = 0;
  auto part = [&](size_t bytes) {
    const size_t at = size;
    size += (bytes + 255) & ~(size_t)255;
    return at;
  };
  const size_t accum = part((size_t)b.rays * 3 * sizeof(unsigned long long));
  const size_t flags = part((size_t)b.rays * sizeof(uint32_t));
  const size_t count = part(sizeof(int32_t));
  const size_t cleared = size;
  const size_t prim = part((size_t)b.rays * 8 * sizeof(float));
  const size_t rgba = part((size_t)p.sample_x * p.sample_y * 4);
  const size_t accum_f = want_accum ? part((size_t)b.rays * 3 * sizeof(float)) : 0;
  void* mem = nullptr;
  HPT_CUDA(cudaMallocFromPoolAsync(&mem, size, pool_, stream));
  b.base = static_cast<uint8_t*>(mem);
  b.accum = reinterpret_cast<unsigned long long*>(b.base + accum);
  b.flags = reinterpret_cast<uint32_t*>(b.base + flags);
  b.prim_count = reinterpret_cast<int32_t*>(b.base + count);
  b.prim = reinterpret_cast<float*>(b.base + prim);
  b.rgba = b.base + rgba;
  if (want_accum) b.accum_f = reinterpret_cast<float*>(b.base + accum_f);
  HPT_CUDA(cudaMemsetAsync(b.base, 0, cleared, stream));
  b.bytes = job_footprint(p, want_accum);
  return HPT_OK;
}

void Engine::free_job(JobBuffers& b) {
  if (b.base) HPT_SOFT(cudaFreeAsync(b.base, stream));
  b = JobBuffers();
}

DevJob Engine::make_job(const JobSpec& js, const JobBuffers& b) const {
  DevJob j;
  memset(&j, 0, sizeof j);
  const hpt_camera& cam = js.camera;
  const hpt_render_params& p = js.params;
  j.scene = capped_scene(js.scene->dev, tuning);
  for (int k = 0; k < 3; ++k) {
    j.view_p[k] = cam.view_p[k];
    j.top[k] = cam.top_dir[k];
    j.right[k] = cam.right_dir[k];
    j.bg[k] = p.background[k];
  }
  j.width = cam.width;
  j.height = cam.height;
  j.nx = p.sample_x * p.supersample_x;
  j.ny = p.sample_y * p.supersample_y;
  j.pano = cam.height < 0 ? 1 : 0;
  // trace_runner.cpp:131-140: shift = int(right_dir.x), times supersample_x.
  j.vr_x_shift = (int)cam.right_dir[0] * p.supersample_x;
  j.spp = p.sample;
  j.depth = p.depth;
  j.disable_diffuse = p.disable_diffuse;
  j.first_sample = p.first_sample;
  j.seed = p.seed;
  j.accum = b.accum;
  j.flags = b.flags;
  j.prim = b.prim;
  j.prim_count = b.prim_count;
  return j;
}

static EngineParams make_params(const Engine& e, DevCtrl* ctrl, DevJob* jobs, DevSlot* slots,
                                int num_slots, const int32_t* order, int32_t* quota_slot,
                                int32_t* quota_prefix, const int32_t* prim_slot,
                                const int64_t* prim_prefix, int prim_n, int capacity,
                                float4* const* Q, uint4* hits, uint4* open,
                                const DevScene* shared) {
  EngineParams P;
  memset(&P, 0, sizeof P);
  P.jobs = jobs;
  P.slots = slots;
  P.num_slots = num_slots;
  P.ctrl = ctrl;
  P.order = order;
  P.quota_slot = quota_slot;
  P.quota_prefix = quota_prefix;
  P.prim_slot = prim_slot;
  P.prim_prefix = prim_prefix;
  P.prim_n = prim_n;
  for (int p = 0; p < 2; ++p) {
    P.Q_o[p] = Q[4 * p + 0];
    P.Q_d[p] = Q[4 * p + 1];
    P.Q_s[p] = Q[4 * p + 2];
    P.Q_r[p] = Q[4 * p + 3];
  }
  P.hits = hits;
  P.open = open;
  P.capacity = capacity;
  P.refill = std::max(1, std::min(32, e.tuning.refill_chunk));
  P.rounds = e.tuning.trav_steps > 0 ? e.tuning.trav_steps : default_tuning().trav_steps;
  if (shared) {
    P.uniform_scene = 1;
    P.uscene = capped_scene(*shared, e.tuning);
  }
  return P;
}

void Engine::reset_ctrl() {
  HPT_SOFT(cudaMemsetAsync(ctrl_, 0, sizeof(DevCtrl), stream));
  if (slots_ > 0) HPT_SOFT(cudaMemsetAsync(slot_state_, 0, (size_t)slots_ * sizeof(DevSlot), stream));
}

// The run's uploads go through pinned staging that is free again when run()
// has synchronised: [0, slots] prim_slot, [slots + 1, 2 slots + 1] order,
// [2 slots + 2] n_order.
hpt_status Engine::admit(const std::vector<int>& slot_ids, const std::vector<DevJob>& jobs,
                         const std::vector<int64_t>& rays, const std::vector<int>& order,
                         const DevScene* shared_scene) {
  const int n = (int)slot_ids.size();
  {
    hpt_status qs = query_occupancy();
    if (qs != HPT_OK) return qs;
  }
  if ((int)order.size() > slots_) return fail(HPT_ERR_INVALID_ARGUMENT, "order larger than slots");
  int32_t* stage = host_i32_ + (slots_ + 1);
  for (size_t k = 0; k < order.size(); ++k) stage[k] = order[k];
  if (!order.empty())
    HPT_CUDA(cudaMemcpyAsync(order_, stage, order.size() * sizeof(int32_t),
                             cudaMemcpyHostToDevice, stream));
  stage[slots_ + 1] = (int32_t)order.size();
  HPT_CUDA(cudaMemcpyAsync(&ctrl_->n_order, &stage[slots_ + 1], sizeof(int32_t),
                           cudaMemcpyHostToDevice, stream));
  for (int k = 0; k < n; ++k) {
    if (slot_ids[k] < 0 || slot_ids[k] >= slots_)
      return fail(HPT_ERR_INVALID_ARGUMENT, "slot %d out of range", slot_ids[k]);
    host_jobs_[slot_ids[k]] = jobs[k];
    HPT_CUDA(cudaMemcpyAsync(jobs_ + slot_ids[k], host_jobs_ + slot_ids[k], sizeof(DevJob),
                             cudaMemcpyHostToDevice, stream));
  }
  host_i64_[0] = 0;
  for (int k = 0; k < n; ++k) {
    host_i32_[k] = slot_ids[k];
    host_i64_[k + 1] = host_i64_[k] + rays[k];
  }
  HPT_CUDA(cudaMemcpyAsync(prim_slot_, host_i32_, n * sizeof(int32_t), cudaMemcpyHostToDevice,
                           stream));
  HPT_CUDA(cudaMemcpyAsync(prim_prefix_, host_i64_, (n + 1) * sizeof(int64_t),
                           cudaMemcpyHostToDevice, stream));
  float4* Q[8] = {Q_o_[0], Q_d_[0], Q_s_[0], Q_r_[0], Q_o_[1], Q_d_[1], Q_s_[1], Q_r_[1]};
  EngineParams P = make_params(*this, ctrl_, jobs_, slot_state_, slots_, order_, quota_slot_,
                               quota_prefix_, prim_slot_, prim_prefix_, n, capacity_, Q, hits_,
                               open_, shared_scene);
  const IsectVariant& v = kIsectVariants[isect_variant()];
  v.primary[P.uniform_scene]<<<trace_grid(host_i64_[n]), v.block, 0, stream>>>(P);
  HPT_CUDA(cudaGetLastError());
  return HPT_OK;
}

// Blocks of a launch over at most `items` rays: all that fit, or for few rays
// one per warp's worth, so that they spread over the SMs.
int Engine::trace_grid(int64_t items) const {
  return (int)std::max<int64_t>(1, std::min<int64_t>(num_sms * occ_isect_, (items + 31) / 32));
}

// --- Asynchronous uploads (serving loop) ------------------------------------
hpt_status Engine::next_staging(StagingSet** out) {
  if (staging_slots_ != slots_) {
    for (StagingSet& st : staging_) {
      if (st.ev) HPT_CUDA(cudaEventSynchronize(st.ev));
      HPT_SOFT(cudaFreeHost(st.jobs));
      HPT_SOFT(cudaFreeHost(st.i32));
      HPT_SOFT(cudaFreeHost(st.i64));
      st.jobs = nullptr;
      st.i32 = nullptr;
      st.i64 = nullptr;
    }
    staging_slots_ = 0;
    const size_t n = (size_t)slots_;
    for (StagingSet& st : staging_) {
      HPT_CUDA(cudaMallocHost(&st.jobs, n * sizeof(DevJob)));
      HPT_CUDA(cudaMallocHost(&st.i32, (3 * n + 3) * sizeof(int32_t)));
      HPT_CUDA(cudaMallocHost(&st.i64, (2 * n + 1) * sizeof(int64_t)));
      if (!st.ev) HPT_CUDA(cudaEventCreateWithFlags(&st.ev, cudaEventDisableTiming));
    }
    staging_slots_ = slots_;
  }
  StagingSet& st = staging_[staging_next_];
  staging_next_ = (staging_next_ + 1) % kStagingRing;
  // The set's previous copies were enqueued kStagingRing uploads ago; wait
  // until they have run before overwriting their source.
  HPT_CUDA(cudaEventSynchronize(st.ev));
  *out = &st;
  return HPT_OK;
}

hpt_status Engine::upload_order(const std::vector<int>& order, StagingSet& st) {
  if ((int)order.size() > slots_) return fail(HPT_ERR_INVALID_ARGUMENT, "order larger than slots");
  int32_t* stage = st.i32 + (slots_ + 1);
  for (size_t k = 0; k < order.size(); ++k) stage[k] = order[k];
  if (!order.empty())
    HPT_CUDA(cudaMemcpyAsync(order_, stage, order.size() * sizeof(int32_t),
                             cudaMemcpyHostToDevice, stream));
  stage[slots_ + 1] = (int32_t)order.size();
  HPT_CUDA(cudaMemcpyAsync(&ctrl_->n_order, &stage[slots_ + 1], sizeof(int32_t),
                           cudaMemcpyHostToDevice, stream));
  return HPT_OK;
}

hpt_status Engine::set_order_async(const std::vector<int>& order) {
  StagingSet* st = nullptr;
  hpt_status s = next_staging(&st);
  if (s != HPT_OK) return s;
  s = upload_order(order, *st);
  if (s != HPT_OK) return s;
  HPT_CUDA(cudaEventRecord(st->ev, stream));
  return HPT_OK;
}

// Uploads n primary-pass entries through a staging set: each entry's job
// into its slot, then the slot list, the ray-count prefix and, with
// `first` / `fin`, the first rays and final flags.
hpt_status Engine::stage_primary(StagingSet& st, int n, const int* slot_ids, const DevJob* jobs,
                                 const int64_t* rays, const int64_t* first, const int* fin) {
  if (n > slots_)
    return fail(HPT_ERR_INVALID_ARGUMENT, "%d primary entries for %d slots", n, slots_);
  for (int k = 0; k < n; ++k) {
    if (slot_ids[k] < 0 || slot_ids[k] >= slots_)
      return fail(HPT_ERR_INVALID_ARGUMENT, "slot %d out of range", slot_ids[k]);
    st.jobs[k] = jobs[k];
    HPT_CUDA(cudaMemcpyAsync(jobs_ + slot_ids[k], st.jobs + k, sizeof(DevJob),
                             cudaMemcpyHostToDevice, stream));
  }
  st.i64[0] = 0;
  // Staging layout: i32 [0, n) slots, [slots + 1, 2 slots + 2] order (see
  // upload_order), [2 slots + 3, + n) final flags; i64 [0, n] prefix,
  // [slots + 1, + n) first rays.
  int32_t* sfin = st.i32 + 2 * slots_ + 3;
  int64_t* sfst = st.i64 + slots_ + 1;
  for (int k = 0; k < n; ++k) {
    st.i32[k] = slot_ids[k];
    st.i64[k + 1] = st.i64[k] + rays[k];
    if (first) {
      sfst[k] = first[k];
      sfin[k] = fin[k];
    }
  }
  HPT_CUDA(cudaMemcpyAsync(prim_slot_, st.i32, n * sizeof(int32_t), cudaMemcpyHostToDevice,
                           stream));
  HPT_CUDA(cudaMemcpyAsync(prim_prefix_, st.i64, (n + 1) * sizeof(int64_t),
                           cudaMemcpyHostToDevice, stream));
  if (first) {
    HPT_CUDA(cudaMemcpyAsync(prim_first_, sfst, n * sizeof(int64_t), cudaMemcpyHostToDevice,
                             stream));
    HPT_CUDA(cudaMemcpyAsync(prim_final_, sfin, n * sizeof(int32_t), cudaMemcpyHostToDevice,
                             stream));
  }
  return HPT_OK;
}

hpt_status Engine::queue_primary(int slot, const DevJob& job, int64_t rays, int64_t first,
                                 bool final_part) {
  if (slot < 0 || slot >= slots_ || rays <= 0 || first < 0)
    return fail(HPT_ERR_INVALID_ARGUMENT, "primary entry: slot %d, %lld rays from %lld", slot,
                (long long)rays, (long long)first);
  for (size_t k = 0; k < pend_slot_.size(); ++k) {
    if (pend_slot_[k] != slot) continue;
    // A later part of the same job, queued before an iteration carried the
    // earlier one: extend that entry.
    if (pend_final_[k] || first != pend_first_[k] + pend_rays_[k])
      return fail(HPT_ERR_INVALID_ARGUMENT, "primary parts of slot %d out of order", slot);
    pend_rays_[k] += rays;
    pend_final_[k] = final_part ? 1 : 0;
    pend_job_[k] = job;
    return HPT_OK;
  }
  pend_slot_.push_back(slot);
  pend_job_.push_back(job);
  pend_rays_.push_back(rays);
  pend_first_.push_back(first);
  pend_final_.push_back(final_part ? 1 : 0);
  return HPT_OK;
}

hpt_status Engine::launch_iteration_async() {
  const int n = (int)pend_slot_.size();
  if (n == 0) {
    launch_iteration(nullptr, nullptr, capacity_, false);
    return HPT_OK;
  }
  hpt_status s = query_occupancy();
  if (s != HPT_OK) return s;
  StagingSet* st = nullptr;
  s = next_staging(&st);
  if (s != HPT_OK) return s;
  s = stage_primary(*st, n, pend_slot_.data(), pend_job_.data(), pend_rays_.data(),
                    pend_first_.data(), pend_final_.data());
  if (s != HPT_OK) return s;
  HPT_CUDA(cudaEventRecord(st->ev, stream));
  pend_slot_.clear();
  pend_job_.clear();
  pend_rays_.clear();
  pend_first_.clear();
  pend_final_.clear();
  float4* Q[8] = {Q_o_[0], Q_d_[0], Q_s_[0], Q_r_[0], Q_o_[1], Q_d_[1], Q_s_[1], Q_r_[1]};
  EngineParams P = make_params(*this, ctrl_, jobs_, slot_state_, slots_, order_, quota_slot_,
                               quota_prefix_, prim_slot_, prim_prefix_, n, capacity_, Q, hits_,
                               open_, nullptr);
  P.prim_first = prim_first_;
  P.prim_final = prim_final_;
  shade_kernel(tuning, P.uniform_scene)<<<num_sms * occ_shade_, 256, 0, stream>>>(P);
  const IsectVariant& v = kIsectVariants[isect_variant()];
  v.both[0]<<<num_sms * occ_isect_, v.block, 0, stream>>>(P);
  HPT_CUDA(cudaGetLastError());
  return HPT_OK;
}

hpt_status Engine::read_state_async(DevSlot* slots, DevCtrl* ctrl, cudaEvent_t ev) {
  if (slots_ > 0)
    HPT_CUDA(cudaMemcpyAsync(slots, slot_state_, (size_t)slots_ * sizeof(DevSlot),
                             cudaMemcpyDeviceToHost, stream));
  HPT_CUDA(cudaMemcpyAsync(ctrl, ctrl_, sizeof(DevCtrl), cudaMemcpyDeviceToHost, stream));
  HPT_CUDA(cudaEventRecord(ev, stream));
  return HPT_OK;
}

hpt_status Engine::ensure_graph(const DevScene* shared_scene, int iterations) {
  // The key covers the whole shared scene, not just its node array: a scene
  // freed and replaced by one whose nodes land at the same address must not
  // reuse a graph that holds the old scene's other pointers.
  const bool shared = shared_scene != nullptr;
  const bool same_scene =
      graph_shared_ == shared &&
      (!shared || memcmp(&graph_scene_, shared_scene, sizeof(DevScene)) == 0);
  if (graph_exec_ && same_scene && graph_capacity_ == capacity_ &&
      graph_slots_ == slots_ && graph_iters_ == iterations && graph_tuning_ == isect_variant() &&
      graph_refill_ == tuning.refill_chunk &&
      graph_steps_ == tuning.trav_steps && graph_max_steps_ == tuning.max_steps &&
      graph_shade_ == tuning.shade_min_blocks)
    return HPT_OK;
  if (graph_exec_) {
    HPT_SOFT(cudaGraphExecDestroy(graph_exec_));
    graph_exec_ = nullptr;
  }
  cudaGraph_t g = nullptr;
  HPT_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
  for (int k = 0; k < iterations; ++k)
    launch_iteration(shared_scene, nullptr, capacity_, false);
  const cudaError_t launch = cudaGetLastError();
  const cudaError_t end = cudaStreamEndCapture(stream, &g);
  if (launch != cudaSuccess) {
    if (g) HPT_SOFT(cudaGraphDestroy(g));
    return cuda_fail(launch, "graph capture");
  }
  HPT_CUDA(end);
  const cudaError_t inst = cudaGraphInstantiate(&graph_exec_, g, 0);
  HPT_SOFT(cudaGraphDestroy(g));
  HPT_CUDA(inst);
  graph_shared_ = shared;
  if (shared) graph_scene_ = *shared_scene;
  graph_capacity_ = capacity_;
  graph_slots_ = slots_;
  graph_iters_ = iterations;
  graph_tuning_ = isect_variant();
  graph_refill_ = tuning.refill_chunk;
  graph_steps_ = tuning.trav_steps;
  graph_max_steps_ = tuning.max_steps;
  graph_shade_ = tuning.shade_min_blocks;
  return HPT_OK;
}

void Engine::launch_iteration(const DevScene* shared_scene, cudaEvent_t* ev, int64_t paths,
                              bool last) {
  float4* Q[8] = {Q_o_[0], Q_d_[0], Q_s_[0], Q_r_[0], Q_o_[1], Q_d_[1], Q_s_[1], Q_r_[1]};
  EngineParams P = make_params(*this, ctrl_, jobs_, slot_state_, slots_, order_, quota_slot_,
                               quota_prefix_, prim_slot_, prim_prefix_, 0, capacity_, Q, hits_,
                               open_, shared_scene);
  if (ev) HPT_SOFT(cudaEventRecord(ev[0], stream));
  const int64_t shade_blocks = std::min<int64_t>(num_sms * occ_shade_, (paths + 255) / 256);
  shade_kernel(tuning, P.uniform_scene)<<<(int)std::max<int64_t>(1, shade_blocks), 256, 0, stream>>>(P);
  if (ev) HPT_SOFT(cudaEventRecord(ev[1], stream));
  const IsectVariant& v = kIsectVariants[isect_variant()];
  if (last) k_ctrl<<<1, 1, 0, stream>>>(P);
  else v.isect[P.uniform_scene]<<<trace_grid(paths), v.block, 0, stream>>>(P);
  if (ev) HPT_SOFT(cudaEventRecord(ev[2], stream));
}

void Engine::launch_resolve(int slot, const JobSpec& js, const JobBuffers& b, float samples) {
  const hpt_render_params& p = js.params;
  dim3 blk(16, 16), grd((p.sample_x + 15) / 16, (p.sample_y + 15) / 16);
  k_resolve<<<grd, blk, 0, stream>>>(jobs_ + slot, p.sample_x, p.sample_y, p.supersample_x,
                                      p.supersample_y, samples > 0.f ? samples : (float)p.sample,
                                      p.brightness, b.rgba, b.accum_f);
}

hpt_status Engine::reserve_pool(size_t bytes) {
  if (bytes == 0) return HPT_OK;
  uint64_t keep = 0;
  HPT_CUDA(cudaMemPoolGetAttribute(pool_, cudaMemPoolAttrReleaseThreshold, &keep));
  if (keep < bytes) {
    keep = bytes;
    HPT_CUDA(cudaMemPoolSetAttribute(pool_, cudaMemPoolAttrReleaseThreshold, &keep));
  }
  void* p = nullptr;
  HPT_CUDA(cudaMallocFromPoolAsync(&p, bytes, pool_, stream));
  HPT_CUDA(cudaFreeAsync(p, stream));
  HPT_CUDA(cudaStreamSynchronize(stream));
  return HPT_OK;
}

hpt_status Engine::set_capped_budget(int64_t paths) {
  ctrl_host_->capped_budget = paths;
  HPT_CUDA(cudaMemcpyAsync(&ctrl_->capped_budget, &ctrl_host_->capped_budget, sizeof(int64_t),
                           cudaMemcpyHostToDevice, stream));
  HPT_CUDA(cudaStreamSynchronize(stream));
  return HPT_OK;
}

hpt_status Engine::read_ctrl(DevCtrl* out) {
  HPT_CUDA(cudaMemcpyAsync(ctrl_host_, ctrl_, sizeof(DevCtrl), cudaMemcpyDeviceToHost, stream));
  HPT_CUDA(cudaStreamSynchronize(stream));
  *out = *ctrl_host_;
  return HPT_OK;
}

hpt_status Engine::run(const std::vector<JobSpec>& jobs, hpt_render_stats* stats) {
  if (init_status_ != HPT_OK) return fail(init_status_, "engine set-up failed");
  HPT_CUDA(cudaSetDevice(device));
  if (jobs.empty()) return HPT_OK;
  // The wavefront never holds more paths than the run has, so the queues
  // are sized to the smaller of the tuning's capacity and the run's paths
  // (results do not depend on the capacity: fixed-point sums, counter RNG).
  int64_t paths = 0;
  for (const JobSpec& js : jobs) {
    const hpt_render_params& p = js.params;
    paths += (int64_t)p.sample_x * p.supersample_x * p.sample_y * p.supersample_y * p.sample;
  }
  hpt_status s = ensure_capacity(
      (int)std::max<int64_t>(1024, std::min<int64_t>(tuning.capacity, paths)));
  if (s != HPT_OK) return s;
  s = ensure_slots((int)jobs.size());
  if (s != HPT_OK) return s;
  const int n = (int)jobs.size();
  std::vector<JobBuffers> bufs(n);
  std::vector<DevJob> djobs;
  std::vector<int> slot_ids(n);
  std::vector<int64_t> rays(n);
  const SceneDev* shared = jobs[0].scene;
  for (int j = 0; j < n; ++j) {
    s = alloc_job(jobs[j], jobs[j].accum_out != nullptr, bufs[j]);
    if (s != HPT_OK) {
      for (int k = 0; k <= j; ++k) free_job(bufs[k]);
      return s;
    }
    djobs.push_back(make_job(jobs[j], bufs[j]));
    slot_ids[j] = j;
    rays[j] = bufs[j].rays;
    if (jobs[j].scene != shared) shared = nullptr;
  }
  // Smallest jobs first.
  std::vector<int> order(n);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return rays[a] * jobs[a].params.sample < rays[b] * jobs[b].params.sample;
  });
  const DevScene* shared_dev = shared ? &shared->dev : nullptr;
  reset_ctrl();
  HPT_SOFT(cudaEventRecord(ev_[0], stream));
  s = admit(slot_ids, djobs, rays, order, shared_dev);
  if (s != HPT_OK) {
    for (auto& b : bufs) free_job(b);
    HPT_SOFT(cudaStreamSynchronize(stream));
    return s;
  }
  HPT_SOFT(cudaEventRecord(ev_[1], stream));
  // Iterate until the device says the wavefront is drained. Batches of
  // iterations are queued ahead; the done flag of batch k is checked while
  // batch k+1 runs (extra iterations after completion are empty launches).
  // When the queue holds every path of the run, all start in the first
  // iteration and each has ended after as many as its depth: no more than
  // those are launched, and beyond kAhead, where most paths have long ended
  // (depths go up to 255), batches as long as the flag is not set.
  const int kBatch = 4, kAhead = 16;
  const bool prof = tuning.profile != 0;
  const bool at_once = paths <= capacity_ && (tuning.use_graph == 0 || prof);
  int max_depth = 1;
  for (const JobSpec& js : jobs) max_depth = std::max(max_depth, js.params.depth);
  int32_t* done_host = done_host_;
  done_host[0] = done_host[1] = 0;
  cudaEvent_t* ev_done = ev_done_;
  std::vector<cudaEvent_t>& pev = pev_;
  if (prof)
    while ((int)pev.size() < 3 * std::max(2 * kBatch, at_once ? max_depth : 0)) {
      cudaEvent_t e = nullptr;
      HPT_CUDA(cudaEventCreate(&e));
      pev.push_back(e);
    }
  float ms_shade = 0.f, ms_isect = 0.f;
  auto harvest = [&](int first, int count) {
    for (int k = first; k < first + count; ++k) {
      float a = 0.f, b = 0.f;
      HPT_SOFT(cudaEventElapsedTime(&a, pev[3 * k], pev[3 * k + 1]));
      HPT_SOFT(cudaEventElapsedTime(&b, pev[3 * k + 1], pev[3 * k + 2]));
      ms_shade += a;
      ms_isect += b;
    }
  };
  // Upper bound on iterations: every live path advances one bounce per
  // iteration, so the wavefront drains within paths * depth / capacity
  // iterations plus one path lifetime; 2x that plus slack is the cap.
  int64_t work = 0;
  for (const JobSpec& js : jobs) {
    const hpt_render_params& p = js.params;
    work += (int64_t)p.sample_x * p.supersample_x * p.sample_y * p.supersample_y * p.sample *
            p.depth;
  }
  const int64_t max_batches = (2 * (work / std::max(1, capacity_) + max_depth) + 64) / kBatch + 4;
  // With use_graph, the kBatch iterations are replayed from one CUDA graph
  // (their parameters live in device memory, so one capture serves every
  // batch); it is captured again when the queues, the slot table or the
  // shared-scene prefix change. Profiling needs per-kernel events: eager.
  const bool use_graph = tuning.use_graph != 0 && !prof;
  if (use_graph) {
    s = ensure_graph(shared_dev, kBatch);
    if (s != HPT_OK) {
      for (auto& b : bufs) free_job(b);
      HPT_SOFT(cudaStreamSynchronize(stream));
      return s;
    }
  }
  int64_t guard = 0;
  bool drained = false;
  int slot = 0;
  bool pending = false;
  auto ask = [&](int k) {
    HPT_SOFT(cudaMemcpyAsync(&done_host[k], &ctrl_->done, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    HPT_SOFT(cudaEventRecord(ev_done[k], stream));
  };
  int launched = 0;  // at_once
  while (at_once && launched < max_depth && !drained) {
    const int upto = std::min(max_depth, launched == 0 ? kAhead : launched + kBatch);
    for (; launched < upto; ++launched)
      launch_iteration(shared_dev, prof ? &pev[3 * launched] : nullptr, paths,
                       launched == max_depth - 1);
    if (max_depth <= kAhead) break;
    ask(slot);
    if (pending) {
      HPT_SOFT(cudaEventSynchronize(ev_done[slot ^ 1]));
      drained = done_host[slot ^ 1] != 0;
    }
    pending = true;
    slot ^= 1;
  }
  while (!at_once) {
    if (use_graph) {
      const cudaError_t launch = cudaGraphLaunch(graph_exec_, stream);
      if (launch != cudaSuccess) {
        for (auto& b : bufs) free_job(b);
        HPT_SOFT(cudaStreamSynchronize(stream));
        return cuda_fail(launch, "graph launch");
      }
    } else {
      for (int k = 0; k < kBatch; ++k)
        launch_iteration(shared_dev, prof ? &pev[(slot * kBatch + k) * 3] : nullptr, capacity_,
                         false);
    }
    ask(slot);
    if (pending) {
      HPT_SOFT(cudaEventSynchronize(ev_done[slot ^ 1]));
      if (prof) harvest((slot ^ 1) * kBatch, kBatch);
      if (done_host[slot ^ 1]) {
        drained = true;
        break;
      }
    }
    pending = true;
    slot ^= 1;
    if (++guard > max_batches) break;
  }
  HPT_SOFT(cudaEventRecord(ev_[2], stream));
  for (int j = 0; j < n; ++j) launch_resolve(j, jobs[j], bufs[j]);
  HPT_SOFT(cudaEventRecord(ev_[3], stream));
  for (int j = 0; j < n; ++j) {
    const hpt_render_params& p = jobs[j].params;
    if (jobs[j].rgba_out)
      HPT_SOFT(cudaMemcpyAsync(jobs[j].rgba_out, bufs[j].rgba, (size_t)p.sample_x * p.sample_y * 4, cudaMemcpyDeviceToHost, stream));
    if (jobs[j].accum_out)
      HPT_SOFT(cudaMemcpyAsync(jobs[j].accum_out, bufs[j].accum_f, (size_t)bufs[j].rays * 3 * sizeof(float), cudaMemcpyDeviceToHost, stream));
  }
  HPT_SOFT(cudaMemcpyAsync(ctrl_host_, ctrl_, sizeof(DevCtrl), cudaMemcpyDeviceToHost, stream));
  HPT_SOFT(cudaMemcpyAsync(slots_host_, slot_state_, n * sizeof(DevSlot), cudaMemcpyDeviceToHost,
                           stream));
  for (auto& b : bufs) free_job(b);
  cudaError_t e = cudaStreamSynchronize(stream);
  if (prof) harvest(at_once ? 0 : slot * kBatch, at_once ? launched : kBatch);
  if (e != cudaSuccess) return cuda_fail(e, "render");
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "render launch");
  int64_t prim = 0;
  for (int64_t r : rays) prim += r;
  if (stats) {
    memset(stats, 0, sizeof *stats);
    stats->primary_rays = prim;
    stats->intersect_queries = (int64_t)ctrl_host_->isect_queries;
    stats->shade_calls = (int64_t)ctrl_host_->shades;
    stats->iterations = (int32_t)ctrl_host_->iterations;
    stats->error_flags = (int32_t)ctrl_host_->err.flags;
    HPT_SOFT(cudaEventElapsedTime(&stats->ms_total, ev_[0], ev_[3]));
    HPT_SOFT(cudaEventElapsedTime(&stats->ms_primary, ev_[0], ev_[1]));
    HPT_SOFT(cudaEventElapsedTime(&stats->ms_loop, ev_[1], ev_[2]));
    stats->ms_shade = prof ? ms_shade : -1.f;
    stats->ms_intersect = prof ? ms_isect : -1.f;
    HPT_SOFT(cudaEventElapsedTime(&stats->ms_resolve, ev_[2], ev_[3]));
    stats->nodes_visited = (int64_t)ctrl_host_->nodes_visited;
    stats->leaves_visited = (int64_t)ctrl_host_->leaves_visited;
    stats->triangle_tests = (int64_t)ctrl_host_->tri_tests;
    stats->triangle_repeats = (int64_t)ctrl_host_->tri_repeats;
    for (int j = 0; j < n; ++j) stats->paths += slots_host_[j].num_paths;
  }
  if (ctrl_host_->err.flags & 2u)
    return fail(HPT_ERR_INVALID_SCENE, "device self-check %d failed (value %lld)",
                ctrl_host_->err.site, (long long)ctrl_host_->err.value);
  if (ctrl_host_->err.flags & 1u)
    return fail(HPT_ERR_TRAVERSAL_LIMIT, "a traversal hit its step cap");
  if (!drained && !ctrl_host_->done)
    return fail(HPT_ERR_TRAVERSAL_LIMIT, "the wavefront did not drain within %lld iterations",
                (long long)(max_batches * kBatch));
  return HPT_OK;
}

}  // namespace hpt
