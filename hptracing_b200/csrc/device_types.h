// Device-side scene and wavefront layouts, shared by the host packer (C++)
// and the CUDA kernels. Plain structs only: no CUDA headers needed here.
#pragma once

#include <cstddef>
#include <cstdint>

namespace hpt {

// --- Traversal tree ------------------------------------------------------
// 8-byte node. meta bits 31..30: 0/1/2 = split axis of an inner node,
// 3 = leaf. Inner nodes: bits 29..0 = index of the left child; the right
// child is stored right after it. Leaves: bits 29..0 = leaf record index.
// word 1: split position (inner) / unused (leaf).
struct DevNode {
  uint32_t meta;
  float split;
};
static_assert(sizeof(DevNode) == 8, "8-byte traversal node");
constexpr uint32_t kLeafKind = 3u;
constexpr uint32_t kIndexMask = 0x3FFFFFFFu;

// Leaf record, 64 bytes (4 x 16 B):
//  [0] lo.x lo.y lo.z  first entry in leaf_refs (int bits)
//  [1] hi.x hi.y hi.z  number of entries (int bits)
//  [2] rope -x, +x, -y, +y   (node index, -1 = leaves the scene)
//  [3] rope -z, +z, reference node index, 0
// The box is the reference node's own box; ropes point to the smallest
// node on the other side of each face that contains the whole face.
struct DevLeaf {
  float lo[3];
  int32_t tri_begin;
  float hi[3];
  int32_t tri_count;
  int32_t rope[6];
  int32_t ref_node;
  int32_t pad;
};
static_assert(sizeof(DevLeaf) == 64, "64-byte leaf record");
static_assert(offsetof(DevLeaf, rope) == 32, "ropes at bytes 32-55 (read as int4 + int2)");

// Triangle record, one per triangle, 48 bytes (3 x 16 B): vertex a,
// e1 = b - a, e2 = c - a (computed in FP32 exactly as the reference's
// _single_intersect does), triangle id and material in the .w slots.
// Leaves reference triangles through 4-byte ids stored in the reference's
// gather order (the reference duplicates a straddling triangle in every
// leaf it touches - tens of references per triangle on its SAH trees - so
// ids keep the records themselves small enough to stay in L2).
struct DevTri {
  float a[3];
  int32_t tri_id;
  float e1[3];
  int32_t material;
  float e2[3];
  int32_t pad;
};
static_assert(sizeof(DevTri) == 48, "48-byte triangle record");

// --- Bounding volume hierarchy ---------------------------------------------
// 8-wide node with child boxes quantised to 8 bits per plane (after the
// published compressed wide layout of Ylitie, Karras and Laine, "Efficient
// Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs", 2017), 160
// bytes (10 x 16 B). A child's plane q on axis a lies at p[a] + q * 2^e[a].
//  slot i is an inner child when bit i of imask is set: its node is
//  child_base + popcount(imask & ((1 << i) - 1)). Otherwise meta[i] is 0 (no
//  child) or a leaf: bits 0-4 = first triangle relative to tri_base, bits
//  5-7 = one bit per triangle (1 to 3 triangles).
// A child has two boxes. A ray of direction d (d / |d| in 127ths) visits it
// by its wide box when it may run almost in the plane of a triangle below
// that the other box does not cover (bvh_build.cpp): |cone . d| <= 127 cone_s.
struct BvhNode {
  float p[3];
  uint8_t e[3];             // biased exponents (float bits e << 23)
  uint8_t imask;
  uint32_t child_base;
  uint32_t tri_base;
  uint8_t meta[8];
  uint8_t qlo[3][8];        // x, y, z lower planes of the 8 slots
  uint8_t qhi[3][8];        // upper planes
  uint8_t wlo[3][8];        // the same of the wide boxes
  uint8_t whi[3][8];
  int8_t cone[8][4];        // x, y, z, cone_s
};
static_assert(sizeof(BvhNode) == 160, "160-byte wide node");

// Triangle record in node order: the DevTri values, and for the certificate
// (bvh_certain in bvh.cuh) the lowest tree node that holds every leaf listing
// the triangle, and flags. kTriIrregular: the tree does not list the triangle
// in exactly the leaves its bounds touch. kTriUnordered: in one of them the
// entries are not in ascending order. Bits 8 + 4 f to 11 + 4 f (f = 2a / 2a + 1:
// the lower / upper bound on axis a): c > 0 when no leaf that lists it ends
// beyond that bound by less than kGapUnit * scene_eps * 2^(c - 1).
struct BvhTri {
  float a[3];
  int32_t tri_id;
  float e1[3];
  int32_t start_node;
  float e2[3];
  uint32_t flags;
};
static_assert(sizeof(BvhTri) == 48, "48-byte triangle record");
constexpr uint32_t kTriIrregular = 64u, kTriUnordered = 128u;

// The distances in BvhTri::flags, in units of DevScene::scene_eps (2e-5 of the
// scene's size).
constexpr float kGapUnit = 0.8f;

// Origins beyond 4 times the scene's size (in units of scene_eps; a coordinate)
// are walked through the tree: the slabs of the wide boxes are as thick as a
// distance of kMaxDistance sizes asks for.
constexpr float kMaxOrigin = 4 / 2e-5f;
constexpr double kMaxDistance = 5 * 1.7320508;

// Boxes of the hierarchy (derived in bvh_build.cpp): the sine of the angle to a
// triangle's plane, times the sine of its angle at vertex a, below which a ray
// counts as running in the plane; and what the walk grows boxes by, per
// distance from the ray's origin (37 roundings of 2^-24 over kGrazing). Boxes
// that begin beyond kCullFactor times the best t so far (16 such roundings
// beyond it), plus the slack of the tree walk's stopping rule, are not visited.
constexpr float kGrazing = 0.005f;
constexpr float kBoxGrowth = 2.2e-6f / kGrazing;
constexpr float kCullFactor = 1.0001f + 1e-6f / kGrazing;

// Entries of a ray's node stack; the builder bounds the depth below it (one
// entry at most per level).
constexpr int kBvhStack = 32;

// Per-texture descriptor: texel offset into the RGBA8 pool, width, height.
struct DevTexInfo {
  int64_t offset;
  int32_t w, h;
};

// Hash of edge directions. The other two components over the largest one, r1
// and r2 in [-1, 1], give a cell of 2^-18 by 2^-18; a bucket of four words holds
// the tags of the cells that edges are in, within kEdgeTolerance (0: none), and
// where it is full the next one goes on.
#ifdef __CUDACC__
#define HPT_SHARED __host__ __device__ __forceinline__
#else
#define HPT_SHARED inline
#endif
constexpr double kEdgeTolerance = 8e-7;
HPT_SHARED uint32_t edge_cell(float r) { return (uint32_t)((r + 1.f) * 262144.f); }
HPT_SHARED uint32_t edge_bucket(uint32_t cell1, uint32_t cell2, uint32_t buckets) {
  const uint32_t h = cell1 * 0x9E3779B1u ^ cell2 * 0x85EBCA77u;
  return (h ^ (h >> 15)) & (buckets - 1u);
}
HPT_SHARED uint32_t edge_tag(uint32_t cell1, uint32_t cell2) {
  return (cell1 * 0xC2B2AE3Du + cell2 * 0x27D4EB2Fu) | 1u;
}

// Pointers of one device-resident scene (all device addresses).
struct DevScene {
  const DevNode* nodes;
  const DevLeaf* leaves;
  const int32_t* leaf_refs;   // triangle ids in leaf (= reference gather) order
  const DevTri* tris;         // indexed by triangle id
  const float* points;      // float4 per vertex
  const float* normals;     // float4 per vertex or null
  const float* texcoords;   // float2 per vertex or null
  const int32_t* geometry;  // int4 (v0, v1, v2, material) per triangle
  const void* materials;    // hpt_ref_material[]
  const int32_t* lights;    // int4 [num_lights]
  const uint32_t* texels;   // RGBA8 pool
  const DevTexInfo* tex_info;
  int32_t num_nodes, num_leaves, num_leaf_tris, num_triangles;
  int32_t num_points, num_normals, num_texcoords, num_materials;
  int32_t num_lights, num_textures;
  float root_lo[3], root_hi[3];
  float scene_eps;          // termination slack in world units
  int32_t max_steps;        // traversal step cap per ray
  const BvhNode* bvh;       // wide nodes, root first
  const BvhTri* btris;      // triangle records in node order
  int32_t num_bvh, num_btris;
  // Emission, ambient colours and normals are finite: a ray of zero strength
  // adds zero wherever it hits.
  int32_t finite_shading;
  // Directions of the triangle edges e2 whose largest component is on axis a
  // (see edge_bucket; used by bvh_no_parallel_edge): the bits of four words a
  // bucket, a power of two of buckets, or none.
  const float* edge_keys[3];
  int32_t num_edge_keys[3];
};

// --- Wavefront job table ------------------------------------------------
// One render job (a frame of one scene) in a slot of the engine's table.
// Read-only while the job runs; its mutable scheduling state is DevSlot.
struct DevJob {
  DevScene scene;
  float view_p[3], top[3], right[3];
  float width, height;
  int32_t nx, ny;           // rays per frame along x and y
  int32_t pano;             // 1 = equirectangular (set_viewdirs_vr)
  int32_t vr_x_shift;       // int(right.x) * supersample_x
  float bg[3];
  int32_t spp, depth, disable_diffuse;
  int32_t first_sample;     // the frame's index of this job's sample 0 (RNG key)
  uint64_t seed;
  unsigned long long* accum;  // 3 x fixed-point u64 per ray
  uint32_t* flags;          // per ray: NaN / +inf / -inf markers (4 bits per channel)
  float* prim;              // primary hit cache, 8 floats per entry
  int32_t* prim_count;      // number of primary hits
  int64_t max_inflight;     // cap on started-but-unfinished paths (0 = none)
};

// Scheduling state of a slot. A job's paths are (primary hit k, sample s)
// pairs enumerated as q = s * hits + k; `cursor` is the next q to start.
struct DevSlot {
  int64_t num_paths;        // hits * spp, set after the primary pass
  int64_t cursor;
  unsigned long long done;  // paths finished (flushed)
  unsigned long long queries;  // secondary intersect queries issued
  int64_t max_inflight;     // copied from the job at admission (0 = none)
  int32_t alloc;            // new paths granted for the coming shade pass
  int32_t active;           // admitted and not yet fully issued
};

// Error word shared by the kernels. flags bit 0: a traversal hit its step
// cap; bit 1: a device self-check failed (builds with HPT_DEVICE_CHECKS),
// in which case site / value describe the first failure.
struct DevErr {
  uint32_t flags;
  int32_t site;
  long long value;
};

// Wavefront control block (device memory, updated by the control kernel).
struct DevCtrl {
  int32_t nQ;               // paths in the queue the coming shade pass reads
  int32_t nR;               // survivors it wrote to the other queue
  int32_t shade_head;       // the shade pass's item cursor
  int32_t parity;           // which queue the coming shade pass reads
  int32_t n_new;            // new paths granted to the coming shade pass
  int32_t done;             // no queued path and nothing left to issue
  int32_t n_quota;          // slots with a grant (quota_slot / quota_prefix)
  int32_t n_order;          // slots in priority order (host-written)
  int64_t iterations;
  // Refill cursors of the intersect and primary kernels. 64-bit: one
  // admission's primary rays may exceed 2^31 (several jobs of up to 2^30
  // rays each).
  unsigned long long isect_head;
  unsigned long long prim_head;
  DevErr err;
  unsigned long long isect_queries;
  unsigned long long shades;
  unsigned long long nodes_visited;
  unsigned long long leaves_visited;
  unsigned long long tri_tests;
  unsigned long long tri_repeats;
  // Self-check builds only: items the shade / intersect passes of the
  // current iteration actually processed, compared by the control kernel
  // with the queue sizes.
  int32_t chk_shade_items;
  int32_t chk_shade_done;
  int32_t chk_isect_done;
  int32_t ticket;           // blocks of the running launch that are done
  // Per queue, after it was traced: rays in the hit list and the open list.
  int32_t n_hit[2], n_open[2];
  // Started-but-unfinished paths all capped slots (max_inflight > 0) may
  // hold together (0 = no shared cap); host-written.
  int64_t capped_budget;
};

// Fixed-point scale of the per-ray accumulators (2^32): integer sums are
// exact and order-independent, so a render is bit-reproducible no matter
// how paths are scheduled.
constexpr double kAccumScale = 4294967296.0;

}  // namespace hpt
