// C ABI: device-resident scenes, render, per-stage entry points, stream
// compaction, batching. (Host-only producers live in capi_host.cpp.)
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/hpt.h"
#include "bvh.cuh"
#include "bvh_build.h"
#include "engine.h"
#include "scene_pack.h"
#include "shading.cuh"
#include "traverse.cuh"

using namespace hpt;

namespace hpt {

namespace {

template <typename T>
hpt_status dev_upload(SceneDev& s, const T* host, size_t count, const T** out) {
  *out = nullptr;
  if (count == 0) return HPT_OK;
  void* p = nullptr;
  HPT_CUDA(cudaMalloc(&p, count * sizeof(T)));
  s.allocations.push_back(p);
  s.bytes += (int64_t)(count * sizeof(T));
  HPT_CUDA(cudaMemcpy(p, host, count * sizeof(T), cudaMemcpyHostToDevice));
  *out = static_cast<const T*>(p);
  return HPT_OK;
}

// Device buffer for stage entry points: upload (optional) and download.
struct DBuf {
  void* p = nullptr;
  size_t bytes = 0;
  ~DBuf() {
    if (p) HPT_SOFT(cudaFree(p));
  }
  hpt_status alloc(size_t b) {
    bytes = b;
    if (b == 0) return HPT_OK;
    HPT_CUDA(cudaMalloc(&p, b));
    return HPT_OK;
  }
  hpt_status up(const void* host, size_t b) {
    hpt_status s = alloc(b);
    if (s != HPT_OK || b == 0) return s;
    HPT_CUDA(cudaMemcpy(p, host, b, cudaMemcpyHostToDevice));
    return HPT_OK;
  }
  hpt_status down(void* host) const {
    if (!host || bytes == 0) return HPT_OK;
    HPT_CUDA(cudaMemcpy(host, p, bytes, cudaMemcpyDeviceToHost));
    return HPT_OK;
  }
  template <typename T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

// One stage call on a scene: its buffers are parts of one allocation from the
// scene's own stream-ordered pool, and everything runs on the scene's stage
// stream. (A cudaMalloc and cudaFree per buffer took 8 to 60 ms of a call on
// 1M rays; the pool keeps up to kStagePoolKeep mapped and goes with the
// scene.)
constexpr uint64_t kStagePoolKeep = 256ull << 20;
class StageCall {
 public:
  explicit StageCall(SceneHandle& h) : h_(h) {}
  ~StageCall() {
    if (base_) HPT_SOFT(cudaFreeAsync(base_, h_.stage_stream));
    if (h_.stage_stream) HPT_SOFT(cudaStreamSynchronize(h_.stage_stream));
  }
  // Reserves a buffer; returns its number.
  int add(size_t bytes) {
    at_.push_back(size_);
    bytes_.push_back(bytes);
    size_ += (bytes + 255) & ~(size_t)255;
    return (int)at_.size() - 1;
  }
  // Allocates what was reserved.
  hpt_status begin() {
    HPT_CUDA(cudaSetDevice(h_.scene.device));
    if (!h_.stage_stream)
      HPT_CUDA(cudaStreamCreateWithFlags(&h_.stage_stream, cudaStreamNonBlocking));
    // Each is made if it is missing: one may have failed in an earlier call.
    if (!h_.stage_pool) {
      cudaMemPoolProps props;
      memset(&props, 0, sizeof props);
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = h_.scene.device;
      HPT_CUDA(cudaMemPoolCreate(&h_.stage_pool, &props));
      uint64_t keep = kStagePoolKeep;
      HPT_CUDA(cudaMemPoolSetAttribute(h_.stage_pool, cudaMemPoolAttrReleaseThreshold, &keep));
    }
    void* p = nullptr;
    HPT_CUDA(cudaMallocFromPoolAsync(&p, size_, h_.stage_pool, h_.stage_stream));
    base_ = static_cast<uint8_t*>(p);
    return HPT_OK;
  }
  template <typename T>
  T* ptr(int k) const {
    return reinterpret_cast<T*>(base_ + at_[k]);
  }
  hpt_status up(int k, const void* host) {
    HPT_CUDA(cudaMemcpyAsync(base_ + at_[k], host, bytes_[k], cudaMemcpyHostToDevice,
                             h_.stage_stream));
    return HPT_OK;
  }
  hpt_status down(int k, void* host) {
    HPT_CUDA(cudaMemcpyAsync(host, base_ + at_[k], bytes_[k], cudaMemcpyDeviceToHost,
                             h_.stage_stream));
    return HPT_OK;
  }
  hpt_status wait() {
    HPT_CUDA(cudaStreamSynchronize(h_.stage_stream));
    return HPT_OK;
  }
  cudaStream_t stream() const { return h_.stage_stream; }

 private:
  SceneHandle& h_;
  uint8_t* base_ = nullptr;
  size_t size_ = 0;
  std::vector<size_t> at_, bytes_;
};

// ---------------------------------------------------------------------------
// Stage kernels (one thread per element).
// ---------------------------------------------------------------------------
__global__ void k_stage_intersect(const DevScene* s, int n, const float* o, const float* d,
                                  int32_t* tri, float* t, float* u, float* v, DevErr* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Ray r{mk(o[3 * i], o[3 * i + 1], o[3 * i + 2]), mk(d[3 * i], d[3 * i + 1], d[3 * i + 2])};
  TravCount cnt{};
  int32_t hit;
  float ht, hu = 0.f, hv = 0.f;
  bvh_query(*s, r, hit, ht, err, cnt);
  if (hit >= 0) {  // the winning test's u, v
    const float4* rec = reinterpret_cast<const float4*>(s->tris + hit);
    float t2;
    mt_test(r, ldg(rec), ldg(rec + 1), ldg(rec + 2), t2, hu, hv);
  }
  tri[i] = hit;
  t[i] = ht;
  u[i] = hu;
  v[i] = hv;
}

__global__ void k_stage_shade(const DevScene* s, int n, const float* o, const float* d,
                              const float* strength, const int32_t* tri, const float* t,
                              uint64_t* seeds, int disable_diffuse, float* contrib,
                              int32_t* branch, float* hit_p, float* normal, float* strength_out,
                              float* param) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t seed = seeds[i];
  const Ray r{mk(o[3 * i], o[3 * i + 1], o[3 * i + 2]), mk(d[3 * i], d[3 * i + 1], d[3 * i + 2])};
  const ShadeOut so = shade_hit(*s, r, mk(strength[3 * i], strength[3 * i + 1], strength[3 * i + 2]),
                                tri[i], t[i], disable_diffuse, seed);
  seeds[i] = seed;
  contrib[3 * i] = so.contrib.x; contrib[3 * i + 1] = so.contrib.y; contrib[3 * i + 2] = so.contrib.z;
  hit_p[3 * i] = so.hit_p.x; hit_p[3 * i + 1] = so.hit_p.y; hit_p[3 * i + 2] = so.hit_p.z;
  normal[3 * i] = so.normal.x; normal[3 * i + 1] = so.normal.y; normal[3 * i + 2] = so.normal.z;
  strength_out[3 * i] = so.strength.x;
  strength_out[3 * i + 1] = so.strength.y;
  strength_out[3 * i + 2] = so.strength.z;
  param[i] = so.param;
  branch[i] = so.branch;
}

__global__ void k_stage_next(const DevScene* s, int n, const int32_t* branch, const float* d,
                             const float* hit_p, const float* normal, const float* strength,
                             const float* param, uint64_t* seeds, float* o_out, float* d_out,
                             float* s_out, int32_t* alive) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t seed = seeds[i];
  const NextOut no = next_direction(*s, branch[i], mk(d[3 * i], d[3 * i + 1], d[3 * i + 2]),
                                    mk(hit_p[3 * i], hit_p[3 * i + 1], hit_p[3 * i + 2]),
                                    mk(normal[3 * i], normal[3 * i + 1], normal[3 * i + 2]),
                                    mk(strength[3 * i], strength[3 * i + 1], strength[3 * i + 2]),
                                    param[i], seed);
  seeds[i] = seed;
  o_out[3 * i] = no.o.x; o_out[3 * i + 1] = no.o.y; o_out[3 * i + 2] = no.o.z;
  d_out[3 * i] = no.d.x; d_out[3 * i + 1] = no.d.y; d_out[3 * i + 2] = no.d.z;
  s_out[3 * i] = no.strength.x; s_out[3 * i + 1] = no.strength.y; s_out[3 * i + 2] = no.strength.z;
  alive[i] = no.alive ? 1 : 0;
}

__global__ void k_stage_raygen(hpt_camera cam, int nx, int ny, int pano, int x_shift, float* o,
                               float* d) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= nx || y >= ny) return;
  const f3 dir = pano ? pano_dir(x, y, x_shift, ny)
                      : pinhole_dir(cam.top_dir, cam.right_dir, cam.width, cam.height, x, y, nx, ny);
  const int64_t idx = (int64_t)nx * y + x;
  o[3 * idx] = cam.view_p[0]; o[3 * idx + 1] = cam.view_p[1]; o[3 * idx + 2] = cam.view_p[2];
  d[3 * idx] = dir.x; d[3 * idx + 1] = dir.y; d[3 * idx + 2] = dir.z;
}

__device__ __forceinline__ uint8_t unorm8(float x) {
  const float v = __fmul_rn(x, 255.0f);
  if (!(v >= 0.f)) return 0;
  if (v >= 255.f) return 255;
  return (uint8_t)__float2int_rn(v);
}

__global__ void k_stage_resolve(const float* accum, int W, int H, int ssx, int ssy, int spp,
                                float brightness, uint8_t* rgba) {
  const int gx = blockIdx.x * blockDim.x + threadIdx.x;
  const int gy = blockIdx.y * blockDim.y + threadIdx.y;
  if (gx >= W || gy >= H) return;
  float p[3] = {0.f, 0.f, 0.f};
  for (int i = 0; i < ssx; ++i)
    for (int j = 0; j < ssy; ++j) {
      const int64_t idx = (int64_t)(gy * ssy + j) * W * ssx + gx * ssx + i;
      for (int c = 0; c < 3; ++c) p[c] = __fadd_rn(p[c], accum[3 * idx + c]);
    }
  uint8_t* out = rgba + 4 * ((int64_t)gy * W + gx);
  for (int c = 0; c < 3; ++c) {
    float x = __fmul_rn(__fdiv_rn(__fdiv_rn(p[c], (float)(ssx * ssy)), (float)spp), brightness);
    out[c] = unorm8(__fsub_rn(1.f, expf(-x)));
  }
  out[3] = 0;
}

// --- Stream compaction: per-warp counts, then a stable scatter. ----------
// The flags are split into rows of 32, and the rows into one contiguous share
// per warp of at most kCompactMaxWarps (8 blocks of 8 warps on each of 148
// SMs: what is resident at once, so large arrays run as one full wave). The
// count pass reads the flags once and stores each row as a 32-bit mask
// (n / 8 bytes in all) and the survivors of each warp's share and of each
// block's; the scatter pass, with the same shares, finds a warp's output
// position by summing the earlier blocks' and warps' counts (L2-resident)
// instead of waiting for a scan, and reads the masks instead of the flags. No
// kernel waits on another block: the two passes are ordered by the stream.
// At n = 2^25, half of them set, the passes read 134 MB and write 67 MB, 31 us
// at the copy rate, in 48.7 us (27 us counting, bound by DRAM; the scatter by
// its instructions per row). One 4,096-flag tile per block, with a memset and
// atomics for the tiles' totals: 55.3 us. At n <= 300,000, where launches
// count, 9.1 us against 12.2.
constexpr int kCompactThreads = 256;
constexpr int kCompactWarps = kCompactThreads / 32;
constexpr int kCompactMaxBlocks = 148 * 8;
constexpr int kCompactMaxWarps = kCompactMaxBlocks * kCompactWarps;
constexpr int kCompactBatch = 16;  // rows a warp has in flight

struct CompactShape {
  int64_t rows;  // of 32 flags
  int share;     // rows per warp, a multiple of kCompactBatch
  int blocks;
};
inline CompactShape compact_shape(int64_t n) {
  CompactShape c;
  c.rows = (n + 31) / 32;
  const int64_t per = (c.rows + kCompactMaxWarps - 1) / kCompactMaxWarps;
  c.share = (int)((per + kCompactBatch - 1) / kCompactBatch * kCompactBatch);
  c.blocks = (int)((c.rows + (int64_t)c.share * kCompactWarps - 1) / ((int64_t)c.share * kCompactWarps));
  return c;
}

__global__ void __launch_bounds__(kCompactThreads)
    k_compact_count(const uint32_t* flags, int n, int64_t rows, int share, uint32_t* masks,
                    int* warp_counts, int* block_counts) {
  __shared__ int sums[kCompactWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t g = (int64_t)blockIdx.x * kCompactWarps + warp;
  const int64_t end = min(rows, (g + 1) * share);
  int count = 0;
  for (int64_t r = g * share; r < end; r += kCompactBatch) {
    const int64_t i = r * 32 + lane;
    uint32_t v[kCompactBatch];
    if ((r + kCompactBatch) * 32 <= n) {
#pragma unroll
      for (int k = 0; k < kCompactBatch; ++k) v[k] = __ldcs(flags + i + 32 * k);
    } else {
#pragma unroll
      for (int k = 0; k < kCompactBatch; ++k) v[k] = i + 32 * k < n ? __ldcs(flags + i + 32 * k) : 0u;
    }
    uint32_t word = 0;
#pragma unroll
    for (int k = 0; k < kCompactBatch; ++k) {
      const uint32_t bits = __ballot_sync(0xFFFFFFFFu, v[k] != 0);
      if (lane == k) word = bits;
    }
    if (lane < kCompactBatch && r + lane < end) masks[r + lane] = word;
    count += __popc(word);
  }
  count = __reduce_add_sync(0xFFFFFFFFu, count);
  if (lane == 0) {
    warp_counts[g] = count;
    sums[warp] = count;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int k = 0; k < kCompactWarps; ++k) sum += sums[k];
    block_counts[blockIdx.x] = sum;
  }
}

// A warp's lanes write a row's survivors to consecutive slots with one
// coalesced store: the row's place comes from a scan of 32 rows' counts, a
// lane's in the row is the number of the row's bits below it. (Places and bits
// go through shared memory, two rows per 16-byte broadcast: 2 us less than
// shuffles at n = 2^25. Staging the survivors for 16-byte stores: no gain.)
// The last block writes the total.
__global__ void __launch_bounds__(kCompactThreads)
    k_compact_scatter(const uint32_t* masks, int64_t rows, int share, const int* warp_counts,
                      const int* block_counts, int* out, int* total) {
  __shared__ int before[kCompactWarps];
  __shared__ __align__(16) uint2 row_sh[kCompactWarps][32];  // a row's place and bits
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint2* row = row_sh[warp];
  cudaGridDependencySynchronize();  // the count pass is done
  int acc = 0;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += kCompactThreads) acc += block_counts[i];
  acc = __reduce_add_sync(0xFFFFFFFFu, acc);
  const int own = lane < kCompactWarps ? warp_counts[blockIdx.x * kCompactWarps + lane] : 0;
  int o = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? own : 0);
  if (lane == 0) before[warp] = acc;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kCompactWarps; ++k) o += before[k];
  const int64_t g = (int64_t)blockIdx.x * kCompactWarps + warp;
  const int64_t end = min(rows, (g + 1) * share);
  const uint32_t below = (1u << lane) - 1u;  // lanes below this one
  uint32_t next = g * share + lane < end ? masks[g * share + lane] : 0u;
  for (int64_t r = g * share; r < end; r += 32) {
    const uint32_t word = next;
    next = r + 32 + lane < end ? masks[r + 32 + lane] : 0u;
    const int c = __popc(word);
    int inc = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
      if (lane >= d) inc += y;
    }
    const int m = __shfl_sync(0xFFFFFFFFu, inc, 31);
    row[lane] = make_uint2((uint32_t)(o + inc - c), word);
    __syncwarp();
    const uint32_t i = (uint32_t)(r * 32) + lane;
#pragma unroll 8
    for (int k = 0; k < 32; k += 2) {
      const uint4 two = *reinterpret_cast<const uint4*>(row + k);
      if ((two.y >> lane) & 1u) out[two.x + __popc(two.y & below)] = (int)(i + 32u * k);
      if ((two.w >> lane) & 1u) out[two.z + __popc(two.w & below)] = (int)(i + 32u * k + 32u);
    }
    o += m;
    __syncwarp();
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == kCompactThreads - 32) *total = o;
}

inline int blocks_for(int64_t n, int bs) { return (int)((n + bs - 1) / bs); }

// Enqueues the two compaction passes on `st` for n > 0 flags. Scratch:
// compact_shape(n)'s rows masks, kCompactMaxWarps and kCompactMaxBlocks counts;
// the survivor count goes to *total. The scatter pass is launched while the
// count pass drains and waits for it on the device.
cudaError_t launch_compact(const uint32_t* flags, int n, uint32_t* masks, int* warp_counts,
                           int* block_counts, int* out, int* total, cudaStream_t st) {
  const CompactShape c = compact_shape(n);
  k_compact_count<<<c.blocks, kCompactThreads, 0, st>>>(flags, n, c.rows, c.share, masks,
                                                        warp_counts, block_counts);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(c.blocks);
  cfg.blockDim = dim3(kCompactThreads);
  cfg.stream = st;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_compact_scatter, (const uint32_t*)masks, c.rows, c.share,
                            (const int*)warp_counts, (const int*)block_counts, out, total);
}

hpt_status check_scene_desc(const hpt_scene_desc& d) {
  if (d.num_points < 0 || d.num_triangles <= 0 || d.num_nodes <= 0 || d.num_leaf_data < 0 ||
      d.num_materials <= 0 || d.num_lights < 0 || d.num_textures < 0 || d.num_normals < 0 ||
      d.num_texcoords < 0)
    return fail(HPT_ERR_INVALID_ARGUMENT, "scene: negative or empty counts");
  if (!d.points || !d.triangles || !d.nodes || !d.materials || (d.num_leaf_data && !d.leaf_data))
    return fail(HPT_ERR_INVALID_ARGUMENT, "scene: missing buffers");
  if (d.num_normals != 0 && d.num_normals != d.num_points)
    return fail(HPT_ERR_INVALID_SCENE,
                "scene: %d normals for %d vertices (normals are indexed by vertex id)",
                d.num_normals, d.num_points);
  if (d.num_texcoords != 0 && d.num_texcoords != d.num_points)
    return fail(HPT_ERR_INVALID_SCENE, "scene: %d texcoords for %d vertices", d.num_texcoords,
                d.num_points);
  const F4* pts = reinterpret_cast<const F4*>(d.points);
  for (int i = 0; i < d.num_points; ++i)
    if (!std::isfinite(pts[i].x) || !std::isfinite(pts[i].y) || !std::isfinite(pts[i].z))
      return fail(HPT_ERR_INVALID_SCENE, "scene: vertex %d is not finite", i);
  const I4* tris = reinterpret_cast<const I4*>(d.triangles);
  for (int i = 0; i < d.num_triangles; ++i) {
    const I4& t = tris[i];
    if (t.x < 0 || t.y < 0 || t.z < 0 || t.x >= d.num_points || t.y >= d.num_points ||
        t.z >= d.num_points)
      return fail(HPT_ERR_INVALID_SCENE, "scene: triangle %d vertex index out of range", i);
    if (t.w < 0 || t.w >= d.num_materials)
      return fail(HPT_ERR_INVALID_SCENE, "scene: triangle %d material %d out of range", i, t.w);
  }
  if (d.num_lights > 0 && !d.lights) return fail(HPT_ERR_INVALID_ARGUMENT, "scene: lights missing");
  const I4* lights = reinterpret_cast<const I4*>(d.lights);
  for (int i = 0; i < d.num_lights; ++i) {
    const I4& t = lights[i];
    if (t.x < 0 || t.y < 0 || t.z < 0 || t.x >= d.num_points || t.y >= d.num_points ||
        t.z >= d.num_points)
      return fail(HPT_ERR_INVALID_SCENE, "scene: light %d vertex index out of range", i);
  }
  for (int i = 0; i < d.num_materials; ++i) {
    const hpt_ref_material& m = d.materials[i];
    if (m.diffuse_texture_id >= d.num_textures || m.ambient_texture_id >= d.num_textures)
      return fail(HPT_ERR_INVALID_SCENE, "scene: material %d references a missing texture", i);
  }
  if (d.num_textures > 0 && !d.texture_data)
    return fail(HPT_ERR_INVALID_ARGUMENT, "scene: texture data missing");
  if (d.texture_dims)
    for (int i = 0; i < d.num_textures; ++i)
      if (d.texture_dims[2 * i] <= 0 || d.texture_dims[2 * i + 1] <= 0)
        return fail(HPT_ERR_INVALID_SCENE, "scene: texture %d has no texels", i);
  return HPT_OK;
}

}  // namespace

hpt_status upload_scene(const hpt_scene_desc& d, SceneDev& out) {
  hpt_status s = check_scene_desc(d);
  if (s != HPT_OK) return s;
  PackedScene pk;
  s = pack_scene(d, 8192, pk);
  if (s != HPT_OK) return s;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return fail(HPT_ERR_CUDA, "no CUDA device");
  if (d.device < 0 || d.device >= ndev) return fail(HPT_ERR_INVALID_ARGUMENT, "bad device %d", d.device);
  HPT_CUDA(cudaSetDevice(d.device));
  out.device = d.device;
  DevScene& ds = out.dev;
  memset(&ds, 0, sizeof ds);
  const DevNode* nodes;
  const DevLeaf* leaves;
  const DevTri* recs;
  const int32_t* refs;
  if ((s = dev_upload(out, pk.nodes.data(), pk.nodes.size(), &nodes)) != HPT_OK) return s;
  if ((s = dev_upload(out, pk.leaves.data(), pk.leaves.size(), &leaves)) != HPT_OK) return s;
  // At least one entry so the pointer is valid even for an empty tree.
  if (pk.refs.empty()) pk.refs.push_back(0);
  if ((s = dev_upload(out, pk.refs.data(), pk.refs.size(), &refs)) != HPT_OK) return s;
  if ((s = dev_upload(out, pk.tris.data(), pk.tris.size(), &recs)) != HPT_OK) return s;
  PackedBvh bvh;
  float scale = 0.f;
  for (int a = 0; a < 3; ++a) {
    ds.root_lo[a] = pk.root_lo[a];
    ds.root_hi[a] = pk.root_hi[a];
    scale = std::max({scale, std::fabs(pk.root_lo[a]), std::fabs(pk.root_hi[a]),
                      pk.root_hi[a] - pk.root_lo[a]});
  }
  ds.scene_eps = 2e-5f * scale;
  build_bvh(d.points, d.triangles, pk, ds.scene_eps, 0, bvh);
  if ((s = dev_upload(out, bvh.nodes.data(), bvh.nodes.size(), &ds.bvh)) != HPT_OK) return s;
  if (bvh.tris.empty()) bvh.tris.emplace_back();
  if ((s = dev_upload(out, bvh.tris.data(), bvh.tris.size(), &ds.btris)) != HPT_OK) return s;
  for (int a = 0; a < 3; ++a) {
    if ((s = dev_upload(out, bvh.edge_keys[a].data(), bvh.edge_keys[a].size(), &ds.edge_keys[a])) !=
        HPT_OK)
      return s;
    ds.num_edge_keys[a] = (int32_t)bvh.edge_keys[a].size();
  }
  ds.finite_shading = 1;
  for (int m = 0; m < d.num_materials; ++m)
    for (int k = 0; k < 3; ++k)
      if (!std::isfinite(d.materials[m].emission[k]) || !std::isfinite(d.materials[m].ambient[k]))
        ds.finite_shading = 0;
  for (int64_t k = 0; k < 4 * (int64_t)d.num_normals; ++k)
    if ((k & 3) != 3 && !std::isfinite(d.normals[k])) ds.finite_shading = 0;
  // (A triangle without area has no normal: 0 times NaN.)
  for (const DevTri& t : pk.tris) {
    const f3 n = cross(mk(t.e1[0], t.e1[1], t.e1[2]), mk(t.e2[0], t.e2[1], t.e2[2]));
    if (!(length(n) > 1e-30f)) ds.finite_shading = 0;
  }
  ds.num_bvh = (int32_t)bvh.nodes.size();
  ds.num_btris = (int32_t)bvh.tris.size();
  ds.nodes = nodes;
  ds.leaves = leaves;
  ds.leaf_refs = refs;
  ds.tris = recs;
  const float* f = nullptr;
  if ((s = dev_upload(out, d.points, 4 * (size_t)d.num_points, &f)) != HPT_OK) return s;
  ds.points = f;
  if ((s = dev_upload(out, d.normals, 4 * (size_t)d.num_normals, &f)) != HPT_OK) return s;
  ds.normals = f;
  if ((s = dev_upload(out, d.texcoords, 2 * (size_t)d.num_texcoords, &f)) != HPT_OK) return s;
  ds.texcoords = f;
  const int32_t* ip = nullptr;
  if ((s = dev_upload(out, d.triangles, 4 * (size_t)d.num_triangles, &ip)) != HPT_OK) return s;
  ds.geometry = ip;
  const hpt_ref_material* mp = nullptr;
  if ((s = dev_upload(out, d.materials, (size_t)d.num_materials, &mp)) != HPT_OK) return s;
  ds.materials = mp;
  if ((s = dev_upload(out, d.lights, 4 * (size_t)d.num_lights, &ip)) != HPT_OK) return s;
  ds.lights = ip;
  std::vector<DevTexInfo> ti(d.num_textures);
  int64_t texels = 0;
  for (int t = 0; t < d.num_textures; ++t) {
    ti[t].offset = texels;
    ti[t].w = d.texture_dims ? d.texture_dims[2 * t] : 512;
    ti[t].h = d.texture_dims ? d.texture_dims[2 * t + 1] : 512;
    texels += (int64_t)ti[t].w * ti[t].h;
  }
  const uint32_t* tx = nullptr;
  if ((s = dev_upload(out, reinterpret_cast<const uint32_t*>(d.texture_data), (size_t)texels, &tx)) != HPT_OK)
    return s;
  ds.texels = tx;
  const DevTexInfo* tip = nullptr;
  if ((s = dev_upload(out, ti.data(), ti.size(), &tip)) != HPT_OK) return s;
  ds.tex_info = tip;
  ds.num_nodes = (int32_t)pk.nodes.size();
  ds.num_leaves = (int32_t)pk.leaves.size();
  ds.num_leaf_tris = (int32_t)pk.refs.size();
  ds.num_triangles = d.num_triangles;
  ds.num_points = d.num_points;
  ds.num_normals = d.num_normals;
  ds.num_texcoords = d.num_texcoords;
  ds.num_materials = d.num_materials;
  ds.num_lights = d.num_lights;
  ds.num_textures = d.num_textures;
  const int64_t cap = 8 * ((int64_t)pk.nodes.size() + (int64_t)pk.refs.size()) + 100000;
  ds.max_steps = (int32_t)std::min<int64_t>(cap, 1 << 30);
  void* p = nullptr;
  HPT_CUDA(cudaMalloc(&p, sizeof(DevScene)));
  out.allocations.push_back(p);
  HPT_CUDA(cudaMemcpy(p, &ds, sizeof(DevScene), cudaMemcpyHostToDevice));
  // A cudaMemcpy from pageable memory may return before its DMA has landed,
  // and the render engines run on non-blocking streams that are not ordered
  // after the legacy stream: wait here so no kernel can read a partially
  // uploaded scene.
  HPT_CUDA(cudaDeviceSynchronize());
  out.d_scene = static_cast<DevScene*>(p);
  out.info.num_triangles = d.num_triangles;
  out.info.num_ref_nodes = d.num_nodes;
  out.info.num_device_nodes = ds.num_nodes;
  out.info.num_leaves = ds.num_leaves;
  out.info.num_leaf_triangles = (int32_t)pk.refs.size();
  out.info.max_depth = pk.max_depth;
  out.info.device_bytes = out.bytes;
  return HPT_OK;
}

void release_scene(SceneDev& s) {
  HPT_SOFT(cudaSetDevice(s.device));
  for (void* p : s.allocations) HPT_SOFT(cudaFree(p));
  s.allocations.clear();
}

}  // namespace hpt

namespace {

// Ranges the engine supports (capacity: queue entries; smem_nodes: accepted,
// without effect; trav_steps: 0 = the default, 1..256 rounds between refills;
// isect_block / isect_min_blocks: a compiled traversal variant,
// 0 min blocks = the block size's default).
hpt_status check_tuning(const hpt_tuning& t) {
  if (t.capacity < 1024 || t.capacity > (1 << 27) || t.smem_nodes < 0 ||
      t.smem_nodes > kMaxSmemNodes || t.refill_chunk < 1 || t.refill_chunk > 32 ||
      (t.isect_block != 128 && t.isect_block != 256) || t.isect_min_blocks < 0 ||
      t.trav_steps < 0 || t.trav_steps > 256 || t.max_steps < 0 ||
      (t.shade_min_blocks != 0 && t.shade_min_blocks != 3 && t.shade_min_blocks != 4))
    return fail(HPT_ERR_INVALID_ARGUMENT, "tuning out of range");
  return HPT_OK;
}

hpt_status check_params(const hpt_camera* cam, const hpt_render_params* p) {
  return check_render_params(cam, p);
}

template <typename F>
hpt_status guarded(F&& f) {
  try {
    return f();
  } catch (const std::bad_alloc&) {
    return fail(HPT_ERR_OUT_OF_MEMORY, "host allocation failed");
  } catch (...) {
    return fail(HPT_ERR_INVALID_ARGUMENT, "unexpected exception");
  }
}

}  // namespace

extern "C" {

int hpt_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    (void)cudaGetLastError();  // "no device" is an answer here, not an error
    return 0;
  }
  return n;
}

hpt_status hpt_scene_create(const hpt_scene_desc* desc, hpt_scene** out) {
  if (!desc || !out) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  *out = nullptr;
  return guarded([&]() -> hpt_status {
    std::unique_ptr<hpt_scene> s(new hpt_scene());
    hpt_status st = upload_scene(*desc, s->h.scene);
    if (st != HPT_OK) {
      release_scene(s->h.scene);
      return st;
    }
    s->h.tuning = default_tuning();
    *out = s.release();
    return HPT_OK;
  });
}

hpt_status hpt_scene_info_get(const hpt_scene* scene, hpt_scene_info* out) {
  if (!scene || !out) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  *out = scene->h.scene.info;
  return HPT_OK;
}

void hpt_scene_destroy(hpt_scene* scene) {
  if (!scene) return;
  {
    std::lock_guard<std::mutex> lk(scene->h.mu);
    scene->h.engine.reset();
    release_scene(scene->h.scene);
    if (scene->h.stage_stream) HPT_SOFT(cudaStreamDestroy(scene->h.stage_stream));
    if (scene->h.stage_pool) HPT_SOFT(cudaMemPoolDestroy(scene->h.stage_pool));
  }
  delete scene;
}

hpt_status hpt_render(hpt_scene* scene, const hpt_camera* camera, const hpt_render_params* params,
                      uint8_t* rgba_out, float* accum_out) {
  if (!scene) return fail(HPT_ERR_INVALID_ARGUMENT, "scene is NULL");
  hpt_status s = check_params(camera, params);
  if (s != HPT_OK) return s;
  return guarded([&]() -> hpt_status {
    std::lock_guard<std::mutex> lk(scene->h.mu);
    if (!scene->h.engine) scene->h.engine.reset(new Engine(scene->h.scene.device));
    scene->h.engine->tuning = scene->h.tuning;
    JobSpec js;
    js.scene = &scene->h.scene;
    js.camera = *camera;
    js.params = *params;
    js.rgba_out = rgba_out;
    js.accum_out = accum_out;
    return scene->h.engine->run({js}, &scene->h.last_stats);
  });
}

hpt_status hpt_render_stats_get(const hpt_scene* scene, hpt_render_stats* out) {
  if (!scene || !out) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  *out = scene->h.last_stats;
  return HPT_OK;
}

hpt_status hpt_tuning_get(const hpt_scene* scene, hpt_tuning* out) {
  if (!scene || !out) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  *out = scene->h.tuning;
  return HPT_OK;
}

hpt_status hpt_tuning_set(hpt_scene* scene, const hpt_tuning* in) {
  if (!scene || !in) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  hpt_status st = check_tuning(*in);
  if (st != HPT_OK) return st;
  std::lock_guard<std::mutex> lk(scene->h.mu);
  scene->h.tuning = *in;
  scene->h.tuning.shade_block = 256;
  scene->h.engine.reset();
  return HPT_OK;
}

hpt_status hpt_raygen(const hpt_camera* camera, int32_t sample_x, int32_t sample_y,
                      int32_t supersample_x, int32_t supersample_y, float* origins,
                      float* directions) {
  if (!camera || !origins || !directions || sample_x <= 0 || sample_y <= 0 || supersample_x <= 0 ||
      supersample_y <= 0)
    return fail(HPT_ERR_INVALID_ARGUMENT, "bad raygen arguments");
  if (camera->height < 0 && supersample_x != supersample_y)
    return fail(HPT_ERR_INVALID_ARGUMENT, "panorama needs supersample_x == supersample_y");
  return guarded([&]() -> hpt_status {
    const int nx = sample_x * supersample_x, ny = sample_y * supersample_y;
    const size_t bytes = (size_t)nx * ny * 3 * sizeof(float);
    DBuf o, d;
    hpt_status s;
    if ((s = o.alloc(bytes)) != HPT_OK || (s = d.alloc(bytes)) != HPT_OK) return s;
    const int pano = camera->height < 0;
    const int shift = (int)camera->right_dir[0] * supersample_x;
    dim3 blk(16, 16), grd((nx + 15) / 16, (ny + 15) / 16);
    k_stage_raygen<<<grd, blk>>>(*camera, nx, ny, pano, shift, o.as<float>(), d.as<float>());
    HPT_CUDA(cudaGetLastError());
    if ((s = o.down(origins)) != HPT_OK) return s;
    return d.down(directions);
  });
}

hpt_status hpt_intersect(hpt_scene* scene, int32_t n, const float* origins,
                         const float* directions, int32_t* tri_out, float* t_out, float* u_out,
                         float* v_out) {
  if (!scene || n < 0 || (n > 0 && (!origins || !directions || !tri_out || !t_out || !u_out || !v_out)))
    return fail(HPT_ERR_INVALID_ARGUMENT, "bad intersect arguments");
  if (n == 0) return HPT_OK;
  return guarded([&]() -> hpt_status {
    std::lock_guard<std::mutex> lk(scene->h.mu);
    const size_t b3 = (size_t)n * 3 * sizeof(float), b1 = (size_t)n * 4;
    StageCall c(scene->h);
    const int o = c.add(b3), d = c.add(b3), tri = c.add(b1), t = c.add(b1), u = c.add(b1),
              v = c.add(b1), err = c.add(sizeof(DevErr));
    hpt_status s;
    if ((s = c.begin()) || (s = c.up(o, origins)) || (s = c.up(d, directions))) return s;
    HPT_CUDA(cudaMemsetAsync(c.ptr<DevErr>(err), 0, sizeof(DevErr), c.stream()));
    k_stage_intersect<<<blocks_for(n, 128), 128, 0, c.stream()>>>(
        scene->h.scene.d_scene, n, c.ptr<float>(o), c.ptr<float>(d), c.ptr<int32_t>(tri),
        c.ptr<float>(t), c.ptr<float>(u), c.ptr<float>(v), c.ptr<DevErr>(err));
    HPT_CUDA(cudaGetLastError());
    DevErr e;
    if ((s = c.down(tri, tri_out)) || (s = c.down(t, t_out)) || (s = c.down(u, u_out)) ||
        (s = c.down(v, v_out)) || (s = c.down(err, &e)) || (s = c.wait()))
      return s;
    if (e.flags & 2u)
      return fail(HPT_ERR_INVALID_SCENE, "device self-check %d failed (value %lld)", e.site,
                  (long long)e.value);
    if (e.flags) return fail(HPT_ERR_TRAVERSAL_LIMIT, "a traversal hit its step cap");
    return HPT_OK;
  });
}

hpt_status hpt_shade(hpt_scene* scene, int32_t n, const float* origins, const float* directions,
                     const float* strengths, const int32_t* tris, const float* ts, uint64_t* seeds,
                     int32_t disable_diffuse, float* contrib, int32_t* branch, float* hit_p,
                     float* normal, float* strength_out, float* param) {
  if (!scene || n < 0 ||
      (n > 0 && (!origins || !directions || !strengths || !tris || !ts || !seeds || !contrib ||
                 !branch || !hit_p || !normal || !strength_out || !param)))
    return fail(HPT_ERR_INVALID_ARGUMENT, "bad shade arguments");
  if (n == 0) return HPT_OK;
  for (int i = 0; i < n; ++i)
    if (tris[i] < 0 || tris[i] >= scene->h.scene.info.num_triangles)
      return fail(HPT_ERR_INVALID_ARGUMENT, "shade: triangle id %d out of range", tris[i]);
  return guarded([&]() -> hpt_status {
    std::lock_guard<std::mutex> lk(scene->h.mu);
    const size_t b3 = (size_t)n * 3 * sizeof(float), b1 = (size_t)n * 4, b8 = (size_t)n * 8;
    StageCall c(scene->h);
    const int o = c.add(b3), d = c.add(b3), st = c.add(b3), tri = c.add(b1), t = c.add(b1),
              sd = c.add(b8), co = c.add(b3), br = c.add(b1), hp = c.add(b3), nm = c.add(b3),
              so = c.add(b3), pa = c.add(b1);
    hpt_status s;
    if ((s = c.begin()) || (s = c.up(o, origins)) || (s = c.up(d, directions)) ||
        (s = c.up(st, strengths)) || (s = c.up(tri, tris)) || (s = c.up(t, ts)) ||
        (s = c.up(sd, seeds)))
      return s;
    k_stage_shade<<<blocks_for(n, 128), 128, 0, c.stream()>>>(
        scene->h.scene.d_scene, n, c.ptr<float>(o), c.ptr<float>(d), c.ptr<float>(st),
        c.ptr<int32_t>(tri), c.ptr<float>(t), c.ptr<uint64_t>(sd), disable_diffuse,
        c.ptr<float>(co), c.ptr<int32_t>(br), c.ptr<float>(hp), c.ptr<float>(nm),
        c.ptr<float>(so), c.ptr<float>(pa));
    HPT_CUDA(cudaGetLastError());
    if ((s = c.down(sd, seeds)) || (s = c.down(co, contrib)) || (s = c.down(br, branch)) ||
        (s = c.down(hp, hit_p)) || (s = c.down(nm, normal)) || (s = c.down(so, strength_out)) ||
        (s = c.down(pa, param)))
      return s;
    return c.wait();
  });
}

hpt_status hpt_next_dir(hpt_scene* scene, int32_t n, const int32_t* branch,
                        const float* directions, const float* hit_p, const float* normal,
                        const float* strengths, const float* param, uint64_t* seeds,
                        float* origins_out, float* directions_out, float* strength_out,
                        int32_t* alive_out) {
  if (!scene || n < 0 ||
      (n > 0 && (!branch || !directions || !hit_p || !normal || !strengths || !param || !seeds ||
                 !origins_out || !directions_out || !strength_out || !alive_out)))
    return fail(HPT_ERR_INVALID_ARGUMENT, "bad next_dir arguments");
  if (n == 0) return HPT_OK;
  return guarded([&]() -> hpt_status {
    std::lock_guard<std::mutex> lk(scene->h.mu);
    const size_t b3 = (size_t)n * 3 * sizeof(float), b1 = (size_t)n * 4, b8 = (size_t)n * 8;
    StageCall c(scene->h);
    const int br = c.add(b1), d = c.add(b3), hp = c.add(b3), nm = c.add(b3), st = c.add(b3),
              pa = c.add(b1), sd = c.add(b8), oo = c.add(b3), dd = c.add(b3), so = c.add(b3),
              al = c.add(b1);
    hpt_status s;
    if ((s = c.begin()) || (s = c.up(br, branch)) || (s = c.up(d, directions)) ||
        (s = c.up(hp, hit_p)) || (s = c.up(nm, normal)) || (s = c.up(st, strengths)) ||
        (s = c.up(pa, param)) || (s = c.up(sd, seeds)))
      return s;
    k_stage_next<<<blocks_for(n, 128), 128, 0, c.stream()>>>(
        scene->h.scene.d_scene, n, c.ptr<int32_t>(br), c.ptr<float>(d), c.ptr<float>(hp),
        c.ptr<float>(nm), c.ptr<float>(st), c.ptr<float>(pa), c.ptr<uint64_t>(sd),
        c.ptr<float>(oo), c.ptr<float>(dd), c.ptr<float>(so), c.ptr<int32_t>(al));
    HPT_CUDA(cudaGetLastError());
    if ((s = c.down(sd, seeds)) || (s = c.down(oo, origins_out)) ||
        (s = c.down(dd, directions_out)) || (s = c.down(so, strength_out)) ||
        (s = c.down(al, alive_out)))
      return s;
    return c.wait();
  });
}

hpt_status hpt_compact(const uint32_t* flags, int32_t n, int32_t* out, int32_t* count) {
  if (n < 0 || !count || (n > 0 && (!flags || !out)))
    return fail(HPT_ERR_INVALID_ARGUMENT, "bad compact arguments");
  *count = 0;
  if (n == 0) return HPT_OK;
  if (hpt_device_count() == 0) return fail(HPT_ERR_CUDA, "no CUDA device");
  return guarded([&]() -> hpt_status {
    DBuf f, o, mk, wc, bc, tot;
    hpt_status s;
    if ((s = f.up(flags, (size_t)n * 4)) || (s = o.alloc((size_t)n * 4)) ||
        (s = mk.alloc((size_t)compact_shape(n).rows * 4)) ||
        (s = wc.alloc(kCompactMaxWarps * 4)) || (s = bc.alloc(kCompactMaxBlocks * 4)) ||
        (s = tot.alloc(4)))
      return s;
    HPT_CUDA(launch_compact(f.as<uint32_t>(), n, mk.as<uint32_t>(), wc.as<int>(), bc.as<int>(),
                            o.as<int>(), tot.as<int>(), 0));
    int total = 0;
    if ((s = tot.down(&total))) return s;
    if (total > 0) HPT_CUDA(cudaMemcpy(out, o.p, (size_t)total * 4, cudaMemcpyDeviceToHost));
    *count = total;
    return HPT_OK;
  });
}

hpt_status hpt_resolve(const float* accum, int32_t sample_x, int32_t sample_y, int32_t supersample_x,
                       int32_t supersample_y, int32_t sample, float brightness, uint8_t* rgba_out) {
  if (!accum || !rgba_out || sample_x <= 0 || sample_y <= 0 || supersample_x <= 0 ||
      supersample_y <= 0 || sample <= 0)
    return fail(HPT_ERR_INVALID_ARGUMENT, "bad resolve arguments");
  if (hpt_device_count() == 0) return fail(HPT_ERR_CUDA, "no CUDA device");
  return guarded([&]() -> hpt_status {
    const size_t rays = (size_t)sample_x * supersample_x * sample_y * supersample_y;
    DBuf a, o;
    hpt_status s;
    if ((s = a.up(accum, rays * 3 * sizeof(float))) || (s = o.alloc((size_t)sample_x * sample_y * 4)))
      return s;
    dim3 blk(16, 16), grd((sample_x + 15) / 16, (sample_y + 15) / 16);
    k_stage_resolve<<<grd, blk>>>(a.as<float>(), sample_x, sample_y, supersample_x, supersample_y,
                                  sample, brightness, o.as<uint8_t>());
    HPT_CUDA(cudaGetLastError());
    return o.down(rgba_out);
  });
}

// --- Batching ---------------------------------------------------------------

struct hpt_batch {
  int device;
  std::unique_ptr<Engine> engine;
  std::vector<JobSpec> jobs;
  hpt_render_stats stats{};
  hpt_tuning tuning = default_tuning();
};

hpt_status hpt_batch_create(int32_t device, hpt_batch** out) {
  if (!out) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  *out = nullptr;
  if (device < 0 || device >= hpt_device_count()) return fail(HPT_ERR_CUDA, "no CUDA device %d", device);
  return guarded([&]() -> hpt_status {
    hpt_batch* b = new hpt_batch();
    b->device = device;
    *out = b;
    return HPT_OK;
  });
}

hpt_status hpt_batch_add(hpt_batch* batch, hpt_scene* scene, const hpt_camera* camera,
                         const hpt_render_params* params, uint8_t* rgba_out, float* accum_out,
                         int32_t* job_id) {
  if (!batch || !scene) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  hpt_status s = check_params(camera, params);
  if (s != HPT_OK) return s;
  if (scene->h.scene.device != batch->device)
    return fail(HPT_ERR_INVALID_ARGUMENT, "scene lives on another device");
  JobSpec js;
  js.scene = &scene->h.scene;
  js.camera = *camera;
  js.params = *params;
  js.rgba_out = rgba_out;
  js.accum_out = accum_out;
  batch->jobs.push_back(js);
  if (job_id) *job_id = (int32_t)batch->jobs.size() - 1;
  return HPT_OK;
}

hpt_status hpt_batch_run(hpt_batch* batch) {
  if (!batch) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  return guarded([&]() -> hpt_status {
    if (!batch->engine) batch->engine.reset(new Engine(batch->device));
    batch->engine->tuning = batch->tuning;
    hpt_status s = batch->engine->run(batch->jobs, &batch->stats);
    batch->jobs.clear();
    return s;
  });
}

hpt_status hpt_batch_stats_get(const hpt_batch* batch, hpt_render_stats* out) {
  if (!batch || !out) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  *out = batch->stats;
  return HPT_OK;
}

hpt_status hpt_batch_tuning_set(hpt_batch* batch, const hpt_tuning* in) {
  if (!batch || !in) return fail(HPT_ERR_INVALID_ARGUMENT, "NULL argument");
  hpt_status st = check_tuning(*in);
  if (st != HPT_OK) return st;
  batch->tuning = *in;
  batch->tuning.shade_block = 256;
  batch->engine.reset();
  return HPT_OK;
}

void hpt_batch_destroy(hpt_batch* batch) { delete batch; }

}  // extern "C"

// ---------------------------------------------------------------------------
// hpt_compact_noalloc: the compaction kernels over caller-owned device
// buffers, with the counts and the masks in static device arrays instead of
// cudaMalloc'd ones. For callers that cannot allocate device memory where
// they call it (allocation synchronises the device and would stall their
// stream; a fixed memory budget leaves nothing to allocate).
// ---------------------------------------------------------------------------
namespace {

// A mask bit per flag (4 MiB per device) and the counts of the warps' and the
// blocks' shares (42 KB).
static __device__ __align__(256) uint32_t g_noalloc_masks[HPT_COMPACT_NOALLOC_MAX_N / 32];
static __device__ __align__(256) int g_noalloc_warp_counts[kCompactMaxWarps];
static __device__ __align__(256) int g_noalloc_block_counts[kCompactMaxBlocks];

struct NoallocScratch {
  uint32_t* masks = nullptr;
  int* warps = nullptr;
  int* blocks = nullptr;
};

// Device addresses of the static scratch arrays, looked up once per device
// with that device current (the first call on a device does this set-up).
// The cached addresses belong to the device's current context: after a
// cudaDeviceReset the caller must not use this entry point again in the
// same process.
hpt_status noalloc_scratch(int device, NoallocScratch* out) {
  static std::mutex mu;
  static std::vector<NoallocScratch> addr;
  std::lock_guard<std::mutex> lk(mu);
  if ((int)addr.size() <= device) addr.resize(device + 1);
  if (!addr[device].masks) {
    void* m = nullptr;
    void* w = nullptr;
    void* b = nullptr;
    HPT_CUDA(cudaGetSymbolAddress(&m, g_noalloc_masks));
    HPT_CUDA(cudaGetSymbolAddress(&w, g_noalloc_warp_counts));
    HPT_CUDA(cudaGetSymbolAddress(&b, g_noalloc_block_counts));
    addr[device].masks = static_cast<uint32_t*>(m);
    addr[device].warps = static_cast<int*>(w);
    addr[device].blocks = static_cast<int*>(b);
  }
  *out = addr[device];
  return HPT_OK;
}

}  // namespace

extern "C" hpt_status hpt_compact_noalloc(const uint32_t* flags, int32_t n, int32_t* out,
                                          int32_t* count, void* stream) {
  if (n < 0 || !count || (n > 0 && (!flags || !out)))
    return fail(HPT_ERR_INVALID_ARGUMENT, "bad compact arguments");
  if (n > HPT_COMPACT_NOALLOC_MAX_N)
    return fail(HPT_ERR_INVALID_ARGUMENT,
                "hpt_compact_noalloc: n = %d exceeds the limit of %d flags (static scratch)", n,
                HPT_COMPACT_NOALLOC_MAX_N);
  int device = 0;
  HPT_CUDA(cudaGetDevice(&device));
  NoallocScratch scratch;
  // The lookup table may grow (host memory): no exception leaves the ABI.
  hpt_status s = guarded([&]() -> hpt_status { return noalloc_scratch(device, &scratch); });
  if (s != HPT_OK) return s;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (n == 0) {
    HPT_CUDA(cudaMemsetAsync(count, 0, sizeof(int32_t), st));
    return HPT_OK;
  }
  // Every scratch entry the scatter reads is written by the count pass; the
  // total goes straight to the caller's counter.
  HPT_CUDA(launch_compact(flags, n, scratch.masks, scratch.warps, scratch.blocks, out, count, st));
  return HPT_OK;
}
