// Host builder of the 8-wide bounding volume hierarchy the closest-hit
// kernels walk (layout in device_types.h, walk in bvh.cuh).
#pragma once

#include <vector>

#include "device_types.h"
#include "host.h"
#include "scene_pack.h"

namespace hpt {

struct PackedBvh {
  std::vector<BvhNode> nodes;
  std::vector<BvhTri> tris;  // in node order
  int max_depth = 0;         // wide levels below the root, < kBvhStack
  std::vector<float> edge_keys[3];  // DevScene::edge_keys
};

// Builds the hierarchy over the triangles of a packed scene and their flags
// for the certificate. points / triangles: the scene's own (4 values each).
// num_threads <= 0: all host cores; the result does not depend on it. Box
// rounding and flags are scaled by scene_eps (DevScene::scene_eps).
void build_bvh(const float* points, const int32_t* triangles, const PackedScene& scene,
               float scene_eps, int num_threads, PackedBvh& out);

}  // namespace hpt
