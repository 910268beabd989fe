// Host packer: reference KD-tree + triangles -> traversal layout.
#pragma once

#include <cmath>
#include <vector>

#include "device_types.h"
#include "host.h"

namespace hpt {

// The direction of the line along (b, c) as one number in (-1, 1]: c over
// |b| + |c|, of the two opposite directions the one with b > 0.
inline float edge_key(float b, float c) {
  const float sum = std::fabs(b) + std::fabs(c);
  return b == 0.f ? 1.f : (b > 0.f ? c : -c) / sum;
}

struct PackedScene {
  std::vector<DevNode> nodes;
  std::vector<DevLeaf> leaves;
  std::vector<int32_t> refs;   // triangle ids in leaf order
  std::vector<DevTri> tris;    // one record per triangle
  float root_lo[3], root_hi[3];
  int max_depth = 0;
};

// The first bfs_nodes node slots are filled breadth-first from the root.
hpt_status pack_scene(const hpt_scene_desc& desc, int bfs_nodes, PackedScene& out);

}  // namespace hpt
