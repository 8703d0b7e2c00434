// quad_build.h — host construction of the four-wide tree that the closest-hit
// kernels walk (QuadNode, wr_device.cuh).
#pragma once

#include <cstdint>
#include <vector>

#include "kdtree_build.h"
#include "wr_device.cuh"

namespace wr {

// what the device needs beside the reference tree's own records
struct QuadLayout {
    std::vector<QuadNode> quads;     // [0] is the root
    std::vector<uint32_t> leaf_up;   // per triangle slot: (pair << 1 | side) of its leaf, UP_ROOT if the root is that leaf
    std::vector<uint4> pair_up;      // per pair: (pair << 1 | side) of its parent and the three above, UP_ROOT past the root
    uint32_t stack = 0;              // entries that the deepest walk can need (a node's other children, all the way down)
};

// Four-wide tree over the reference tree's leaves (their own boxes, bit for
// bit) by the surface-area heuristic, and the reference tree's parent links.
// Leaves with a vertex that is not finite lie above it, for every ray.  A scene
// of more than QUAD_MAX_SLOTS triangles gets an empty `quads` (the batch kernel
// and the wavefront walk the reference's tree, the other renderers' rays take
// reference_search one by one).
QuadLayout build_quads(const HostTree& t, int threads);

}  // namespace wr
