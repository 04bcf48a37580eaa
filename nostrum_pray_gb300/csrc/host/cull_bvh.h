// The culling hierarchy: a bounding-volume hierarchy over the scene's
// triangles, each once, in the device's node layout. It finds every triangle
// that a ray can hit; which of those hits the reference's tree would report
// is decided at the hit (flatten.h).
#pragma once

#include <cstdint>
#include <vector>

#include "../device_layout.h"
#include "geom.h"
#include "threads.h"

namespace pray_gpu {

struct CullBvh {
    // Root at 0, slot 1 unused, the children of an interior node side by side,
    // pairs in depth-first order. Boxes are unpadded triangle bounds; leaves
    // index `order`.
    std::vector<GNode> nodes;
    std::vector<uint32_t> order;  // triangle ids, leaves concatenated
};

// Over every triangle: binned surface-area splits over box centres, leaves of
// at most `leaf_max` triangles (1 to kCullLeaf), at most kCullDepth levels
// below the root as long as halving can reach that: the kernels need their
// larger traversal stack from there on. The same result for any number of
// threads (0: every hardware thread).
constexpr int kCullLeaf = 4, kCullDepth = 31;
CullBvh build_cull_bvh(const std::vector<TriPre> &tris, int leaf_max, Threads &threads);
inline CullBvh build_cull_bvh(const std::vector<TriPre> &tris, int leaf_max, int threads) {
    Threads budget(threads);
    return build_cull_bvh(tris, leaf_max, budget);
}

}  // namespace pray_gpu
