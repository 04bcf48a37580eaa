// Flattening of a built tree into the device layout (device_layout.h).
//
// The reference's tree is copied node for node (nodes, the exact copy): its
// boxes are tested on the GPU with the reference's slab arithmetic, so the GPU
// visits exactly the leaves the reference's depth-first traversal would
// reach. Each triangle record keeps its depth-first position in the
// reference's leaf order, the tie-break key.
//
// The culling copy (cull) is for rays whose inverse direction (and its product
// with the origin) is finite and whose origin lies within cull_radius2 of
// cull_center. It is a hierarchy of its own (cull_bvh.h) over the triangles
// that the reference's tree holds, each once, whose boxes are the triangles'
// bounds padded by a relative 2^-16 and by a share of the way that a ray from
// within that ball can have come (2^-16 of the scene's diagonal where the ball
// reaches four diagonals around the scene; less in a smaller one, which scenes
// with fine detail in a large extent get: flatten.cpp choose_region): a ray
// skips a box only if it cannot come within that pad of any triangle inside,
// and for such origins the pad exceeds the float error of the slab test and
// the distance by which a hit that the one-sided Moeller-Trumbore test reports
// can lie off its triangle (up to grazing angles; flatten.cpp gives the
// bounds). So every hit that the reference could report is found, and a hit
// counts if the reference reaches a leaf that holds the triangle: for finite
// inverse directions the reference's slab test is monotone in the box (a box
// inside another gives an interval inside the other's) and its boxes are
// nested, so it reaches a leaf exactly when the leaf's own box passes. Each
// triangle record of the culling copy therefore names its owners, the leaves
// that hold it, in depth-first order; the first one whose box passes the
// reference's test gives the hit's key, and a hit without one is dropped. Long
// lists are trees (Flattener::put_owners): leaf after leaf, a two-triangle
// floor under 64 spheres of 82k triangles (1,737 leaves own it) cost 265 boxes
// per hit and 1,569 in the worst ray.
// Other rays use the exact copy.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "../device_layout.h"
#include "cull_bvh.h"
#include "geom.h"
#include "kdtree.h"

namespace pray_gpu {

struct DeviceImage {
    std::vector<GNode> nodes;   // the exact copy
    std::vector<GNode> cull;    // the culling copy (child indices from its own start); empty: none
    float cull_center[3] = {0.f, 0.f, 0.f};
    float cull_radius2 = -1.f;  // origins within sqrt of this of cull_center use the culling copy
    std::vector<GTri> tris;     // triangles of the culling copy, then leaf references of the exact copy
    uint64_t refs = 0;          // the latter
    uint64_t culled() const { return tris.size() - refs; }
    std::vector<GOwner> owners; // owner lists of triangles with more than one
};

// The child pairs of a culling copy on a 16-bit grid (GPair; pair p holds nodes
// 2p and 2p + 1; pair 0 is unused). Every box is rounded outwards by one to
// two cells: one cell more than the grid needs, for the rounding of the
// distances that the kernels compute from grid steps (slab_grid). leaf_word:
// the device's word of a leaf node. False: the boxes do not fit a grid, or grow
// too much on one.
struct GridImage {
    std::vector<GPair> pairs;
    float org[3] = {0.f, 0.f, 0.f}, scale = 1.f;
};
bool grid_for_device(const std::vector<GNode> &cull, uint32_t (*leaf_word)(const GNode &), GridImage &out);

// bvh: the hierarchy of the culling copy (build_cull_bvh over pre); NULL: none.
void flatten_for_device(const BuiltTree &t, const std::vector<TriPre> &pre, const CullBvh *bvh, DeviceImage &out);

// Structural check of both copies before upload: child pairs and leaf ranges
// in bounds, each node reached once, every triangle reference reached once,
// depth within the kernels' traversal stack (the deepest node's depth goes to
// *max_depth when given).
bool validate_device_image(const DeviceImage &img, std::string &why, int *max_depth = nullptr);

}  // namespace pray_gpu
