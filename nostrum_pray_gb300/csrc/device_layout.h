// Device-resident scene layout (shared by the host flattener and the kernels).
//
// Nodes: 32-byte records, the two children of an interior node stored side by
// side (one 64-byte, 64-byte-aligned pair), so one visit fetches both child
// boxes and tests them before descending (root at index 0, slot 1 unused).
//   interior: a = index of the first child of its pair, b = 0
//   leaf:     a = first triangle reference, b = kLeafFlag | reference count
// In the culling copy on the device, a leaf's a is one word that holds both
// (kCullCountShift), so that a traversal keeps one word per node.
// Every node keeps its own box (tight triangle bounds for the median tree,
// the voxel for the SAH tree) so the kernels apply the reference's slab test
// to exactly the boxes the reference tests.
//
// Triangle records, 48 bytes each:
//   v0 = (a.xyz, triangle id as bits), e1 = (b - a, key), e2 = (c - a, owner)
// First the culling copy's triangles, each once, in its leaf order (first, so
// that its leaves' words number nothing else): with one owner (a leaf of the
// exact copy) owner is that leaf's node and key its position there, with more
// owner is kOwnerList | the entries of its list (GOwner) and key the first
// entry's index. Then the references of the exact copy, one per leaf entry, in
// depth-first leaf order (a triangle in two SAH leaves is stored twice): key is
// the reference's position in this order, which breaks distance ties, owner
// kNoOwner.
// Shading records: per triangle id, normal (w: 1 for emitters) and colour.
#pragma once

#include <cstdint>

namespace pray_gpu {

constexpr uint32_t kLeafFlag = 0x80000000u;
// Device word of a culling leaf: kLeafFlag | (count - 1) << kCullCountShift |
// first record (counts up to 4, records below 2^kCullCountShift; kernels number
// all records in an int).
constexpr int kCullCountShift = 29;
constexpr bool cull_records_fit(uint64_t refs, uint64_t tris) {
    return tris < (1ull << kCullCountShift) && refs + tris < (1ull << 31);
}
constexpr uint32_t kOwnerList = 0x80000000u, kNoOwner = 0x7FFFFFFFu;
constexpr int kMaxTreeDepth = 30;        // deepest reference tree the API accepts
constexpr int kMaxTraversalDepth = 62;   // deepest device hierarchy (reference tree or culling copy)

struct alignas(32) GNode {  // 32-byte aligned: one 256-bit load per node (traverse.cuh ldg_node)
    float lo[3];
    uint32_t a;
    float hi[3];
    uint32_t b;
};
static_assert(sizeof(GNode) == 32, "GNode must be 32 bytes");

struct alignas(16) GTri {
    float v0[4];
    float e1[4];
    float e2[4];
};
static_assert(sizeof(GTri) == 48, "GTri must be 48 bytes");

// An entry of a triangle's owner list. A leaf of the exact copy: its node and
// the reference's position there. Or an ancestor of the entries that follow:
// its node, and kOwnerGroup | the number in the list of the first entry that is
// not below it, to go on from where its box misses.
constexpr uint32_t kOwnerGroup = 0x80000000u;
struct alignas(8) GOwner {
    uint32_t node, key;
};

struct alignas(16) GShade {
    float n[4];
    float c[4];
};

// The two children of an interior node of the culling copy with their boxes on
// a scene-wide grid of 16-bit steps: planes x0 y0 z0 x1 y1 z1 (box min, max),
// two per word, low half first. Ray queries and the wavefront's passes read
// these, half the bytes of two GNodes, where a scene has them. Words as in the culling copy, but an interior child's is the
// index of its own pair.
struct alignas(32) GPair {
    uint32_t q0[3], w0, q1[3], w1;
};

// Launch-time view of a device scene.
struct DevScene {
    const GNode *nodes;  // n_nodes nodes of the exact copy (the reference's tree), then the culling copy
                         // (for finite-direction rays whose origin is within cull_r2 of cull_c), then, from
                         // grid_base on, its child pairs on the grid (GPair)
    const GTri *tris;
    const GOwner *owners;
    const GShade *shade;
    uint32_t n_nodes, n_refs, n_tris;
    float tol;  // absolute distance tolerance for culling boxes behind the origin
    uint32_t depth;  // deepest node level of the hierarchy (root 0): a traversal pushes at most this many nodes
    float cull_c[3], cull_r2;  // centre and squared radius of the region of origins served by the culling copy
    uint32_t grid_base;  // 0: no grid pairs
    float grid_org[3], grid_scale;  // grid origin, 1 / cell (a power of two)
    // emitting triangles (for next-event estimation): geometry as GTri (v0.w
    // = triangle id) and the inclusive prefix sums of their areas
    const GTri *emit_tris;
    const float *emit_cdf;
    uint32_t n_emit;
    float emit_area;
};

}  // namespace pray_gpu
