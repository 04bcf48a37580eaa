// Device-side ray traversal and intersection shared by the tracing kernels.
//
// Every translation unit that includes this file is built with --fmad=false
// and IEEE division / square root, so each float operation rounds as in the
// reference's scalar build compiled without FMA contraction.
//
// Traversal: one ray per thread, iterative, with a short per-thread stack.
// Both children of a node are fetched together and tested; the nearer is
// entered first and the farther pushed. Rays with finite inverse directions
// and origins near the scene walk the culling copy (host/flatten.h): its boxes
// are padded and tested in FMA form (slab_fma, slab_grid), each triangle
// stands there once, and a hit counts if a leaf of the reference's tree that
// holds the triangle passes the reference's infinite-line slab test
// (BoundingBox::intersect, include/geometry.h:151-164; owned). The others walk
// the exact copy, the reference's tree, with that test at every box. Instead of
// the reference's visit-everything depth-first order
// (KDTree::intersectRecursive, src/kd_tree.cpp:237-279), boxes that start
// beyond the best hit found so far are skipped: the result is the
// lexicographic minimum of (distance, depth-first reference position) over
// the references the reference itself tests, which is exactly the triangle
// it returns. The skip bounds keep a relative margin (kPruneRel) and an
// absolute margin (DevScene::tol) so that rounding in a box's entry or exit
// distance never drops a box holding the winning triangle.
#pragma once

#include <cfloat>
#include <cstdint>

#include "device_layout.h"
#include "host/camera.h"

namespace pray_gpu {
namespace dev {

constexpr float kPruneRel = 1.0f + 1.0f / 4096.0f;
constexpr int kStack = 64;
static_assert(kStack > kMaxTraversalDepth, "stack must hold a full root-to-leaf path");

struct RayF {
    float ox, oy, oz;
    float dx, dy, dz;
    float ix, iy, iz;
};

__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }

// Ray ctor of include/geometry.h:82-87: normalise, then 1/direction.
__device__ __forceinline__ RayF make_ray(float ox, float oy, float oz, float dx, float dy, float dz) {
    RayF r;
    r.ox = ox, r.oy = oy, r.oz = oz;
    const float n2 = dx * dx + dy * dy + dz * dz;
    if (n2 > 0) {
        const float inv = 1.0f / sqrtf(n2);
        dx *= inv, dy *= inv, dz *= inv;
    }
    r.dx = dx, r.dy = dy, r.dz = dz;
    r.ix = 1.0f / dx, r.iy = 1.0f / dy, r.iz = 1.0f / dz;
    return r;
}

// Three-input minimum / maximum (one instruction on sm_100 and later). Like
// fminf / fmaxf, a NaN operand is ignored unless all are NaN.
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// BoundingBox::intersect, include/geometry.h:151-164. `finite`: all three
// inverse direction components are finite, so no slab value can be NaN; then
// fminf/fmaxf return the same values as the reference's std::min/std::max
// selects (they can differ only in the sign of a zero, which no comparison
// sees), at one instruction each. Otherwise the select form reproduces the
// reference's NaN behaviour.
__device__ __forceinline__ bool slab(const float4 &lo, const float4 &hi, const RayF &r, bool finite, float &tn,
                                     float &tf) {
    const float t1x = (lo.x - r.ox) * r.ix, t2x = (hi.x - r.ox) * r.ix;
    const float t1y = (lo.y - r.oy) * r.iy, t2y = (hi.y - r.oy) * r.iy;
    const float t1z = (lo.z - r.oz) * r.iz, t2z = (hi.z - r.oz) * r.iz;
    if (finite) {
        // the same values as fmaxf(fmaxf(a, b), fmaxf(c, -FLT_MAX)) and its mirror
        tn = max3f(fminf(t1x, t2x), fminf(t1y, t2y), fmaxf(fminf(t1z, t2z), -FLT_MAX));
        tf = min3f(fmaxf(t1x, t2x), fmaxf(t1y, t2y), fminf(fmaxf(t1z, t2z), FLT_MAX));
    } else {
        tn = smax(smax(smin(t1x, t2x), smin(t1y, t2y)), smax(smin(t1z, t2z), -FLT_MAX));
        tf = smin(smin(smax(t1x, t2x), smax(t1y, t2y)), smin(smax(t1z, t2z), FLT_MAX));
    }
    return tn <= tf;
}

__device__ __forceinline__ bool slab(const float4 &lo, const float4 &hi, const RayF &r, float &tn, float &tf) {
    return slab(lo, hi, r, false, tn, tf);
}

// The slab test on the culling copy's padded boxes as one FMA per plane:
// (p - o) * inv computed as p * inv + (-o * inv), with no = -o * inv rounded
// once per ray (finite: the caller checks). Its error against the exact
// plane distance is below 2^-24 (2 |o| + |p|) |inv| per axis. The padding
// of a culling box moves each plane by at least 2^-16 (|p| + D) (D the
// scene's diagonal) and culling origins lie within 4 D of the scene's
// centre, so |o| < |p| + 4.5 D and the error is below 1/25 of the pad, on
// entry and exit alike: the pad still holds the triangle hits it was sized
// for (host/flatten.cpp), so no box that the exact ray crosses around a hit
// fails the test or the pruning bound.
//
// Entry and exit take the three-input min / max and drop the reference's clamps to
// -FLT_MAX / FLT_MAX: with a finite inverse direction and finite o * inv no
// plane distance of a finite box is NaN, so the clamps change only an
// infinite entry or exit into FLT_MAX, which no comparison here sees. Boxes of
// empty leaves (infinite or NaN coordinates, no triangles) may then fail where
// they passed before, which drops no triangle.
__device__ __forceinline__ bool slab_fma(const float4 &lo, const float4 &hi, const RayF &r, float nox, float noy,
                                         float noz, float &tn, float &tf) {
    const float t1x = fmaf(lo.x, r.ix, nox), t2x = fmaf(hi.x, r.ix, nox);
    const float t1y = fmaf(lo.y, r.iy, noy), t2y = fmaf(hi.y, r.iy, noy);
    const float t1z = fmaf(lo.z, r.iz, noz), t2z = fmaf(hi.z, r.iz, noz);
    tn = max3f(fminf(t1x, t2x), fminf(t1y, t2y), fminf(t1z, t2z));
    tf = min3f(fmaxf(t1x, t2x), fmaxf(t1y, t2y), fmaxf(t1z, t2z));
    return tn <= tf;
}

// The same on a grid box (GPair), in units of the grid's cell: a 16-bit step q
// becomes the float 2^23 + q by a byte permute, and the distance of its plane
// is (2^23 + q) * inv + no with no = (org - o) / cell * inv - 2^23 * inv, so a
// plane costs a permute and an FMA. Error, in cells: 0.5 from the rounding of
// no (magnitude about 2^23 inv), 0.15 from (org - o) / cell * inv and the
// FMA's own rounding (origins lie within 10 extents of the grid's origin, an
// extent is at most 2^16 cells): below the one cell that each box was widened
// for it (host/flatten.h).
__device__ __forceinline__ float grid_lo(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7610)); }
__device__ __forceinline__ float grid_hi(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7632)); }
__device__ __forceinline__ void slab_grid(float q0, float q1, float q2, const RayF &r, float nox, float noy, float noz,
                                          float &tn, float &tf) {
    const uint32_t a = __float_as_uint(q0), b = __float_as_uint(q1), c = __float_as_uint(q2);
    const float t1x = fmaf(grid_lo(a), r.ix, nox), t1y = fmaf(grid_hi(a), r.iy, noy);
    const float t1z = fmaf(grid_lo(b), r.iz, noz), t2x = fmaf(grid_hi(b), r.ix, nox);
    const float t2y = fmaf(grid_lo(c), r.iy, noy), t2z = fmaf(grid_hi(c), r.iz, noz);
    tn = max3f(fminf(t1x, t2x), fminf(t1y, t2y), fminf(t1z, t2z));
    tf = min3f(fmaxf(t1x, t2x), fmaxf(t1y, t2y), fmaxf(t1z, t2z));
}

// One-sided Moeller-Trumbore, include/geometry.h:242-262, with the det
// threshold as a parameter (the reference's EPSILON is 1e-4).
__device__ __forceinline__ bool intersect_tri(const float4 &v0, const float4 &e1, const float4 &e2, const RayF &r,
                                              float eps, float &t) {
    const float px = r.dy * e2.z - r.dz * e2.y;
    const float py = r.dz * e2.x - r.dx * e2.z;
    const float pz = r.dx * e2.y - r.dy * e2.x;
    const float det = e1.x * px + e1.y * py + e1.z * pz;
    if (det < eps) return false;
    const float tx = r.ox - v0.x, ty = r.oy - v0.y, tz = r.oz - v0.z;
    const float un = tx * px + ty * py + tz * pz;
    // Early out before the division, only where the reference's
    // u = un * (1 / det) is certainly < 0 or > 1: un below -2^-125.6 * det
    // keeps the product a negative normal number; un above det * (1 + 2^-20)
    // keeps it above 1 whatever the two roundings.
    if (un < -(det * 2.4e-38f) || un > det * 1.00000095367431640625f) return false;
    const float inv = 1.0f / det;
    const float u = un * inv;
    if (u < 0.f || u > 1.f) return false;
    const float qx = ty * e1.z - tz * e1.y;
    const float qy = tz * e1.x - tx * e1.z;
    const float qz = tx * e1.y - ty * e1.x;
    const float v = (r.dx * qx + r.dy * qy + r.dz * qz) * inv;
    if (v < 0.f || u + v > 1.f) return false;
    t = (e2.x * qx + e2.y * qy + e2.z * qz) * inv;
    return true;
}

__device__ __forceinline__ float4 ldg4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }

// Whether the reference reports hits of a triangle record of the culling copy
// on this ray, and with which key: it holds the triangle in the leaves that
// own it, in depth-first order, and reaches one of them exactly when its own
// box passes the reference's slab test (host/flatten.h). In a list the leaves
// below an ancestor whose box misses are passed over (boxes are nested).
// References of the exact copy have no owner: the walk came through their
// leaf. e1w, e2w: the record's key and owner words.
__device__ __forceinline__ bool owned(const DevScene &s, const RayF &r, float e1w, float e2w, uint32_t &key);

// One node (box lo + payload a, box hi + payload b) in one 256-bit read-only
// load: nodes are 32-byte aligned, so a lane's node is one 32-byte sector and
// one load instruction instead of two 16-byte ones (half the L1 wavefronts
// of the incoherent per-lane walks, half the load instructions of the packet
// walk).
__device__ __forceinline__ void ldg_node(const GNode *n, float4 &lo, float4 &hi) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w), "=f"(hi.x), "=f"(hi.y), "=f"(hi.z), "=f"(hi.w)
        : "l"(n));
}

__device__ __forceinline__ bool owned(const DevScene &s, const RayF &r, float e1w, float e2w, uint32_t &key) {
    key = __float_as_uint(e1w);
    const uint32_t owner = __float_as_uint(e2w);
    if (owner == kNoOwner) return true;
    const bool list = owner & kOwnerList;
    const uint32_t n = list ? owner & ~kOwnerList : 1u, first = key;
    for (uint32_t i = 0; i < n;) {
        uint32_t node = owner;
        if (list) {
            const uint2 o = __ldg(reinterpret_cast<const uint2 *>(s.owners + first + i));
            node = o.x, key = o.y;
        }
        float4 lo, hi;
        ldg_node(s.nodes + node, lo, hi);
        float tn, tf;
        const bool pass = slab(lo, hi, r, true, tn, tf), group = key & kOwnerGroup;
        if (pass && !group) return true;
        i = group && !pass ? key & ~kOwnerGroup : i + 1;
    }
    return false;
}

// Closest hit (kAny = false): returns the reference position of the winning
// triangle or -1, and its distance in t.
// Any hit (kAny = true): returns >= 0 as soon as a triangle with t > 0 and
// t * t < d2 is found (the occlusion test of src/pray.cpp:42).
// Fetch counts of one traversal (only maintained when kCount is set).
struct FetchCount {
    uint32_t pairs = 0, tris = 0;
};

// Warp-collective traversal: every lane of the warp must call it together
// (inactive lanes pass valid = false). Structure after Aila & Laine,
// "Understanding the Efficiency of Ray Traversal on GPUs" (HPG 2009): the
// warp first walks interior nodes until every lane holds a leaf ("postponing"
// the first leaf it meets and speculatively continuing), then intersects the
// postponed leaves together, so lanes do the same kind of work at the same
// time.
//
// The per-lane state lives in Trav, so that a kernel can also run the
// traversal round by round and hand a lane whose ray is done a new ray
// (dynamic fetch): trav_start tests the root, trav_round runs one interior
// phase and one leaf phase for the whole warp, and a lane is done when
// active() turns false.
//
// Closest hit: best = index of the winning triangle record or -1, its
// distance in best_t. Any hit: best >= 0 once a triangle with t > 0 and
// t * t < d2 is found (the occlusion test of src/pray.cpp:42). A traversal
// looks for one or the other for the whole warp.
enum TravMode { kClosest = 0, kAnyHit = 1 };

struct Trav {
    // the current node and the postponed leaf, one word each: an interior
    // node's first child, or a leaf (kLeafFlag; culling copy: count and first
    // record, exact copy: its node)
    uint32_t w, lw;
    uint32_t node_off;  // 0: the exact copy, else the culling copy's nodes or (kGrid) its grid pairs (finite
                        // inverse direction, near origin); kGrid: kLeafFlag | the culling copy's nodes, for the
                        // subtraction form
    float cur_tn, leaf_tn, limit, back;  // grid pairs: in cells
    float best_t;
    float nox, noy, noz;  // culling copy: -origin / direction (slab_fma), or slab_grid's
    int best, sp;
    uint32_t best_key;
    bool have_node, have_leaf, finite;
    __device__ __forceinline__ bool active() const { return have_node || have_leaf; }
    __device__ __forceinline__ bool on_leaf() const { return have_node && (w & kLeafFlag); }
};

// The traversal stack of one lane (kept apart from Trav so that the scalar
// state stays in registers): a node's word and its entry distance, one 8-byte
// local access per push or pop.
template <int kStackN>
struct TravStack {
    uint2 e[kStackN];
};

// The next stacked node that can still hold a closer hit.
template <int kStackN>
__device__ __forceinline__ void pop_node(Trav &T, const TravStack<kStackN> &S) {
    while (T.sp > 0) {
        const uint2 e = S.e[--T.sp];
        T.cur_tn = __uint_as_float(e.y);
        if (T.cur_tn <= T.limit) {
            T.w = e.x;
            return;
        }
    }
    T.have_node = false;
}

// Triangle records of a leaf word.
__device__ __forceinline__ void leaf_range(const DevScene &s, uint32_t node_off, uint32_t w, uint32_t &first,
                                           uint32_t &end) {
    if (node_off) {
        first = w & ((1u << kCullCountShift) - 1u);
        end = first + ((w >> kCullCountShift) & 3u) + 1u;
    } else {
        const GNode *n = s.nodes + (w & ~kLeafFlag);
        first = __ldg(&n->a);
        end = first + (__ldg(&n->b) & ~kLeafFlag);
    }
}

// Whether the walk tests boxes in FMA form (culling copy; kGrid: grid pairs).
template <int kMode, bool kGrid>
__device__ __forceinline__ bool fast_boxes(const DevScene &s, const Trav &T) {
    if (!kGrid) return T.node_off != 0u;
    return kMode == kClosest ? (int)T.node_off > 0 : T.node_off == s.grid_base;
}

// kGrid (scenes with grid pairs): the culling copy's boxes come from its grid
// pairs: one 32-byte load per pair instead of two, for twelve byte permutes
// more. The divergent walks of ray queries and of the wavefront's extension and
// occlusion passes, which whole nodes bind to L1 throughput (83 to 89 % of its
// peak under ncu), gain: room 1024^2 at 16 spp 37.43 -> 34.00 ms, 300k closest
// hits 178 -> 168 us, 100k occlusion rays 105 -> 98 us. The others are bound by
// instruction issue or registers
// and lose (per-pixel paths of 512^2 at 1 spp 832 -> 950 us, 12 scenes 6.18 ->
// 6.44 ms) and keep whole nodes.
template <int kMode, bool kGrid>
__device__ __forceinline__ void trav_start(const DevScene &s, const RayF &r, float d2, bool valid, Trav &T) {
    T.best_t = FLT_MAX;
    T.best = -1;
    T.best_key = 0xFFFFFFFFu;
    T.limit = kMode == kAnyHit ? sqrtf(d2) * kPruneRel : FLT_MAX;
    T.back = -s.tol;
    T.w = T.lw = 0;
    T.cur_tn = T.leaf_tn = 0.f;
    T.have_node = T.have_leaf = false;
    T.sp = 0;
    if (!kGrid) {
        T.finite = isfinite(r.ix) && isfinite(r.iy) && isfinite(r.iz);
        T.nox = -(r.ox * r.ix), T.noy = -(r.oy * r.iy), T.noz = -(r.oz * r.iz);
    }
    const float cx = r.ox - s.cull_c[0], cy = r.oy - s.cull_c[1], cz = r.oz - s.cull_c[2];
    if (kGrid) {
        // 2^23 inverses, and 2^20 cells of inverses, stay finite; larger ones
        // walk the culling copy's nodes in the subtraction form (100k rays in
        // the room with one inverse of 1e33: 209 us, on the exact copy 1,296)
        constexpr float kMaxInv = 1e30f;
        const bool near = cx * cx + cy * cy + cz * cz <= s.cull_r2;
        const bool grid = near && fabsf(r.ix) < kMaxInv && fabsf(r.iy) < kMaxInv && fabsf(r.iz) < kMaxInv;
        T.finite = grid || (isfinite(r.ix) && isfinite(r.iy) && isfinite(r.iz));
        T.node_off = grid ? s.grid_base : near && T.finite ? s.n_nodes | (kMode == kClosest ? kLeafFlag : 0u) : 0u;
    } else {
        T.node_off = (T.finite && isfinite(T.nox) && isfinite(T.noy) && isfinite(T.noz) &&
                      cx * cx + cy * cy + cz * cz <= s.cull_r2)
                         ? s.n_nodes
                         : 0u;
    }
    if (valid) {
        float tn, tf;
        const GNode *root = s.nodes + (T.node_off ? s.n_nodes : 0u);
        float4 rlo, rhi;
        ldg_node(root, rlo, rhi);
        if (slab(rlo, rhi, r, tn, tf)) {
            T.w = __float_as_uint(rlo.w);
            if (!T.node_off && (__float_as_uint(rhi.w) & kLeafFlag)) T.w = kLeafFlag;  // (node 0)
            T.cur_tn = tn;
            T.have_node = true;
            if (kGrid && fast_boxes<kMode, kGrid>(s, T)) {
                if (!(T.w & kLeafFlag)) T.w /= 2;
                T.cur_tn *= s.grid_scale, T.limit *= s.grid_scale, T.back *= s.grid_scale;
                constexpr float kBias = 8388608.f;
                T.nox = fmaf(-kBias, r.ix, (s.grid_org[0] - r.ox) * s.grid_scale * r.ix);
                T.noy = fmaf(-kBias, r.iy, (s.grid_org[1] - r.oy) * s.grid_scale * r.iy);
                T.noz = fmaf(-kBias, r.iz, (s.grid_org[2] - r.oz) * s.grid_scale * r.iz);
            }
        }
    }
}

template <int kMode, bool kGrid, bool kCount, int kStackN>
__device__ __forceinline__ void trav_round(const DevScene &s, const RayF &r, float eps, float d2, Trav &T,
                                           TravStack<kStackN> &S, FetchCount *fc) {
    static_assert(kStackN >= 2 && kStackN <= kStack, "stack entries");
    constexpr unsigned kFull = 0xFFFFFFFFu;
    // 1. interior nodes, until every lane has found a leaf
    while (true) {
        const bool interior = T.have_node && !(T.w & kLeafFlag);
        if (!__any_sync(kFull, interior && !T.have_leaf)) break;
        if (interior) {
            if (kCount) fc->pairs++;
            const GNode *c = s.nodes + (kGrid && kMode == kClosest ? T.w + (T.node_off & ~kLeafFlag) : T.w + T.node_off);
            float4 l0, h0, l1, h1;
            ldg_node(c, l0, h0);
            if (!kGrid) ldg_node(c + 1, l1, h1);
            uint32_t w0 = __float_as_uint(l0.w), w1 = __float_as_uint(kGrid ? h0.w : l1.w);
            float tn0, tf0, tn1, tf1;
            bool v0, v1;
            // entered: tn <= tf, not beyond the best hit, not behind the origin
            if (fast_boxes<kMode, kGrid>(s, T)) {
                if (kGrid) {
                    slab_grid(l0.x, l0.y, l0.z, r, T.nox, T.noy, T.noz, tn0, tf0);
                    slab_grid(h0.x, h0.y, h0.z, r, T.nox, T.noy, T.noz, tn1, tf1);
                } else {
                    slab_fma(l0, h0, r, T.nox, T.noy, T.noz, tn0, tf0);
                    slab_fma(l1, h1, r, T.nox, T.noy, T.noz, tn1, tf1);
                }
                tn0 = fmaxf(tn0, T.back), tn1 = fmaxf(tn1, T.back);
                v0 = tn0 <= fminf(tf0, T.limit), v1 = tn1 <= fminf(tf1, T.limit);
            } else {
                if (kGrid) {
                    ldg_node(c + 1, l1, h1);
                    w1 = __float_as_uint(l1.w);
                }
                v0 = slab(l0, h0, r, T.finite, tn0, tf0) && tn0 <= T.limit && tf0 >= T.back;
                v1 = slab(l1, h1, r, T.finite, tn1, tf1) && tn1 <= T.limit && tf1 >= T.back;
                if (!kGrid || !T.node_off) {
                    if (__float_as_uint(h0.w) & kLeafFlag) w0 = kLeafFlag | T.w;
                    if (__float_as_uint(h1.w) & kLeafFlag) w1 = kLeafFlag | (T.w + 1);
                }
            }
            if (v0 && v1) {
                const bool first0 = tn0 <= tn1;
                S.e[T.sp++] = make_uint2(first0 ? w1 : w0, __float_as_uint(first0 ? tn1 : tn0));
                T.w = first0 ? w0 : w1;
                T.cur_tn = first0 ? tn0 : tn1;
            } else if (v0 || v1) {
                T.w = v0 ? w0 : w1;
                T.cur_tn = v0 ? tn0 : tn1;
            } else {
                pop_node(T, S);
            }
            if (T.on_leaf() && !T.have_leaf) {
                // first leaf: postpone it and keep walking
                T.lw = T.w, T.leaf_tn = T.cur_tn;
                T.have_leaf = true;
                pop_node(T, S);
            }
        }
    }
    // 2. leaves: the postponed one, then any leaf the walk stopped on
    while (true) {
        const bool work = T.have_leaf || T.on_leaf();
        if (!__any_sync(kFull, work)) break;
        if (work) {
            uint32_t fw;
            float ftn;
            if (T.have_leaf) {
                fw = T.lw, ftn = T.leaf_tn;
                T.have_leaf = false;
            } else {
                fw = T.w, ftn = T.cur_tn;
                pop_node(T, S);
            }
            if (ftn <= T.limit) {
                uint32_t fa, end;
                leaf_range(s, T.node_off, fw, fa, end);
                for (uint32_t i = fa; i < end; i++) {
                    if (kCount) fc->tris++;
                    const GTri *Tr = s.tris + i;
                    const float4 v0 = ldg4(Tr->v0), e1 = ldg4(Tr->e1), e2 = ldg4(Tr->e2);
                    float t;
                    if (intersect_tri(v0, e1, e2, r, eps, t) && t > 0) {
                        uint32_t key;
                        if (kMode == kAnyHit) {
                            if (d2 > t * t && owned(s, r, e1.w, e2.w, key)) {
                                T.best = (int)i;
                                T.have_node = T.have_leaf = false;
                                T.sp = 0;
                                break;
                            }
                        } else if (t < T.best_t || (T.best >= 0 && t == T.best_t)) {
                            // key: depth-first position in the reference's leaf order
                            if (owned(s, r, e1.w, e2.w, key) && (t < T.best_t || key < T.best_key)) {
                                T.best_t = t;
                                T.best = (int)i;
                                T.best_key = key;
                                T.limit = t * kPruneRel;
                                if (kGrid && fast_boxes<kMode, kGrid>(s, T)) T.limit *= s.grid_scale;
                            }
                        }
                    }
                }
            }
        }
    }
}

template <bool kAny, bool kCount = false, int kStackN = kStack, bool kGrid = false>
__device__ __forceinline__ int traverse(const DevScene &s, const RayF &r, float eps, float d2, bool valid,
                                        float &best_t, FetchCount *fc = nullptr) {
    constexpr int kMode = kAny ? kAnyHit : kClosest;
    Trav T;
    TravStack<kStackN> S;
    trav_start<kMode, kGrid>(s, r, d2, valid, T);
    while (__any_sync(0xFFFFFFFFu, T.active())) trav_round<kMode, kGrid, kCount>(s, r, eps, d2, T, S, fc);
    best_t = T.best_t;
    return T.best;
}

// Warp-packet traversal for coherent rays (the primary and occlusion rays of
// a pixel tile), after the packet traversals of Wald et al. (EG 2001) and
// Garanzha & Loop (2010): the warp walks one node sequence of the culling
// copy with a mask of the lanes whose own box tests passed, so node and
// triangle loads are warp-uniform (one broadcast each) and the traversal
// stack is one shared stack per warp (`stk`: 2 x kStackN words of shared
// memory: node word, lane mask) instead of one per lane. Every lane still
// applies its own slab test (with its own pruning bound) to every box on its
// way and its own triangle test to every reference of the leaves it reaches,
// so it returns the same lexicographic minimum as traverse(); only the order
// of visits differs (the warp enters first the child that is nearer for most
// of the lanes entering both), and a lane whose bound shrank after a node was
// pushed still visits it (a popped node's box is not at hand: only its word is
// on the stack). Box tests run in FMA
// form (slab_fma). Only for warps whose valid lanes all use the culling
// copy.
template <bool kAny, bool kCount, int kStackN>
__device__ __forceinline__ int traverse_packet(const DevScene &s, const RayF &r, float eps, float d2, bool valid,
                                               float &best_t, uint32_t *stk, FetchCount *fc) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    const GNode *nodes = s.nodes + s.n_nodes;
    const float nox = -(r.ox * r.ix), noy = -(r.oy * r.iy), noz = -(r.oz * r.iz);
    float limit = kAny ? sqrtf(d2) * kPruneRel : FLT_MAX;
    const float back = -s.tol;
    best_t = FLT_MAX;
    int best = -1;
    uint32_t best_key = 0xFFFFFFFFu;
    uint32_t w;
    unsigned mask;
    {
        float4 lo, hi;
        ldg_node(nodes, lo, hi);
        float tn, tf;
        mask = __ballot_sync(kFull, valid && slab_fma(lo, hi, r, nox, noy, noz, tn, tf));
        w = __float_as_uint(lo.w);
    }
    int sp = 0;
    while (mask) {
        const bool in = (mask >> lane) & 1u;
        if (!(w & kLeafFlag)) {
            const GNode *c = nodes + w;
            float4 l0, h0, l1, h1;
            ldg_node(c, l0, h0);
            ldg_node(c + 1, l1, h1);
            if (kCount && in) fc->pairs++;
            float tn0, tf0, tn1, tf1;
            slab_fma(l0, h0, r, nox, noy, noz, tn0, tf0);
            slab_fma(l1, h1, r, nox, noy, noz, tn1, tf1);
            const bool v0 = in && fmaxf(tn0, back) <= fminf(tf0, limit);
            const bool v1 = in && fmaxf(tn1, back) <= fminf(tf1, limit);
            const unsigned m0 = __ballot_sync(kFull, v0), m1 = __ballot_sync(kFull, v1);
            if (m0 && m1) {
                const unsigned both = m0 & m1;
                const unsigned near0 = __ballot_sync(kFull, v0 && v1 && tn0 <= tn1);
                const bool go0 = both ? 2 * __popc(near0) >= __popc(both) : __popc(m0) >= __popc(m1);
                if (lane == 0) {
                    stk[sp] = __float_as_uint(go0 ? l1.w : l0.w);
                    stk[kStackN + sp] = go0 ? m1 : m0;
                }
                sp++;
                w = __float_as_uint(go0 ? l0.w : l1.w);
                mask = go0 ? m0 : m1;
                continue;
            }
            if (m0 | m1) {
                w = __float_as_uint(m0 ? l0.w : l1.w);
                mask = m0 | m1;
                continue;
            }
        } else {
            // the lanes in the mask test the leaf's references
            bool open = in;
            uint32_t first, end;
            leaf_range(s, s.n_nodes, w, first, end);
            for (uint32_t i = first; i < end; i++) {
                const GTri *Tr = s.tris + i;
                const float4 v0 = ldg4(Tr->v0), e1 = ldg4(Tr->e1), e2 = ldg4(Tr->e2);
                if (open) {
                    if (kCount) fc->tris++;
                    float t;
                    if (intersect_tri(v0, e1, e2, r, eps, t) && t > 0) {
                        uint32_t key;
                        if (kAny) {
                            if (d2 > t * t && owned(s, r, e1.w, e2.w, key)) {
                                best = (int)i;
                                open = false;
                            }
                        } else if (t < best_t || (best >= 0 && t == best_t)) {
                            if (owned(s, r, e1.w, e2.w, key) && (t < best_t || key < best_key)) {
                                best_t = t;
                                best = (int)i;
                                best_key = key;
                                limit = t * kPruneRel;
                            }
                        }
                    }
                }
                if (kAny && !__any_sync(kFull, open)) break;
            }
        }
        // next node: the top of the stack, without the lanes already done
        const unsigned done = kAny ? __ballot_sync(kFull, best >= 0) : 0u;
        mask = 0;
        __syncwarp();
        while (sp > 0 && !mask) {
            sp--;
            w = stk[sp];
            mask = stk[kStackN + sp] & ~done;
        }
        __syncwarp();
    }
    return best;
}

// traverse_packet where every valid lane of the warp uses the culling copy
// (and has a finite o * inv on every axis), else traverse(); all lanes of
// the warp call it together.
template <bool kAny, bool kCount, int kStackN>
__device__ __forceinline__ int traverse_coherent(const DevScene &s, const RayF &r, float eps, float d2, bool valid,
                                                 float &best_t, uint32_t *stk, FetchCount *fc = nullptr) {
    // the packet's FMA slab test also needs o * inv finite
    const bool finite = isfinite(r.ix) && isfinite(r.iy) && isfinite(r.iz) && isfinite(r.ox * r.ix) &&
                        isfinite(r.oy * r.iy) && isfinite(r.oz * r.iz);
    const float cx = r.ox - s.cull_c[0], cy = r.oy - s.cull_c[1], cz = r.oz - s.cull_c[2];
    const bool cull = finite && cx * cx + cy * cy + cz * cz <= s.cull_r2;
    if (__all_sync(0xFFFFFFFFu, !valid || cull))
        return traverse_packet<kAny, kCount, kStackN>(s, r, eps, d2, valid, best_t, stk, fc);
    return traverse<kAny, kCount, kStackN>(s, r, eps, d2, valid, best_t, fc);
}

// Primary ray of pixel (px, py), src/scene_preprocessor.cpp:124-134.
__device__ __forceinline__ RayF primary_ray(const CameraConsts &c, uint32_t px, uint32_t py) {
    const float x = (2 * (((float)px + 0.5f) * c.inv_w) - 1) * c.angle;
    const float y = (1 - 2 * (((float)py + 0.5f) * c.inv_h)) * c.angle / c.aspect;
    const float dx = x * c.m[0][0] + y * c.m[1][0] + c.m[2][0];
    const float dy = x * c.m[0][1] + y * c.m[1][1] + c.m[2][1];
    const float dz = x * c.m[0][2] + y * c.m[1][2] + c.m[2][2];
    return make_ray(c.pos[0], c.pos[1], c.pos[2], dx, dy, dz);
}

// static_cast<uint8_t>(v * 255 + 0.5) on the reference's targets: truncate to
// int, keep the low byte.
__device__ __forceinline__ uint32_t quantise(float v) { return (uint32_t)(int32_t)(v * 255.f + 0.5f) & 0xFFu; }

// Pixel index of thread i: warps cover kWarpTileW x kWarpTileH pixel tiles,
// tiles row-major.
constexpr uint32_t kWarpTileW = 8, kWarpTileH = 4;
static_assert(kWarpTileW * kWarpTileH == 32, "a warp tile holds 32 pixels");

__host__ __device__ __forceinline__ uint64_t warp_tiles(uint32_t w, uint32_t h) {
    return (uint64_t)((w + kWarpTileW - 1) / kWarpTileW) * ((h + kWarpTileH - 1) / kWarpTileH);
}

__device__ __forceinline__ bool pixel_of(uint64_t i, uint32_t w, uint32_t h, uint32_t &px, uint32_t &py) {
    const uint32_t tiles_x = (w + kWarpTileW - 1) / kWarpTileW;
    const uint64_t tile = i >> 5;
    const uint32_t lane = (uint32_t)i & 31u;
    px = (uint32_t)(tile % tiles_x) * kWarpTileW + lane % kWarpTileW;
    py = (uint32_t)(tile / tiles_x) * kWarpTileH + lane / kWarpTileW;
    return px < w && py < h;
}

}  // namespace dev
}  // namespace pray_gpu
