#include "flatten.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

namespace pray_gpu {

namespace {

constexpr float kPadRel = 1.0f / 65536.0f;
// Every padded box also grows by this fraction of the scene's diagonal D, and
// only rays whose origin lies within kCullReach diagonals of the scene's
// centre use padded boxes (the others take the exact copy). Float errors grow
// with the distance travelled, not with a box's coordinates: for an origin at
// distance R from the centre, each endpoint of a slab test errs by at most
// 3u(R + D) (u = 2^-24), and a hit that Moeller-Trumbore reports can lie off
// its triangle by about u(R + D) / (sin a sin b), a the triangle's smallest
// angle and b the ray's angle to its plane. The pad, 2^8 u D, keeps such hits
// inside their boxes for sin a sin b down to 1/50 at the reach limit (1/170
// for origins inside the scene). The warp-packet walk's FMA form of the slab
// test (p * inv - o * inv) adds at most 1/25 of the pad.
constexpr float kPadScene = 1.0f / 65536.0f;
constexpr float kCullReach = 4.0f;
// Where such pads are large against the triangles, the culling copy serves a
// smaller ball of origins: growth is the mean factor by which the pads grow the
// area of the leaves' boxes inside it. Walks of 300k rays near an 81,920-triangle
// sphere of radius 1 on a two-triangle floor, node pairs / triangles per ray:
// growth 1.04 (half-width 3) 21 / 5, 2.2 (100) 25 / 10, 3.9 (2,000, a ball of
// 2,828) 30 / 16, 8.6 (400, all origins) 41 / 33, 64 (2,000, all origins) 221 /
// 394, where the reference's tree, which the origins outside take, costs 26 /
// 92. Up to kRegionGrowth the wider ball is kept, and always where the
// reference's tree has large leaves (kRegionLeaf: the mean size of the leaf that
// a reference is in), which origins outside the ball would scan.
constexpr double kRegionGrowth = 4.0, kRegionLeaf = 64.0;
constexpr int kRegionSteps = 8;
constexpr size_t kRegionSample = 4096;  // leaves looked at
// Grid pairs are made where rounding to the grid grows the boxes' area by no
// more than this on the average. 300k closest hits / 4 spp of next-event paths
// (1024^2) of that sphere, with the grid against whole nodes, us: growth 1.03
// (half-width 3) 173 to 183 / 2,474 to 2,438, 1.13 (10) 182 to 185 / 2,660 to
// 2,566, 1.25 (20) 199 to 186 / 2,870 to 2,654, 1.85 (100) 330 to 245 / 4,383 to
// 3,359; the 101,156-triangle room, 1.03: 166 to 176 / (16 spp) 34.2 to 37.6 ms.
constexpr double kGridGrowth = 1.1;
constexpr size_t kGridSample = 8192;  // boxes looked at
// Moeller-Trumbore's error in u and v is u(R + D) over the sine of the angle
// between the two edges it works with (ab, ac) and of b, along those edges.
// Where that angle's sine is below kSliver the pad does not cover it: such a
// triangle's bounds grow along its edges by the error at sin b = 1/2, or its
// box is that of the leaves that hold it (hits of one without area can lie
// anywhere on the rays that reach them), whichever is smaller. Triangles per
// ray at 60 cylinders of 64 strips: 2.0, with every sliver boxed as its leaves
// 460 (median tree), 62 (SAH), all of them (one leaf). 200k rays at 3,000 slivers
// of any sine from 1e-9 up: the distances of the reference's tree.
constexpr double kSliver = 1.0 / 50.0, kSliverGrazing = 1.0 / 2.0;
// References of a leaf up to which it stands for the slivers it holds.
constexpr uint32_t kSliverLeaf = 64;
// Most leaves of an owner list that stand without an ancestor before them.
constexpr size_t kOwnerRun = 4;

void grow(GNode &g, const GNode &b) {
    for (int k = 0; k < 3; k++) g.lo[k] = std::min(g.lo[k], b.lo[k]), g.hi[k] = std::max(g.hi[k], b.hi[k]);
}

double half_area(const GNode &g) {
    const double x = (double)g.hi[0] - g.lo[0], y = (double)g.hi[1] - g.lo[1], z = (double)g.hi[2] - g.lo[2];
    return x * y + y * z + z * x;
}

// The origins that the culling copy serves (a ball) and the pads it needs for
// them.
struct Region {
    float c[3], radius;
    float pad_all;  // > 0: the absolute part of every box's pad; else it depends on the box's distance
    // the absolute part of a box's pad
    float absolute(const GNode &a) const {
        if (pad_all > 0.f) return pad_all;
        double far2 = 0.0;  // from c to the box's farthest corner
        for (int k = 0; k < 3; k++) {
            const double d = std::max(std::fabs((double)a.lo[k] - c[k]), std::fabs((double)a.hi[k] - c[k]));
            far2 += d * d;
        }
        return (float)((radius + std::sqrt(far2)) * (kPadScene / (kCullReach + 1.0f)));
    }
    // b = a, padded
    void pad(const GNode &a, GNode &b) const {
        const float all = absolute(a);
        for (int k = 0; k < 3; k++) {
            const float p = (std::fabs(a.lo[k]) + std::fabs(a.hi[k]) + (a.hi[k] - a.lo[k])) * kPadRel + all + 1e-30f;
            b.lo[k] = a.lo[k] - p;
            b.hi[k] = a.hi[k] + p;
        }
    }
};

// The widest region whose pads leave the leaves' boxes near their own size: the
// reach of kCullReach diagonals around the scene, or, where the scene holds
// something fine and small (a mesh on a floor a thousand times its size),
// balls an eighth of that and so on around the middle of its leaves. cull:
// unpadded boxes. shrink: smaller balls are allowed.
Region choose_region(const std::vector<GNode> &cull, const Aabb &root, float diag, bool shrink) {
    Region wide;
    for (int k = 0; k < 3; k++) wide.c[k] = 0.5f * (root.lo[k] + root.hi[k]);
    wide.radius = kCullReach * diag;
    wide.pad_all = diag * kPadScene;
    if (!shrink) return wide;
    std::vector<uint32_t> leaves;  // a sample
    for (size_t i = 0; i < cull.size(); i++)
        if (i != 1 && (cull[i].b & kLeafFlag) && half_area(cull[i]) > 0.0 && std::isfinite(half_area(cull[i])))
            leaves.push_back((uint32_t)i);
    if (leaves.empty()) return wide;
    if (leaves.size() > kRegionSample) {
        const size_t step = leaves.size() / kRegionSample;
        for (size_t i = 0; i < kRegionSample; i++) leaves[i] = leaves[i * step];
        leaves.resize(kRegionSample);
    }
    // mean growth of the area of the leaves whose centre lies in the region
    auto growth = [&](const Region &r) {
        double sum = 0.0;
        size_t n = 0;
        for (uint32_t i : leaves) {
            const GNode &g = cull[i];
            double d2 = 0.0;
            for (int k = 0; k < 3; k++) {
                const double d = 0.5 * ((double)g.lo[k] + g.hi[k]) - r.c[k];
                d2 += d * d;
            }
            if (d2 > (double)r.radius * r.radius) continue;
            GNode p = g;
            r.pad(g, p);
            sum += std::min(half_area(p) / half_area(g), 64.0), n++;
        }
        return n ? sum / n : 0.0;
    };
    if (growth(wide) <= kRegionGrowth) return wide;
    Region r = wide;
    r.pad_all = 0.f;
    for (int k = 0; k < 3; k++) {
        std::vector<float> at;
        for (uint32_t i : leaves) at.push_back(0.5f * (cull[i].lo[k] + cull[i].hi[k]));
        std::nth_element(at.begin(), at.begin() + at.size() / 2, at.end());
        r.c[k] = at[at.size() / 2];
    }
    for (int step = 0; step < kRegionSteps; step++) {
        r.radius /= 8.f;
        if (growth(r) <= kRegionGrowth) break;
    }
    return r;
}

struct Flattener {
    const BuiltTree &t;
    const std::vector<TriPre> &pre;
    DeviceImage &out;
    size_t culled, at = 0;              // records of the culling copy, references placed
    std::vector<uint32_t> first_pos{};  // of each node of the exact copy: its first reference's position

    void put_tri(size_t at, uint32_t tri, uint32_t key, uint32_t owner) {
        const TriPre &p = pre[tri];
        GTri &g = out.tris[at];
        for (int k = 0; k < 3; k++) g.v0[k] = p.a[k], g.e1[k] = p.ab[k], g.e2[k] = p.ac[k];
        std::memcpy(&g.v0[3], &tri, 4);
        std::memcpy(&g.e1[3], &key, 4);
        std::memcpy(&g.e2[3], &owner, 4);
    }

    // Reference node p into slot, its subtree after it; leaves in depth-first
    // order. leaf_of[i] receives the node of the leaf that holds reference i.
    void put(int32_t p, uint32_t slot, std::vector<uint32_t> &leaf_of) {
        const FlatNode &n = t.nodes[p];
        first_pos.resize(out.nodes.size());
        first_pos[slot] = (uint32_t)at;
        GNode g;
        for (int k = 0; k < 3; k++) g.lo[k] = n.box.lo[k], g.hi[k] = n.box.hi[k];
        g.a = 0;
        g.b = 0;
        if (n.left < 0) {
            g.a = (uint32_t)(culled + at);
            g.b = kLeafFlag | n.count;
            for (uint32_t i = n.first; i < n.first + n.count; i++) {
                put_tri(culled + at, t.refs[i], i, kNoOwner);
                leaf_of[i] = slot;
                at++;
            }
            out.nodes[slot] = g;
            return;
        }
        const uint32_t pair = (uint32_t)out.nodes.size();
        out.nodes.resize(out.nodes.size() + 2);
        g.a = pair;
        out.nodes[slot] = g;
        put(n.left, pair, leaf_of);
        put(n.right, pair + 1, leaf_of);
    }

    // The box of triangle tri, held by the leaves of the n references at pos, if
    // it is a sliver.
    bool sliver_box(uint32_t tri, const Region &region, const uint32_t *pos, size_t n,
                    const std::vector<uint32_t> &leaf_of, GNode &box) const {
        const TriPre &p = pre[tri];
        const F3 &a = p.ab, &b = p.ac;
        const double c[3] = {(double)a[1] * b[2] - (double)a[2] * b[1], (double)a[2] * b[0] - (double)a[0] * b[2],
                             (double)a[0] * b[1] - (double)a[1] * b[0]};
        auto len = [](double x, double y, double z) { return std::sqrt(x * x + y * y + z * z); };
        const double area = len(c[0], c[1], c[2]), la = len(a[0], a[1], a[2]), lb = len(b[0], b[1], b[2]);
        // (an edge of no length: the determinant is zero for every ray; not
        // finite: every ray enters its box)
        if (!(area <= kSliver * la * lb) || la == 0.0 || lb == 0.0 || !std::isfinite(la + lb)) return false;
        for (int k = 0; k < 3; k++) box.lo[k] = p.box.lo[k], box.hi[k] = p.box.hi[k];
        const double sine = area / (la * lb);
        double by = region.absolute(box) * kSliver / (kSliverGrazing * sine);
        GNode held;
        for (int k = 0; k < 3; k++) held.lo[k] = INFINITY, held.hi[k] = -INFINITY;
        bool small = n > 0;
        for (size_t i = 0; i < n && small; i++) {
            const GNode &leaf = out.nodes[leaf_of[pos[i]]];
            small = (leaf.b & ~kLeafFlag) <= kSliverLeaf;
            grow(held, leaf);
        }
        if (!small) by = std::min(by, std::max(la, lb));
        for (int k = 0; k < 3; k++) {
            const float e = (float)(by * (std::fabs(a[k]) / la + std::fabs(b[k]) / lb));
            box.lo[k] -= e;
            box.hi[k] += e;
        }
        if (small && !(half_area(box) < half_area(held))) box = held;
        return true;
    }

    // The owner list of a triangle with the references at pos[0, n), all below
    // `node` of the exact copy; its entries are numbered from `list`. Above
    // kOwnerRun leaves their nearest common ancestor stands before them (but
    // for the whole list's, whose box a ray that hits the triangle hardly
    // misses), so that a ray tests the ancestors that it meets instead of every
    // leaf: a large triangle over a fine mesh has thousands.
    void put_owners(const uint32_t *pos, size_t n, uint32_t node, size_t list, const std::vector<uint32_t> &leaf_of,
                    bool whole) {
        size_t left = 0;
        while (n > kOwnerRun && !(out.nodes[node].b & kLeafFlag)) {
            const uint32_t pair = out.nodes[node].a;
            left = std::lower_bound(pos, pos + n, first_pos[pair + 1]) - pos;
            if (left && left < n) break;
            node = left ? pair : pair + 1;
        }
        if (!left || left == n) {
            for (size_t i = 0; i < n; i++) out.owners.push_back(GOwner{leaf_of[pos[i]], pos[i]});
            return;
        }
        const size_t at = out.owners.size();
        if (!whole) out.owners.push_back(GOwner{node, 0});
        const uint32_t pair = out.nodes[node].a;
        put_owners(pos, left, pair, list, leaf_of, false);
        put_owners(pos + left, n - left, pair + 1, list, leaf_of, false);
        if (!whole) out.owners[at].key = kOwnerGroup | (uint32_t)(out.owners.size() - list);
    }
};

}  // namespace

void flatten_for_device(const BuiltTree &t, const std::vector<TriPre> &pre, const CullBvh *bvh, DeviceImage &out) {
    out = DeviceImage{};
    out.nodes.assign(2, GNode{});
    const Aabb &root = t.nodes[0].box;
    double d2 = 0.0;
    for (int k = 0; k < 3; k++) d2 += ((double)root.hi[k] - root.lo[k]) * ((double)root.hi[k] - root.lo[k]);
    const float diag = (float)std::sqrt(d2);
    const bool sized = !t.refs.empty() && std::isfinite(diag);
    out.refs = t.refs.size();
    // (no culling copy where its leaves' words could not hold the records' numbers)
    const bool cull = bvh && sized && cull_records_fit(out.refs, pre.size());
    const size_t culled = cull ? pre.size() : 0;
    out.tris.resize(culled + out.refs);
    Flattener f{t, pre, out, culled};
    std::vector<uint32_t> leaf_of(t.refs.size());
    f.put(0, 0, leaf_of);
    if (!cull) return;
    // each triangle's references, in depth-first order
    std::vector<uint32_t> first(pre.size() + 1, 0);
    for (uint32_t tri : t.refs) first[tri + 1]++;
    for (size_t i = 0; i < pre.size(); i++) first[i + 1] += first[i];
    std::vector<uint32_t> at(first.begin(), first.end() - 1), of(t.refs.size());
    for (uint32_t i = 0; i < (uint32_t)t.refs.size(); i++) of[at[t.refs[i]]++] = i;
    for (size_t i = 0; i < culled; i++) {
        const uint32_t tri = bvh->order[i], a = first[tri], n = first[tri + 1] - a;
        if (n == 1) {
            f.put_tri(i, tri, of[a], leaf_of[of[a]]);
            continue;
        }
        const size_t list = out.owners.size();
        f.put_owners(of.data() + a, n, 0, list, leaf_of, true);
        f.put_tri(i, tri, (uint32_t)list, kOwnerList | (uint32_t)(out.owners.size() - list));
    }
    out.cull = bvh->nodes;
    double scanned = 0.0;
    for (const FlatNode &n : t.nodes)
        if (n.left < 0) scanned += (double)n.count * n.count;
    const Region region = choose_region(out.cull, root, diag, scanned <= kRegionLeaf * out.refs);
    for (int k = 0; k < 3; k++) out.cull_center[k] = region.c[k];
    out.cull_radius2 = region.radius * region.radius;
    // the slivers' boxes; children come after their parents
    std::vector<std::pair<uint32_t, GNode>> thin;  // positions in bvh->order
    for (uint32_t i = 0; i < (uint32_t)bvh->order.size(); i++) {
        const uint32_t tri = bvh->order[i];
        GNode box;
        if (!f.sliver_box(tri, region, of.data() + first[tri], first[tri + 1] - first[tri], leaf_of, box)) continue;
        thin.push_back({i, box});
    }
    if (!thin.empty()) {
        for (size_t slot = out.cull.size(); slot-- > 0;) {
            GNode &g = out.cull[slot];
            if (slot == 1) continue;
            if (!(g.b & kLeafFlag)) {
                grow(g, out.cull[g.a]), grow(g, out.cull[g.a + 1]);
                continue;
            }
            const uint32_t end = g.a + (g.b & ~kLeafFlag);
            for (auto it = std::lower_bound(thin.begin(), thin.end(), g.a,
                                            [](const auto &t, uint32_t at) { return t.first < at; });
                 it != thin.end() && it->first < end; ++it)
                grow(g, it->second);
        }
    }
    for (GNode &g : out.cull) region.pad(g, g);
}

bool grid_for_device(const std::vector<GNode> &cull, uint32_t (*leaf_word)(const GNode &), GridImage &out) {
    out = GridImage{};
    if (cull.size() < 4) return false;  // no interior node
    double lo[3], hi[3], ext = 0.0;
    for (int k = 0; k < 3; k++) lo[k] = cull[0].lo[k], hi[k] = cull[0].hi[k];
    for (size_t i = 2; i < cull.size(); i++)
        for (int k = 0; k < 3; k++)
            lo[k] = std::min(lo[k], (double)cull[i].lo[k]), hi[k] = std::max(hi[k], (double)cull[i].hi[k]);
    for (int k = 0; k < 3; k++) {
        if (!std::isfinite(lo[k]) || !std::isfinite(hi[k])) return false;
        ext = std::max(ext, hi[k] - lo[k]);
    }
    // the smallest power-of-two cell whose 65,536 steps hold every box and two
    // cells around it from a float origin
    int e = 0;
    std::frexp(ext / 65528.0, &e);
    if (!(ext > 0.0)) return false;
    for (;; e++) {
        if (e < -90 || e > 90) return false;
        const double cell = std::ldexp(1.0, e);
        bool fits = true;
        for (int k = 0; k < 3; k++) {
            float o = (float)(lo[k] - 3.0 * cell);
            if ((double)o > lo[k] - 3.0 * cell) o = std::nextafter(o, -INFINITY);
            out.org[k] = o;
            fits = fits && (hi[k] - o) / cell <= 65532.0;
        }
        if (fits) break;
    }
    const double scale = std::ldexp(1.0, -e);
    out.scale = (float)scale;
    auto steps = [&](const GNode &n, uint32_t q[6]) {
        for (int k = 0; k < 3; k++) {
            q[k] = (uint32_t)(std::floor(((double)n.lo[k] - out.org[k]) * scale) - 1.0);
            q[3 + k] = (uint32_t)(std::ceil(((double)n.hi[k] - out.org[k]) * scale) + 1.0);
        }
    };
    // the mean growth of the boxes' area, over a sample
    double growth = 0.0;
    size_t seen = 0;
    for (size_t i = 2; i < cull.size(); i += cull.size() / kGridSample + 1) {
        const double area = half_area(cull[i]);
        if (!(area > 0.0)) continue;
        uint32_t q[6];
        steps(cull[i], q);
        const double x = q[3] - q[0], y = q[4] - q[1], z = q[5] - q[2];
        growth += std::min((x * y + y * z + z * x) / (scale * scale) / area, 64.0), seen++;
    }
    if (seen && growth > kGridGrowth * seen) return false;
    out.pairs.resize(cull.size() / 2);
    for (size_t p = 1; p < out.pairs.size(); p++) {
        GPair &g = out.pairs[p];
        for (int c = 0; c < 2; c++) {
            const GNode &n = cull[2 * p + c];
            uint32_t q[6];
            steps(n, q);
            uint32_t *w = c ? g.q1 : g.q0;
            for (int k = 0; k < 3; k++) w[k] = q[2 * k] | q[2 * k + 1] << 16;
            (c ? g.w1 : g.w0) = (n.b & kLeafFlag) ? leaf_word(n) : n.a / 2;
        }
    }
    return true;
}

namespace {

// nodes' leaves hold triangle records [begin, end).
bool validate_nodes(const std::vector<GNode> &nodes, uint64_t begin, uint64_t end, std::string &why, int &deepest) {
    const uint64_t nn = nodes.size();
    if (nn < 2) {
        why = "device image has no root";
        return false;
    }
    // iterative walk from the root: every child pair and leaf range in
    // bounds, every node reached once, depth within the traversal stack
    std::vector<uint8_t> seen(nn, 0);
    std::vector<std::pair<uint32_t, int>> todo{{0u, 0}};
    seen[0] = 1;
    uint64_t refs = 0;
    while (!todo.empty()) {
        const auto [i, d] = todo.back();
        todo.pop_back();
        if (d > kMaxTraversalDepth) {
            why = "device hierarchy deeper than the traversal stack";
            return false;
        }
        deepest = std::max(deepest, d);
        const GNode &g = nodes[i];
        if (g.b & kLeafFlag) {
            const uint64_t cnt = g.b & ~kLeafFlag;
            if (cnt && (g.a < begin || (uint64_t)g.a + cnt > end)) {
                why = "leaf range out of bounds";
                return false;
            }
            refs += cnt;
            continue;
        }
        if (g.b != 0 || (g.a & 1u) || (uint64_t)g.a + 1 >= nn || g.a < 2) {
            why = "child pair out of bounds";
            return false;
        }
        for (uint32_t c = g.a; c <= g.a + 1; c++) {
            if (seen[c]) {
                why = "node reached twice";
                return false;
            }
            seen[c] = 1;
            todo.push_back({c, d + 1});
        }
    }
    if (refs != end - begin) {
        why = "a node copy does not reach every triangle record once";
        return false;
    }
    return true;
}

}  // namespace

bool validate_device_image(const DeviceImage &img, std::string &why, int *max_depth) {
    int deepest = 0;
    if (!validate_nodes(img.nodes, img.culled(), img.tris.size(), why, deepest)) return false;
    if (!img.cull.empty()) {
        if (!validate_nodes(img.cull, 0, img.culled(), why, deepest)) return false;
        for (uint64_t i = 0; i < img.culled(); i++) {
            uint32_t key, owner;
            std::memcpy(&key, &img.tris[i].e1[3], 4);
            std::memcpy(&owner, &img.tris[i].e2[3], 4);
            const uint64_t n = owner & kOwnerList ? owner & ~kOwnerList : 0;
            bool ok = owner & kOwnerList ? key + n <= img.owners.size() : owner < img.nodes.size();
            for (uint64_t k = 0; ok && k < n; k++) {
                const GOwner &o = img.owners[key + k];
                const uint64_t next = o.key & ~kOwnerGroup;
                ok = o.node < img.nodes.size() && (!(o.key & kOwnerGroup) || (next > k && next <= n));
            }
            if (!ok) {
                why = "owner out of bounds";
                return false;
            }
        }
    }
    if (max_depth) *max_depth = deepest;
    return true;
}

}  // namespace pray_gpu
