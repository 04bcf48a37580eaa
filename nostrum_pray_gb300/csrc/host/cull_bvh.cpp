#include "cull_bvh.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace pray_gpu {

namespace {

constexpr int kBins = 16;
// Costs of one node visit (two boxes) and of one triangle test, relative. A
// visit outweighs a test: a warp walks its lanes' nodes one by one, but
// tests their leaves together.
constexpr double kVisit = 1.5, kTest = 1.0;
constexpr size_t kParallel = 1024;  // subtrees from this size on may get a thread of their own

// x, y, z and an unused lane: one vector register on either host
typedef float V4 __attribute__((vector_size(16)));
typedef int I4 __attribute__((vector_size(16)));
inline V4 vmin(V4 a, V4 b) { return a < b ? a : b; }
inline V4 vmax(V4 a, V4 b) { return a > b ? a : b; }

struct Box {
    V4 lo, hi;
    void clear() {
        lo = V4{INFINITY, INFINITY, INFINITY, INFINITY};
        hi = -lo;
    }
    void add(const Box &b) { lo = vmin(lo, b.lo), hi = vmax(hi, b.hi); }
    double half_area() const {
        const double x = (double)hi[0] - lo[0], y = (double)hi[1] - lo[1], z = (double)hi[2] - lo[2];
        return x * y + y * z + z * x;
    }
};

struct Prim {
    Box box;
    // twice the centre; 0 where the bounds are not finite (such triangles
    // still get a box that every ray enters)
    V4 c;
    uint32_t id;
};

struct Builder {
    std::vector<Prim> prims;
    int leaf_max;
    Threads &threads;
    // node pairs by the position of their split: the subtree over [lo, hi)
    // uses pairs lo .. hi - 2, so parallel subtrees share nothing
    struct Node {
        Box box;
        uint32_t pair, lo, count;  // interior: pair index; leaf: count > 0
    };
    std::vector<Node> root, pairs;

    static int levels(size_t n, int leaf) {  // halvings until at most `leaf` are left
        int d = 0;
        while (n > (size_t)leaf) n = (n + 1) / 2, d++;
        return d;
    }

    void build(Node &node, size_t lo, size_t hi, int depth) {
        const size_t n = hi - lo;
        Box bounds, centres;
        bounds.clear(), centres.clear();
        for (size_t i = lo; i < hi; i++) {
            const Prim &p = prims[i];
            bounds.add(p.box);
            centres.lo = vmin(centres.lo, p.c), centres.hi = vmax(centres.hi, p.c);
        }
        node.box = bounds;
        node.pair = 0, node.lo = (uint32_t)lo, node.count = (uint32_t)n;
        if (n <= 1) return;
        int best_axis = -1, best_bin = 0;
        double best = INFINITY;
        V4 scale = {0.f, 0.f, 0.f, 0.f};
        for (int k = 0; k < 3; k++) {
            const float e = centres.hi[k] - centres.lo[k];
            scale[k] = e > 0.f && std::isfinite(e) ? kBins * 0.9999f / e : 0.f;
        }
        const V4 from = centres.lo, last = V4{1.f, 1.f, 1.f, 1.f} * (float)(kBins - 1);
        auto bins_of = [&](const Prim &p) { return __builtin_convertvector(vmin((p.c - from) * scale, last), I4); };
        const bool halve = depth + levels(n, leaf_max) >= kCullDepth;
        if (!halve) {
            // bins without a triangle are skipped: they change no box and no cost
            Box box[3][kBins];
            uint32_t count[3][kBins], used[3] = {0, 0, 0};
            for (size_t i = lo; i < hi; i++) {
                const Prim &p = prims[i];
                const I4 at = bins_of(p);
                for (int k = 0; k < 3; k++) {
                    const int b = at[k];
                    if (used[k] >> b & 1u) {
                        box[k][b].add(p.box);
                        count[k][b]++;
                    } else {
                        used[k] |= 1u << b;
                        box[k][b] = p.box;
                        count[k][b] = 1;
                    }
                }
            }
            for (int k = 0; k < 3; k++) {
                int bins[kBins], m = 0;
                for (uint32_t u = used[k]; u; u &= u - 1) bins[m++] = __builtin_ctz(u);
                if (m < 2 || scale[k] == 0.f) continue;
                double right[kBins];
                Box acc = box[k][bins[m - 1]];
                for (int q = m - 1; q > 0; q--) {
                    if (q < m - 1) acc.add(box[k][bins[q]]);
                    right[q] = acc.half_area();
                }
                acc = box[k][bins[0]];
                uint32_t c = 0;
                for (int q = 0; q + 1 < m; q++) {
                    if (q) acc.add(box[k][bins[q]]);
                    c += count[k][bins[q]];
                    const double cost = acc.half_area() * c + right[q + 1] * (double)(n - c);
                    if (cost < best) best = cost, best_axis = k, best_bin = bins[q];
                }
            }
        }
        if (n <= (size_t)leaf_max) {
            const double area = bounds.half_area();
            if (best_axis < 0 || !(kVisit * area + kTest * best < kTest * (double)n * area)) return;  // leaf
        }
        size_t mid = lo + n / 2;
        if (best_axis >= 0) {
            mid = std::partition(prims.begin() + lo, prims.begin() + hi,
                                 [&](const Prim &p) { return bins_of(p)[best_axis] <= best_bin; }) -
                  prims.begin();
        } else {
            // equal centres, or no levels to spare: halves along the longest axis
            int axis = 0;
            for (int k = 1; k < 3; k++)
                if (centres.hi[k] - centres.lo[k] > centres.hi[axis] - centres.lo[axis]) axis = k;
            std::nth_element(prims.begin() + lo, prims.begin() + mid, prims.begin() + hi,
                             [&](const Prim &x, const Prim &y) {
                                 const float a = x.c[axis], b = y.c[axis];
                                 return a < b || (a == b && x.id < y.id);
                             });
        }
        const size_t pair = mid - 1;  // one split position each: unique in [lo, hi - 2]
        node.count = 0, node.pair = (uint32_t)pair;
        Node &l = pairs[2 * pair], &r = pairs[2 * pair + 1];
        std::future<void> other;
        if (n >= kParallel) other = threads.start([&, mid] { build(l, lo, mid, depth + 1); });
        if (!other.valid()) build(l, lo, mid, depth + 1);
        build(r, mid, hi, depth + 1);
        if (other.valid()) other.get();
    }

    void emit(const Node &n, uint32_t slot, std::vector<GNode> &out) const {
        GNode g;
        for (int k = 0; k < 3; k++) g.lo[k] = n.box.lo[k], g.hi[k] = n.box.hi[k];
        if (n.count) {
            g.a = n.lo, g.b = kLeafFlag | n.count;
            out[slot] = g;
            return;
        }
        const uint32_t at = (uint32_t)out.size();
        g.a = at, g.b = 0;
        out[slot] = g;
        out.resize(out.size() + 2);
        emit(pairs[2 * (size_t)n.pair], at, out);
        emit(pairs[2 * (size_t)n.pair + 1], at + 1, out);
    }
};

}  // namespace

CullBvh build_cull_bvh(const std::vector<TriPre> &tris, int leaf_max, Threads &threads) {
    CullBvh out;
    out.nodes.assign(2, GNode{});
    const size_t n = tris.size();
    if (n == 0) {
        for (int k = 0; k < 3; k++) out.nodes[0].lo[k] = INFINITY, out.nodes[0].hi[k] = -INFINITY;
        out.nodes[0].b = kLeafFlag;
        return out;
    }
    Builder b{{}, std::min(std::max(1, leaf_max), kCullLeaf), threads, {}, {}};
    b.prims.resize(n);
    auto has_nan = [](const Aabb &t) {
        bool nan = false;
        for (int k = 0; k < 3; k++) nan = nan || std::isnan(t.lo[k]) || std::isnan(t.hi[k]);
        return nan;
    };
    // a triangle with a NaN is hit by no ray (its distance is NaN): it gets a
    // box that is in the way of nothing, another triangle's
    size_t sound = 0;
    while (sound + 1 < n && has_nan(tris[sound].box)) sound++;
    for (size_t i = 0; i < n; i++) {
        Prim &p = b.prims[i];
        const Aabb &t = tris[has_nan(tris[i].box) ? sound : i].box;
        p.id = (uint32_t)i;
        for (int k = 0; k < 3; k++) {
            const bool ok = std::isfinite(t.lo[k]) && std::isfinite(t.hi[k]);
            p.box.lo[k] = ok ? t.lo[k] : -INFINITY, p.box.hi[k] = ok ? t.hi[k] : INFINITY;
            const float c = t.lo[k] + t.hi[k];
            p.c[k] = std::isfinite(c) ? c : 0.f;
        }
    }
    b.root.resize(1);
    b.pairs.resize(2 * std::max<size_t>(n - 1, 1));
    b.build(b.root[0], 0, n, 0);
    out.nodes.reserve(2 * n + 2);
    b.emit(b.root[0], 0, out.nodes);
    out.order.resize(n);
    for (size_t i = 0; i < n; i++) out.order[i] = b.prims[i].id;
    return out;
}

}  // namespace pray_gpu
