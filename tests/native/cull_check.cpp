// Checks of the host side of the culling hierarchy that need no GPU
// (tests/test_culling_cpu.py builds and runs it). Mode by argv[1]; prints one
// line of results, exit status 0 when the mode ran to its end.
#include <pthread.h>
#include <dlfcn.h>

#include <algorithm>
#include <atomic>
#include <cerrno>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <utility>
#include <vector>

#include "cull_bvh.h"
#include "flatten.h"
#include "kdtree.h"

using namespace pray_gpu;

// Thread creation as this program's libraries see it: fails once `g_left`
// threads have been made; counts the threads at work.
static std::atomic<int> g_left{1 << 30}, g_running{0}, g_most{0};
struct Started {
    void *(*f)(void *);
    void *arg;
};
static void *counted(void *p) {
    const Started s = *static_cast<Started *>(p);
    delete static_cast<Started *>(p);
    const int n = ++g_running;
    for (int m = g_most; m < n && !g_most.compare_exchange_weak(m, n);) {}
    void *r = s.f(s.arg);
    g_running--;
    return r;
}
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
    if (g_left.fetch_sub(1) <= 0) return EAGAIN;
    auto *s = new Started{f, arg};
    const int e = real(t, a, counted, s);
    if (e) delete s;
    return e;
}

static std::vector<float> soup(size_t n, double spread, unsigned seed) {
    std::mt19937 g(seed);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    std::vector<float> v(9 * n);
    for (size_t i = 0; i < n; i++) {
        const double c[3] = {u(g), u(g), u(g)};
        for (int k = 0; k < 9; k++) v[9 * i + k] = (float)(c[k % 3] + spread * (2 * u(g) - 1));
    }
    return v;
}

// threads <limit>: the hierarchy over 40,000 triangles with 16 threads asked
// for and at most `limit` to be had equals the single-threaded one.
static int threads_mode(int limit) {
    const auto verts = soup(40000, 0.02, 1);
    const auto pre = precompute_triangles(verts.data(), verts.size() / 9, 1);
    const CullBvh a = build_cull_bvh(pre, 4, 1);
    g_left = limit;
    const CullBvh b = build_cull_bvh(pre, 4, 16);
    const bool same = a.order == b.order && a.nodes.size() == b.nodes.size() &&
                      !std::memcmp(a.nodes.data(), b.nodes.data(), a.nodes.size() * sizeof(GNode));
    std::printf("same %d\n", same ? 1 : 0);
    return same ? 0 : 1;
}

// budget <n>: most threads that ran at once, the caller included, while a tree
// and its hierarchy were built on a budget of n as a scene's creation does.
static int budget_mode(int n) {
    const auto verts = soup(200000, 0.01, 2);
    Threads threads(n);
    const auto pre = precompute_triangles(verts.data(), verts.size() / 9, threads);
    TreeOptions opt;
    opt.kind = kTreeSah;
    CullBvh bvh;
    auto cull = threads.start([&] { bvh = build_cull_bvh(pre, 4, threads); });
    const BuiltTree tree = build_tree(pre, opt, threads);
    if (cull.valid()) cull.get();
    else bvh = build_cull_bvh(pre, 4, threads);
    std::printf("most %d nodes %zu %zu\n", 1 + g_most.load(), tree.nodes.size(), bvh.nodes.size());
    return 0;
}

struct Ray {
    float o[3], d[3], inv[3];
};
static Ray ray_to(const double o[3], const double p[3]) {
    Ray r;
    double d[3], l = 0;
    for (int k = 0; k < 3; k++) d[k] = p[k] - o[k], l += d[k] * d[k];
    for (int k = 0; k < 3; k++) r.o[k] = (float)o[k], r.d[k] = (float)(d[k] / std::sqrt(l)), r.inv[k] = 1.0f / r.d[k];
    return r;
}
// the reference's slab test for finite inverses
static bool slab(const GNode &n, const Ray &r) {
    float tn = -3.4e38f, tf = 3.4e38f;
    for (int k = 0; k < 3; k++) {
        const float a = (n.lo[k] - r.o[k]) * r.inv[k], b = (n.hi[k] - r.o[k]) * r.inv[k];
        tn = std::max(tn, std::min(a, b)), tf = std::min(tf, std::max(a, b));
    }
    return tn <= tf;
}
static uint32_t word(float f) {
    uint32_t w;
    std::memcpy(&w, &f, 4);
    return w;
}

// A two-triangle floor of half-width 10 under `n` small triangles in a thin
// layer, the SAH tree at its deepest.
static std::vector<float> floor_scene(size_t n) {
    auto v = soup(n, 0.004, 3);
    for (size_t i = 0; i < v.size(); i++) v[i] = i % 3 == 1 ? v[i] + 0.3f : 20.f * (v[i] - 0.5f);
    const float q[18] = {-10, 0, -10, -10, 0, 10, 10, 0, 10, -10, 0, -10, 10, 0, 10, 10, 0, -10};
    v.insert(v.end(), q, q + 18);
    return v;
}

// owners <n>: over rays from above at the floor, the first owner whose box
// passes, as the kernels walk a record's list, against every leaf that holds
// the triangle; the leaves of the floor's lists, and the boxes tested per ray
// on the average and at most.
static int owners_mode(size_t n) {
    const auto verts = floor_scene(n);
    const auto pre = precompute_triangles(verts.data(), verts.size() / 9, 0);
    TreeOptions opt;
    opt.kind = kTreeSah, opt.sah_ct = 1.f;
    const BuiltTree tree = build_tree(pre, opt);
    const CullBvh bvh = build_cull_bvh(pre, 4, 0);
    DeviceImage img;
    flatten_for_device(tree, pre, &bvh, img);
    std::string why;
    if (!validate_device_image(img, why)) return std::printf("%s\n", why.c_str()), 1;
    std::mt19937 g(5);
    std::uniform_real_distribution<double> u(-10, 10);
    size_t leaves = 0, tests = 0, most = 0, hits = 0, wrong = 0;
    const int kRays = 20000;
    for (uint32_t tri = (uint32_t)n; tri < n + 2; tri++) {
        size_t at = 0;
        while (word(img.tris[at].v0[3]) != tri) at++;
        const uint32_t first = word(img.tris[at].e1[3]), owner = word(img.tris[at].e2[3]), count = owner & 0x7FFFFFFFu;
        if (!(owner & kOwnerList)) return std::printf("no list\n"), 1;
        std::vector<std::pair<uint32_t, uint32_t>> all;  // (position, leaf)
        for (uint32_t i = 0; i < img.nodes.size(); i++) {
            const GNode &l = img.nodes[i];
            if (i == 1 || !(l.b & kLeafFlag)) continue;
            for (uint32_t k = l.a; k < l.a + (l.b & ~kLeafFlag); k++)
                if (word(img.tris[k].v0[3]) == tri) all.push_back({k - (uint32_t)img.culled(), i});
        }
        std::sort(all.begin(), all.end());
        leaves += all.size();
        for (int q = 0; q < kRays; q++) {
            const double o[3] = {u(g), 4.0 + 0.3 * u(g), u(g)}, p[3] = {u(g), 0, u(g)};
            const Ray r = ray_to(o, p);
            uint32_t want = ~0u, got = ~0u;
            for (const auto &[pos, leaf] : all)
                if (slab(img.nodes[leaf], r)) {
                    want = pos;
                    break;
                }
            size_t t = 0;
            for (uint32_t i = 0; i < count && got == ~0u;) {
                uint32_t e[2];
                std::memcpy(e, &img.owners[first + i], 8);
                const bool pass = slab(img.nodes[e[0]], r), group = e[1] >> 31;
                t++;
                if (pass && !group) got = e[1];
                i = !pass && group ? e[1] & 0x7FFFFFFFu : i + 1;
            }
            wrong += got != want, hits += want != ~0u, tests += t, most = std::max(most, t);
        }
    }
    std::printf("leaves %zu wrong %zu hits %zu mean %.1f most %zu\n", leaves, wrong, hits, tests / (2.0 * kRays), most);
    return 0;
}

// Triangles of the culling copy's leaves whose boxes the ray's line passes.
static size_t line_triangles(const DeviceImage &img, const Ray &r) {
    size_t tris = 0;
    std::vector<uint32_t> todo{0};
    while (!todo.empty()) {
        const GNode &n = img.cull[todo.back()];
        todo.pop_back();
        if (!slab(n, r)) continue;
        if (n.b & kLeafFlag) tris += n.b & ~kLeafFlag;
        else todo.push_back(n.a), todo.push_back(n.a + 1);
    }
    return tris;
}

// grid <half-width>: whether the cube's scene as in mixed_mode, on a floor of
// that half-width, gets grid pairs; how much wider than the boxes they are
// (triangles per ray on the grid's boxes over those on the whole nodes').
static int grid_mode(float half) {
    auto verts = soup(30000, 0.01, 4);
    const float h = half, q[18] = {-h, 0, -h, -h, 0, h, h, 0, h, -h, 0, -h, h, 0, h, h, 0, -h};
    verts.insert(verts.end(), q, q + 18);
    const auto pre = precompute_triangles(verts.data(), verts.size() / 9, 0);
    const BuiltTree tree = build_tree(pre, TreeOptions{});
    const CullBvh bvh = build_cull_bvh(pre, 4, 0);
    DeviceImage img;
    flatten_for_device(tree, pre, &bvh, img);
    GridImage grid;
    const bool made = grid_for_device(img.cull, [](const GNode &n) { return n.a; }, grid);
    double ratio = 1.0;
    if (made) {
        DeviceImage wide = img;
        for (size_t p = 1; p < grid.pairs.size(); p++)
            for (int c = 0; c < 2; c++) {
                const uint32_t *w = c ? grid.pairs[p].q1 : grid.pairs[p].q0;
                const uint32_t s[6] = {w[0] & 0xFFFF, w[0] >> 16, w[1] & 0xFFFF, w[1] >> 16, w[2] & 0xFFFF, w[2] >> 16};
                GNode &n = wide.cull[2 * p + c];
                for (int k = 0; k < 3; k++) {
                    n.lo[k] = grid.org[k] + (float)(s[k] / (double)grid.scale);
                    n.hi[k] = grid.org[k] + (float)(s[3 + k] / (double)grid.scale);
                }
            }
        std::mt19937 g(5);
        std::uniform_real_distribution<double> u(-1, 2);
        size_t a = 0, b = 0;
        for (int i = 0; i < 2000; i++) {
            const double o[3] = {u(g), u(g), u(g)}, p[3] = {u(g), u(g), u(g)};
            const Ray r = ray_to(o, p);
            a += line_triangles(img, r), b += line_triangles(wide, r);
        }
        ratio = (double)b / a;
    }
    std::printf("made %d ratio %.3f\n", made ? 1 : 0, ratio);
    return 0;
}

// slivers <strips> <leaf size>: 30 cylinders of thin strips (two triangles
// each); triangles per ray as above.
static int slivers_mode(int strips, int leaf_size) {
    std::mt19937 g(1);
    std::uniform_real_distribution<double> u(-1, 1);
    std::vector<float> verts;
    for (int c = 0; c < 30; c++) {
        const double o[3] = {3 * u(g), 3 * u(g), 3 * u(g)}, radius = 0.3 + 0.2 * u(g), height = 2.5 + 1.5 * u(g);
        for (int i = 0; i < strips; i++) {
            const double a = 2 * M_PI * i / strips, b = 2 * M_PI * (i + 1) / strips;
            auto put = [&](double at, double y) {
                for (double x : {o[0] + radius * std::cos(at), o[1] + y, o[2] + radius * std::sin(at)})
                    verts.push_back((float)x);
            };
            put(a, 0), put(a, height), put(b, 0), put(b, 0), put(a, height), put(b, height);
        }
    }
    const auto pre = precompute_triangles(verts.data(), verts.size() / 9, 0);
    TreeOptions opt;
    opt.leaf_size = leaf_size;
    const BuiltTree tree = build_tree(pre, opt);
    const CullBvh bvh = build_cull_bvh(pre, 4, 0);
    DeviceImage img;
    flatten_for_device(tree, pre, &bvh, img);
    const int kRays = 2000;
    size_t tris = 0;
    for (int i = 0; i < kRays; i++) {
        const double o[3] = {6 * u(g), 6 * u(g), 6 * u(g)}, p[3] = {3 * u(g), 3 * u(g), 3 * u(g)};
        tris += line_triangles(img, ray_to(o, p));
    }
    std::printf("tris %.2f\n", (double)tris / kRays);
    return 0;
}

// mixed <half-width>: 30,000 small triangles in a unit cube on a two-triangle
// floor of that half-width, median tree; leaf triangles per ray whose boxes the ray's line
// passes in the culling copy, for rays between points near the cube, and
// whether their origins are the culling copy's to serve.
static int mixed_mode(float half) {
    auto verts = soup(30000, 0.01, 4);
    const float h = half, q[18] = {-h, 0, -h, -h, 0, h, h, 0, h, -h, 0, -h, h, 0, h, h, 0, -h};
    verts.insert(verts.end(), q, q + 18);
    const auto pre = precompute_triangles(verts.data(), verts.size() / 9, 0);
    TreeOptions opt;
    const BuiltTree tree = build_tree(pre, opt);
    const CullBvh bvh = build_cull_bvh(pre, 4, 0);
    DeviceImage img;
    flatten_for_device(tree, pre, &bvh, img);
    std::mt19937 g(5);
    std::uniform_real_distribution<double> u(-1, 2);
    const int kRays = 2000;
    size_t tris = 0, served = 0;
    for (int i = 0; i < kRays; i++) {
        const double o[3] = {u(g), u(g), u(g)}, p[3] = {u(g), u(g), u(g)};
        const Ray r = ray_to(o, p);
        float d2 = 0;
        for (int k = 0; k < 3; k++) d2 += (r.o[k] - img.cull_center[k]) * (r.o[k] - img.cull_center[k]);
        served += d2 <= img.cull_radius2;
        tris += line_triangles(img, r);
    }
    std::printf("tris %.2f served %.3f\n", (double)tris / kRays, (double)served / kRays);
    return 0;
}

// fits <references> <triangles>: whether such a scene gets a culling copy.
static int fits_mode(uint64_t refs, uint64_t tris) {
    std::printf("fits %d\n", cull_records_fit(refs, tris) ? 1 : 0);
    return 0;
}

int main(int argc, char **argv) {
    const std::string mode = argc > 1 ? argv[1] : "";
    if (mode == "threads") return threads_mode(std::atoi(argv[2]));
    if (mode == "budget") return budget_mode(std::atoi(argv[2]));
    if (mode == "owners") return owners_mode((size_t)std::atoll(argv[2]));
    if (mode == "mixed") return mixed_mode((float)std::atof(argv[2]));
    if (mode == "slivers") return slivers_mode(std::atoi(argv[2]), std::atoi(argv[3]));
    if (mode == "grid") return grid_mode((float)std::atof(argv[2]));
    if (mode == "fits") return fits_mode(std::strtoull(argv[2], nullptr, 0), std::strtoull(argv[3], nullptr, 0));
    return 2;
}
