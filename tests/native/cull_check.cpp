// Checks of the host side of the culling hierarchy that need no GPU
// (tests/test_culling_cpu.py builds and runs it). Mode by argv[1]; prints one
// line of results, exit status 0 when the mode ran to its end.
#include <pthread.h>
#include <dlfcn.h>

#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>

#include "cull_bvh.h"
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

int main(int argc, char **argv) {
    const std::string mode = argc > 1 ? argv[1] : "";
    if (mode == "threads") return threads_mode(std::atoi(argv[2]));
    if (mode == "budget") return budget_mode(std::atoi(argv[2]));
    return 2;
}
