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
// threads have been made.
static std::atomic<int> g_left{1 << 30};
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
    if (g_left.fetch_sub(1) <= 0) return EAGAIN;
    return real(t, a, f, arg);
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

int main(int argc, char **argv) {
    const std::string mode = argc > 1 ? argv[1] : "";
    if (mode == "threads") return threads_mode(std::atoi(argv[2]));
    return 2;
}
