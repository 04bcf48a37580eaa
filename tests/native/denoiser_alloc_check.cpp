// The denoiser's allocations without a GPU: denoise_net.cpp linked against a
// fake CUDA runtime whose device has a given number of bytes, and against
// launchers that do nothing (tests/test_denoiser_alloc_cpu.py builds and runs
// it). Prints what is allocated after each step.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

#include "denoise_net.h"

static size_t g_limit = SIZE_MAX, g_used = 0;
static std::map<void *, size_t> g_live;

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = nullptr;
    if (g_used > g_limit || n > g_limit - g_used) return cudaErrorMemoryAllocation;
    // (a device pointer: nothing reads or writes through it but cudaMemcpy)
    *p = std::malloc(n < (1u << 23) ? n : 16);
    g_live[*p] = n;
    g_used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    auto it = g_live.find(p);
    if (it == g_live.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    g_used -= it->second;
    g_live.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *, const void *, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}

namespace pray_gpu {
namespace dn {
using bf = __nv_bfloat16;
using st_t = cudaStream_t;
cudaError_t tc_conv_plan(TcConvPlan &p, const bf *x, int n, int h, int w, int cin, int cout, bool, int, bool) {
    p.x = x, p.n = n, p.h = h, p.w = w, p.cin = cin, p.cout = cout, p.grid = 152;
    return cudaSuccess;
}
size_t tc_packed_weight_elems(int cin_pad, int cout) { return (size_t)9 * cin_pad * ((cout + 15) / 16 * 16); }
cudaError_t tc_pack_all(const TcPackJob *, int, size_t, st_t) { return cudaSuccess; }
cudaError_t conv3x3_forward_tc(const TcConvPlan &, const bf *, const float *, bf *, float *, int *, st_t,
                               const TcFuse *, bool) {
    return cudaSuccess;
}
cudaError_t tc_wgrad_plan(TcWgradPlan &p, const TcWgradConv *, int, int) {
    p.partial_floats = 1 << 20;
    return cudaSuccess;
}
void tc_wgrad_place(TcWgradPlan &, float *) {}
cudaError_t wgrad_all_tc(const TcWgradPlan &, int *, st_t) { return cudaSuccess; }
cudaError_t grad_finish(const TcWgradPlan &, const BiasJob *, int, const float *, int, float *, float, st_t) {
    return cudaSuccess;
}
cudaError_t conv3x3_forward(const bf *, const bf *, const float *, bf *, float *, int, int, int, int, int, bool,
                            st_t) {
    return cudaSuccess;
}
cudaError_t conv3x3_backward(const bf *, const bf *, const float *, float *, float *, float *, int, int, int, int,
                             int, st_t) {
    return cudaSuccess;
}
cudaError_t relu_mask(const bf *, const float *, float *, size_t, st_t) { return cudaSuccess; }
cudaError_t avgpool(const bf *, bf *, int, int, int, int, st_t) { return cudaSuccess; }
cudaError_t avgpool_backward(const float *, float *, int, int, int, int, st_t) { return cudaSuccess; }
cudaError_t upsample_backward(const float *, float *, int, int, int, int, int, st_t) { return cudaSuccess; }
cudaError_t split_add(const float *, float *, size_t, int, int, int, st_t) { return cudaSuccess; }
cudaError_t pack_input(const float *, const __half *, bf *, bf *, size_t, size_t, st_t) { return cudaSuccess; }
cudaError_t upsample_concat(const bf *, const bf *, bf *, int, int, int, int, int, st_t) { return cudaSuccess; }
cudaError_t l1_loss(const float *, const float *, const __half *, float *, float *, float *, size_t, st_t) {
    return cudaSuccess;
}
int l1_blocks(size_t) { return 608; }
cudaError_t l1_loss_tc(const float *, const float *, const __half *, bf *, float *, size_t, size_t, st_t) {
    return cudaSuccess;
}
cudaError_t add_input(float *, const bf *, int, size_t, st_t) { return cudaSuccess; }
cudaError_t expm1_out(const float *, const __half *, float *, size_t, st_t) { return cudaSuccess; }
cudaError_t adam(float *, const float *, float *, float *, bf *, size_t, float, float, float, float, int, st_t) {
    return cudaSuccess;
}
cudaError_t to_bf16(const float *, bf *, size_t, st_t) { return cudaSuccess; }
}  // namespace dn
}  // namespace pray_gpu

using namespace pray_gpu;

// backward <tensor cores> <free bytes>: gradients of 2 x 64 x 64 while only
// <free bytes> are left for the backward pass, three times, then without the
// limit; the bytes in use after each.
static int backward_mode(bool tc, size_t left) {
    Denoiser d;
    if (d.init(1) != cudaSuccess) return 3;
    d.set_tensor_cores(tc);
    float rad, target;
    __half feat;
    for (int i = 0; i < 4; i++) {
        if (d.forward(&rad, &feat, 2, 64, 64, nullptr) != cudaSuccess) return 4;
        if (i == 0) {
            std::printf("%zu", g_used);
            g_limit = g_used + left;
        }
        if (i == 3) g_limit = SIZE_MAX;
        const cudaError_t e = d.backward(&target, nullptr);
        std::printf(" %d:%zu", (int)e, g_used);
    }
    std::printf("\n");
    return 0;
}

// resize: a pass of 2 x 64 x 64, then one of 1 x 64 x 64 without memory for it,
// twice: it has to fail both times.
static int resize_mode() {
    Denoiser d;
    if (d.init(1) != cudaSuccess) return 3;
    float rad;
    __half feat;
    std::printf("%d", (int)d.forward(&rad, &feat, 2, 64, 64, nullptr));
    g_limit = 1 << 20;
    if (g_used < g_limit) return 4;
    for (int i = 0; i < 2; i++) std::printf(" %d", (int)d.forward(&rad, &feat, 1, 64, 64, nullptr));
    g_limit = SIZE_MAX;
    std::printf(" %d\n", (int)d.forward(&rad, &feat, 1, 64, 64, nullptr));
    return 0;
}

int main(int argc, char **argv) {
    const std::string mode = argc > 1 ? argv[1] : "";
    if (mode == "backward") return backward_mode(std::atoi(argv[2]) != 0, (size_t)std::atoll(argv[3]));
    if (mode == "resize") return resize_mode();
    return 2;
}
