// 3x3 convolution forward on the 5th-generation tensor cores (tcgen05), BF16
// operands, FP32 accumulation in tensor memory (TMEM).
//
// Activations are planar in 8-channel chunks, [image][channel / 8][y][x][8]
// (16 bytes per pixel and chunk), which is the layout the tensor cores read
// from shared memory, so a halo is copied as whole rows.
//
// Implicit GEMM without an im2col copy. A tile is 16 x 8 output pixels (M =
// 128) x a chunk of the output channels (N, a multiple of 16). Its input halo,
// 18 x 10 pixels x Cin, is loaded by one
// 4-D TMA copy (rows of 160 contiguous bytes; out-of-image pixels arrive
// as zeros, which is the convolution's padding) into planes of
// [y][x][8 channels]. With channels-last tensors the same halo is a box of
// 16-byte rows, ten times as many requests (512^2 frame: 262 us against 216 us
// planar). In the planes the A operand of
// tap (dy, dx) for 16 channels is the halo itself seen through a shared-memory
// matrix descriptor: the tile's 8-pixel rows are the 8-row core-matrix
// groups (stride 160 bytes = one halo row), the two 8-channel chunks are the
// K-direction core matrices (stride = one plane), and the start address moves
// by (dy * 10 + dx) * 16 bytes. So all nine taps read the same halo and the
// threads gather nothing. The weights are packed once (tc_pack_all) as
// [tap][8-channel chunk][row][8] BF16 - exactly the no-swizzle K-major
// core-matrix layout - and a CTA copies the rows of its channels tap by tap.
// One thread issues the kind::f16 MMAs (M 128, N Npad, K 16) and commits them
// to mbarriers. See k_conv_tc for the pipeline and tc_conv_plan for the split.
//
// The epilogue also performs the network's glue (TcFuse): 2 x 2 average
// pooling, nearest 2x upsampling into a concatenation, the residual add and
// the output transform, as extra stores of the values it holds.
//
// Every mbarrier wait is bounded: on timeout the kernel records an error,
// stops issuing, waits (bounded) for the copies and MMAs it issued, and frees
// its TMEM.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "denoise_ops.h"

namespace pray_gpu {
namespace dn {

static_assert(sizeof(CUtensorMap) == sizeof(TcConvPlan::tmap), "tensor map size");

namespace {

constexpr int kTileW = 8, kTileH = 16;
constexpr int kHaloW = kTileW + 2, kHaloH = kTileH + 2;
constexpr uint32_t kPlaneBytes = kHaloW * kHaloH * 16;  // one 8-channel halo plane (2880), planes back to back
constexpr uint32_t kRowBytes = kHaloW * 16;             // one halo row of one plane (160)
constexpr uint32_t kWaitLimit = 1u << 24;
constexpr size_t kSmemMax = 227 * 1024;
constexpr size_t kSmemPerSm = 228 * 1024;
constexpr int kTaps = 9;

struct TcArgs {
    const __nv_bfloat16 *w;  // packed weights [tap][chunk][row][8]
    const float *bias;       // forward
    __nv_bfloat16 *y;
    float *y32;
    int n, h, wd, cin, cout, npad, relu;
    int tiles_x, tiles_y;
    int ring;                // halo slots
    int wstages;             // kTaps: every tap's weights resident; else a ring of taps
    int nsplit;              // > 1: blockIdx.y picks output channels [y * npad, (y + 1) * npad), the weight
                             // rows by TMA (wmap) from the packing of all rows
    int acc_slots, acc_stride, tmem_cols;  // accumulators, TMEM columns from one to the next
    uint32_t halo_stride, w_off, bias_off, bar_off;  // shared-memory layout (the halos are at 0)
    int *err;
    TcFuse f;                // extra stores of the epilogue
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Programmatic dependent launch. A convolution launched with programmatic
// stream serialisation may start while the previous kernel of the stream
// still runs: its prologue (barriers, tensor memory, weight copies) overlaps
// that kernel's tail, and the thread that loads the input waits here for the
// previous kernel to complete (and its writes to be visible) before the first
// input copy. Every global store of the kernel follows that wait (the
// epilogue runs after the MMAs, which follow the input copies). Once past it,
// the CTA lets the next kernel launch. Launched without the attribute, both
// instructions return at once.
__device__ __forceinline__ void grid_dependency_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Shared-memory matrix descriptor: start, leading (K-direction) and stride
// (8-row group) byte offsets, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N and M.
__host__ __device__ constexpr uint32_t inst_desc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kWaitLimit; i++) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// A tile of a planar tensor, every chunk: box (8 * columns, rows, chunks, 1
// image) at column x, row y; a halo starts at -1 (zero fill).
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap *map, uint32_t bar, int x, int y, int img) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, "
        "%6}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(8 * x), "r"(y), "r"(0), "r"(img)
        : "memory");
}

// A slice of packed weights: box (8 channels, npad rows, taps x chunks) of the
// 3-D map (8, npad_full, 9 x cin / 8) at rows from n, (tap, chunk) from k.
__device__ __forceinline__ void tma_w(uint32_t dst, const CUtensorMap *map, uint32_t bar, int n, int k) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
        "[%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(n), "r"(k)
        : "memory");
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void mma(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
        : "memory");
}

// One lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.u32 %0, 1, 0, P;\n}\n" : "=r"(p));
    return p != 0;
}

// The MMAs of one tap over kPairs pairs of 8-channel chunks. a: the halo at
// the tap's offset, b: the tap's packed weights, both in 16-byte units; bpair:
// weights of a chunk pair (2 npad); acc: 0 for the tile's first MMA. Only the
// start addresses of the descriptors change, by constants once unrolled: an
// MMA of N = 32 takes the tensor cores 41 clocks (4 KB + 1 KB of operands at
// 128 bytes per clock), which the issuing thread keeps up with only if it has
// little to compute per MMA (rebuilding descriptors in a rolled loop took it
// 95 to 220 clocks per MMA, whatever N).
template <int kPairs>
__device__ __forceinline__ void issue_tap(uint32_t tmem, uint32_t a, uint32_t b, uint32_t bpair, uint32_t idesc,
                                          uint32_t acc) {
    constexpr uint32_t kPair = 2 * (kPlaneBytes >> 4);
    constexpr uint64_t ahi = ((uint64_t)(kPlaneBytes >> 4) << 16) | ((uint64_t)(kRowBytes >> 4) << 32) | (1ull << 46);
    const uint64_t bhi = ((uint64_t)(bpair >> 1) << 16) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
#pragma unroll
    for (int p = 0; p < kPairs; p++) {
        mma(tmem, ahi | (a + p * kPair), bhi | b, idesc, acc);
        acc = 1;
        b += bpair;
    }
}

// All nine taps, accumulated in (tap, chunk) order (one or two chunk pairs:
// the taps of a row unrolled too).
template <int kPairs>
__device__ __forceinline__ void issue_tile(uint32_t tmem, uint32_t a, uint32_t b, uint32_t bpair, uint32_t idesc) {
    uint32_t acc = 0;
#pragma unroll 1
    for (int dy = 0; dy < 3; dy++, a += kRowBytes >> 4) {
#pragma unroll(kPairs <= 2 ? 3 : 1)
        for (int dx = 0; dx < 3; dx++, b += kPairs * bpair) {
            issue_tap<kPairs>(tmem, a + dx, b, bpair, idesc, acc);
            acc = 1;
        }
    }
}

__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// The epilogue's arithmetic on pairs: FP32 add, BF16 rounding, and max(., 0)
// of a rounded pair (the same value as rounding max(., 0): NaN gives 0).
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t pair(uint32_t lo, uint32_t hi) { return (uint64_t)hi << 32 | lo; }
__device__ __forceinline__ uint32_t round2(uint64_t v) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "r"((uint32_t)(v >> 32)), "r"((uint32_t)v));
    return d;
}
__device__ __forceinline__ uint32_t relu2(uint32_t v) {
    uint32_t d;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(v), "r"(0u));
    return d;
}
// The two values of a BF16 pair as FP32.
__device__ __forceinline__ uint64_t widen2(uint32_t w) { return pair(w << 16, w & 0xFFFF0000u); }

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// TMEM columns [c, c + 16 kBlocks) of the warp's 32 lanes.
template <int kBlocks>
__device__ __forceinline__ void load_tmem(uint32_t taddr, uint32_t *r) {
#pragma unroll
    for (int b = 0; b < kBlocks; b++)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
            "[%16];"
            : "=r"(r[16 * b]), "=r"(r[16 * b + 1]), "=r"(r[16 * b + 2]), "=r"(r[16 * b + 3]), "=r"(r[16 * b + 4]),
              "=r"(r[16 * b + 5]), "=r"(r[16 * b + 6]), "=r"(r[16 * b + 7]), "=r"(r[16 * b + 8]),
              "=r"(r[16 * b + 9]), "=r"(r[16 * b + 10]), "=r"(r[16 * b + 11]), "=r"(r[16 * b + 12]),
              "=r"(r[16 * b + 13]), "=r"(r[16 * b + 14]), "=r"(r[16 * b + 15])
            : "r"(taddr + 16 * b)
            : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// What a convolution stores (a kernel instance each): the BF16 outputs; also
// their 2 x 2 averages and a copy into a concatenation; also (or only) the
// outputs upsampled into a concatenation; FP32 outputs (channels last), with
// the residual and the output transform; and the three of a backward-data
// convolution (TcFuse::grad).
enum EpiMode { kEpiY, kEpiPool, kEpiUp, kEpiF32, kEpiGradMask, kEpiGradCat, kEpiGradUnpool };

// A warp's share of a tile: one pixel per lane (tile row m = pixel (m / 8,
// m % 8)), the planes' size and where the pixel's first stores go.
struct EpiPixel {
    int lane;
    bool valid, pool_valid;
    uint32_t px, pp;       // pixels of a plane, of a pooled plane
    uint4 *y, *cat, *pool; // the tile's chunk n0 / 8 at the lane's pixel
    size_t pix;            // channels-last pixel
    const __nv_bfloat16 *res;
    // backward: gradient and mask (16 bytes per pixel and chunk), the FP32 share
    // (32 bytes) at chunk n0 / 8 of the lane's pixel, block or low-resolution
    // pixel; the warp's bias sums (npad floats)
    uint4 *g;
    const uint4 *mask;
    float4 *skip;
    float *bsum;
};

// v where the BF16 pair m is positive, else 0.
__device__ __forceinline__ uint64_t mask2(uint64_t v, uint32_t m) {
    const bool a = __uint_as_float(m << 16) > 0.f, b = __uint_as_float(m & 0xFFFF0000u) > 0.f;
    return pair(a ? (uint32_t)v : 0u, b ? (uint32_t)(v >> 32) : 0u);
}

// Adds the sums over the warp's lanes of 16 values each (pairs) to
// sums[0..16): halves are exchanged so that every step adds half as many
// values; lane 2 c ends with channel c (in the order of its bits).
__device__ __forceinline__ void lane_sums16(const uint64_t *p, int lane, float *sums) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    float v[16];
#pragma unroll
    for (int k = 0; k < 8; k++) v[2 * k] = __uint_as_float((uint32_t)p[k]), v[2 * k + 1] = __uint_as_float((uint32_t)(p[k] >> 32));
#pragma unroll
    for (int n = 8, o = 16; n >= 1; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k < n) {
                const float got = __shfl_xor_sync(kFull, up ? v[k] : v[k + n], o);
                v[k] = (up ? v[k + n] : v[k]) + got;
            }
    }
    v[0] += __shfl_xor_sync(kFull, v[0], 1);
    const int c = (lane >> 4 & 1) * 8 + (lane >> 3 & 1) * 4 + (lane >> 2 & 1) * 2 + (lane >> 1 & 1);
    if (!(lane & 1)) sums[c] += v[0];
}

// The backward stores (TcFuse::grad) of 16 channels; q: chunk from the CTA's
// first, c0: channel from the CTA's first, c: channel.
template <int kMode>
__device__ __forceinline__ void store_grad16(const TcArgs &P, const uint32_t *r, const EpiPixel &e, int q, int c0,
                                             int c) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    uint64_t v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = pair(r[2 * k], r[2 * k + 1]);
    if (kMode == kEpiGradCat && c >= P.f.low_c) {
        if (e.valid) {
            float4 *o = e.skip + (size_t)q * 2 * e.px;
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const uint64_t a = v[4 * j + 2 * k], b = v[4 * j + 2 * k + 1];
                    o[(size_t)j * 2 * e.px + k] = make_float4(
                        __uint_as_float((uint32_t)a), __uint_as_float((uint32_t)(a >> 32)),
                        __uint_as_float((uint32_t)b), __uint_as_float((uint32_t)(b >> 32)));
                }
        }
        return;
    }
    if (kMode == kEpiGradMask) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            uint4 m = make_uint4(0u, 0u, 0u, 0u);
            if (e.valid) m = e.mask[(size_t)(q + j) * e.px];
            const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int k = 0; k < 4; k++) v[4 * j + k] = mask2(v[4 * j + k], mw[k]);
            if (e.valid)
                e.g[(size_t)(q + j) * e.px] = make_uint4(round2(v[4 * j]), round2(v[4 * j + 1]), round2(v[4 * j + 2]),
                                                         round2(v[4 * j + 3]));
        }
        lane_sums16(v, e.lane, e.bsum + c0);
    }
    if (kMode == kEpiGradCat) {
        // 2 x 2 sums (row-major), as in the pooling: each lane of a block ends
        // with two of the eight channel pairs
        const bool odd = e.lane & 1, low = e.lane & 8;
        uint64_t a[4], b[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint64_t got = __shfl_xor_sync(kFull, odd ? v[k] : v[4 + k], 1);
            a[k] = odd ? got : v[k], b[k] = odd ? v[4 + k] : got;
        }
        uint2 m = make_uint2(0u, 0u);
        const size_t at = (size_t)(q + (odd ? 1 : 0)) * e.pp;
        if (e.pool_valid) m = reinterpret_cast<const uint2 *>(e.mask + at)[low ? 1 : 0];
        uint64_t sum[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint64_t ga = __shfl_xor_sync(kFull, low ? a[k] : a[2 + k], 8);
            const uint64_t gb = __shfl_xor_sync(kFull, low ? b[k] : b[2 + k], 8);
            const uint64_t ta = low ? ga : a[k], tb = low ? gb : b[k];          // the upper row's
            const uint64_t ba = low ? a[2 + k] : ga, bb = low ? b[2 + k] : gb;  // the lower row's
            sum[k] = mask2(add2(add2(add2(ta, tb), ba), bb), k ? m.y : m.x);
        }
        if (e.pool_valid) reinterpret_cast<uint2 *>(e.g + at)[low ? 1 : 0] = make_uint2(round2(sum[0]), round2(sum[1]));
        // over the warp's eight blocks (lane bits 1, 2 and 4)
#pragma unroll
        for (int o : {2, 4, 16})
#pragma unroll
            for (int k = 0; k < 2; k++) sum[k] = add2(sum[k], __shfl_xor_sync(kFull, sum[k], o));
        if ((e.lane & ~9) == 0) {
            float *d = e.bsum + c0 + (odd ? 8 : 0) + (low ? 4 : 0);
#pragma unroll
            for (int k = 0; k < 2; k++)
                d[2 * k] += __uint_as_float((uint32_t)sum[k]), d[2 * k + 1] += __uint_as_float((uint32_t)(sum[k] >> 32));
        }
    }
    if (kMode == kEpiGradUnpool) {
        const uint32_t W2 = 2 * (uint32_t)P.wd;
        const uint64_t quarter = pair(0x3E800000u, 0x3E800000u);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            uint64_t s[4] = {};  // the chunk's sums over the four pixels
            uint64_t share[4];
#pragma unroll
            for (int k = 0; k < 4; k++) asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(share[k]) : "l"(v[4 * j + k]), "l"(quarter));
            if (e.valid) {
                const size_t plane = (size_t)(q + j) * 4 * e.px;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const size_t at = plane + (i >> 1) * W2 + (i & 1);
                    const uint4 m = e.mask[at];
                    const ulonglong2 *sk = reinterpret_cast<const ulonglong2 *>(e.skip + 2 * at);
                    const ulonglong2 s0 = sk[0], s1 = sk[1];
                    const uint64_t g0 = mask2(add2(s0.x, share[0]), m.x), g1 = mask2(add2(s0.y, share[1]), m.y);
                    const uint64_t g2 = mask2(add2(s1.x, share[2]), m.z), g3 = mask2(add2(s1.y, share[3]), m.w);
                    e.g[at] = make_uint4(round2(g0), round2(g1), round2(g2), round2(g3));
                    s[0] = add2(s[0], g0), s[1] = add2(s[1], g1), s[2] = add2(s[2], g2), s[3] = add2(s[3], g3);
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) v[4 * j + k] = s[k];
        }
        lane_sums16(v, e.lane, e.bsum + c0);
    }
}

// The stores of 16 channels (chunk q and q + 1 from the CTA's first;
// accumulators r) of a lane's pixel: bias + ReLU as BF16 (planar: the eight
// pixels of a tile row are 128 contiguous bytes per chunk) or FP32, plus the
// extra stores of P.f. bias: the 16 channels' (shared memory); c: the first.
template <int kMode>
__device__ __forceinline__ void store16(const TcArgs &P, const uint32_t *r, const EpiPixel &e, int q, int c,
                                        const float *bias) {
    uint64_t v[8];
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const uint4 b = *reinterpret_cast<const uint4 *>(bias + 2 * k);
        v[k] = add2(pair(r[2 * k], r[2 * k + 1]), pair(b.x, b.y));
        v[k + 1] = add2(pair(r[2 * k + 2], r[2 * k + 3]), pair(b.z, b.w));
    }
    if (kMode == kEpiF32) {
        if (!e.valid) return;
        uint2 res = make_uint2(0u, 0u);  // four channels of the residual
        if (e.res) res = *reinterpret_cast<const uint2 *>(e.res);
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int co = c + k;
            if (co >= P.cout) break;
            float u = __uint_as_float((uint32_t)(k & 1 ? v[k / 2] >> 32 : v[k / 2]));
            if (P.relu) u = fmaxf(u, 0.f);
            if (k < 4 && e.res) {
                const uint32_t w = k < 2 ? res.x : res.y;
                u += __uint_as_float(k & 1 ? w & 0xFFFF0000u : w << 16);
            }
            if (P.y32) P.y32[e.pix * P.cout + co] = u;
            if (P.f.rad)
                P.f.rad[e.pix * 3 + co] =
                    expm1f(u) * (fmaxf(__half2float(P.f.feat[7 * e.pix + co]), 0.f) + kDemodFloor);
        }
        return;
    }
    uint32_t w[8];
#pragma unroll
    for (int k = 0; k < 8; k++) w[k] = P.relu ? relu2(round2(v[k])) : round2(v[k]);
    const uint4 lo = make_uint4(w[0], w[1], w[2], w[3]), hi = make_uint4(w[4], w[5], w[6], w[7]);
    if (e.valid && P.y) {
        uint4 *o = e.y + (size_t)q * e.px;
        o[0] = lo, o[e.px] = hi;
    }
    if (kMode == kEpiUp && e.valid) {
        // the pixel's 2 x 2 block: two neighbours (32 bytes) in each of two rows
        const uint32_t W2 = 2 * (uint32_t)P.wd;
        uint4 *o = e.cat + (size_t)q * 4 * e.px;
        o[0] = lo, o[1] = lo, o[W2] = lo, o[W2 + 1] = lo;
        o += 4 * e.px;
        o[0] = hi, o[1] = hi, o[W2] = hi, o[W2 + 1] = hi;
    }
    if (kMode == kEpiPool) {
        if (e.valid) {
            uint4 *o = e.cat + (size_t)q * e.px;
            o[0] = lo, o[e.px] = hi;
        }
        // A warp holds four whole tile rows: a 2 x 2 block is lanes l (even
        // row and column), l + 1, l + 8, l + 9. Each of the four averages two
        // of the eight channel pairs: the lanes of a column pair exchange
        // halves, then the rows exchange quarters, both values of each row
        // kept so that the sum is in the order of k_avgpool (row-major).
        constexpr unsigned kFull = 0xFFFFFFFFu;
        const bool odd = e.lane & 1, low = e.lane & 8;
        uint32_t a[4], b[4];  // the row's left and right pixel, four pairs
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t got = __shfl_xor_sync(kFull, odd ? w[k] : w[4 + k], 1);
            a[k] = odd ? got : w[k], b[k] = odd ? w[4 + k] : got;
        }
        uint32_t o[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t ga = __shfl_xor_sync(kFull, low ? a[k] : a[2 + k], 8);
            const uint32_t gb = __shfl_xor_sync(kFull, low ? b[k] : b[2 + k], 8);
            const uint32_t ta = low ? ga : a[k], tb = low ? gb : b[k];          // the upper row's
            const uint32_t ba = low ? a[2 + k] : ga, bb = low ? b[2 + k] : gb;  // the lower row's
            const uint64_t s = add2(add2(add2(widen2(ta), widen2(tb)), widen2(ba)), widen2(bb));
            o[k] = pack2(0.25f * __uint_as_float((uint32_t)s), 0.25f * __uint_as_float((uint32_t)(s >> 32)));
        }
        // pairs 0-3 are the first chunk, 4-7 the second
        if (e.pool_valid) {
            uint2 *d = reinterpret_cast<uint2 *>(e.pool + (size_t)(q + (odd ? 1 : 0)) * e.pp) + (low ? 1 : 0);
            *d = make_uint2(o[0], o[1]);
        }
    }
}

// Epilogue of one tile: the calling warp reads TMEM lanes 32q..32q+31 (q =
// quad, the warp's lane quadrant: its warp index mod 4) from column `tmem`
// on, 32 columns at a time.
template <int kMode>
__device__ __forceinline__ void epilogue(const TcArgs &P, uint32_t tmem, int img, int y0, int x0, int quad, int n0,
                                         const float *bias, float *bsum) {
    constexpr bool kGrad = kMode == kEpiGradMask || kMode == kEpiGradCat || kMode == kEpiGradUnpool;
    EpiPixel e;
    e.lane = (int)(threadIdx.x & 31);
    const int m = quad * 32 + e.lane, yy = y0 + (m >> 3), xx = x0 + (m & 7);
    e.valid = yy < P.h && xx < P.wd;
    e.px = (uint32_t)P.h * (uint32_t)P.wd;
    const uint32_t at = (uint32_t)yy * (uint32_t)P.wd + (uint32_t)xx;
    const int q0 = n0 >> 3;
    if (kMode == kEpiF32) {
        e.pix = (size_t)img * e.px + at;
        e.res = P.f.res ? P.f.res + ((size_t)img * (P.f.res_c >> 3) * e.px + at) * 8 : nullptr;
    } else if (!kGrad) {
        e.y = reinterpret_cast<uint4 *>(P.y) + ((size_t)img * (P.cout >> 3) + q0) * e.px + at;
    }
    if (kMode == kEpiPool || kMode == kEpiUp) {
        const size_t plane = (size_t)img * (P.f.cat_c >> 3) + (P.f.cat_off >> 3) + q0;
        e.cat = reinterpret_cast<uint4 *>(P.f.cat);
        if (kMode == kEpiUp) e.cat += plane * 4 * e.px + 4 * (size_t)yy * P.wd + 2 * xx;
        else e.cat += plane * e.px + at;
    }
    if (kMode == kEpiPool) {
        const int ho = P.h >> 1, wo = P.wd >> 1, yo = yy >> 1, xo = xx >> 1;
        e.pool_valid = yo < ho && xo < wo;
        e.pp = (uint32_t)ho * (uint32_t)wo;
        e.pool = reinterpret_cast<uint4 *>(P.f.pool) + ((size_t)img * (P.cout >> 3) + q0) * e.pp + (uint32_t)yo * wo + xo;
    }
    if (kGrad) {
        size_t plane, pos;  // of mask and g
        const size_t planes = (size_t)img * (P.cout >> 3) + q0;
        e.bsum = bsum;
        if (kMode == kEpiGradMask) {
            plane = planes * e.px, pos = at;
        } else if (kMode == kEpiGradCat) {
            e.pp = (uint32_t)(P.h >> 1) * (uint32_t)(P.wd >> 1);
            e.pool_valid = e.valid;  // (h and w are even where a concatenation is)
            plane = ((size_t)img * (P.f.low_c >> 3) + q0) * e.pp;
            pos = (size_t)(yy >> 1) * (P.wd >> 1) + (xx >> 1);
            // the chunk at or after low_c (store_grad16 uses it from there on)
            e.skip = reinterpret_cast<float4 *>(P.f.skip) +
                     (((size_t)img * ((P.cout - P.f.low_c) >> 3) + q0) * e.px + at) * 2 -
                     (size_t)(P.f.low_c >> 3) * e.px * 2;
        } else {
            plane = planes * 4 * e.px, pos = 4 * (size_t)yy * P.wd + 2 * xx;
            e.skip = reinterpret_cast<float4 *>(P.f.skip) + 2 * (plane + pos);
        }
        e.mask = reinterpret_cast<const uint4 *>(P.f.mask) + plane + pos;
        e.g = reinterpret_cast<uint4 *>(P.f.g) + plane + pos;
    }
    auto store = [&](const uint32_t *v, int c0) {
        if constexpr (kGrad) store_grad16<kMode>(P, v, e, c0 >> 3, c0, n0 + c0);
        else store16<kMode>(P, v, e, c0 >> 3, n0 + c0, bias + c0);
    };
    const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16);
    uint32_t r[32];
    int c0 = 0;
    for (; c0 + 32 <= P.npad; c0 += 32) {
        load_tmem<2>(taddr + c0, r);
        store(r, c0);
        store(r + 16, c0 + 16);
    }
    if (c0 < P.npad) {
        load_tmem<1>(taddr + c0, r);
        store(r, c0);
    }
}

__device__ __forceinline__ void mbar_init_count(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

constexpr int kEpiGroups = 3;  // groups of four epilogue warps
constexpr int kEpiWarps = 4 * kEpiGroups;
constexpr int kConvThreads = 64 + 32 * kEpiWarps;

// A position in a ring of n slots and its phase (the parity of the completed
// rounds), moved on without divisions: the roles' loops are one thread's or
// one warp's serial chains, and the divisions by the ring sizes and the tile
// counts took more time per tile than 9 MMAs do.
struct Ring {
    int n, slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ explicit Ring(int slots) : n(slots) {}
    __device__ __forceinline__ void next() {
        if (++slot == n) slot = 0, phase ^= 1u;
    }
};

// Every `step`-th tile from `first` on: image, row and column of tiles.
struct TileWalk {
    int img, ty, tx, d_img, d_ty, d_tx, tiles_x, tiles_y;
    __device__ __forceinline__ TileWalk(int first, int step, int tx_n, int ty_n) : tiles_x(tx_n), tiles_y(ty_n) {
        const int per = tx_n * ty_n;
        img = first / per, d_img = step / per;
        first -= img * per, step -= d_img * per;
        ty = first / tx_n, tx = first - ty * tx_n;
        d_ty = step / tx_n, d_tx = step - d_ty * tx_n;
    }
    __device__ __forceinline__ int x0() const { return tx * kTileW; }
    __device__ __forceinline__ int y0() const { return ty * kTileH; }
    __device__ __forceinline__ void next() {
        img += d_img, ty += d_ty, tx += d_tx;
        if (tx >= tiles_x) tx -= tiles_x, ty++;
        if (ty >= tiles_y) ty -= tiles_y, img++;
    }
};

// The state that the roles of a convolution's CTA share.
struct ConvCta {
    uint32_t halo0, wbase, bars, tmem;
    int items;
    volatile int *abort_flag, *h_issued, *h_waited, *w_issued, *w_waited;
    // barriers: halo loaded [H], halo released [H], accumulator full [A],
    // drained [A], weights loaded [S], weights released [S], final drain
    int hfull, hfree, afull, afree, wfull, wfree, dbar;
    __device__ __forceinline__ uint32_t bar(int i) const { return bars + 8u * (uint32_t)i; }
};

// The MMA role (one thread) for Cin = 16 kPairs.
template <int kPairs>
__device__ __forceinline__ void conv_mma(const TcArgs &P, const ConvCta &C) {
    const int H = P.ring, S = P.wstages, A = P.acc_slots;
    const bool resident = S == kTaps;
    const uint32_t idesc = inst_desc(128, P.npad), bpair = 2 * P.npad, wtap = (uint32_t)P.cin * P.npad * 2;
    bool ok = true;
    Ring h(H), a(A), w(S);
    if (resident) {
        ok = mbar_wait(C.bar(C.wfull), 0);
        if (ok) *C.w_waited = 1;
    }
    for (int i = 0; i < C.items && ok && !*C.abort_flag; i++) {
        if (!(ok = mbar_wait(C.bar(C.hfull + h.slot), h.phase))) break;
        *C.h_waited = i + 1;
        if (i >= A && !(ok = mbar_wait(C.bar(C.afree + a.slot), a.phase ^ 1u))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = C.tmem + (uint32_t)(a.slot * P.acc_stride);
        const uint32_t hb = (C.halo0 + (uint32_t)h.slot * P.halo_stride) >> 4;
        if (resident) {
            issue_tile<kPairs>(acc, hb, C.wbase >> 4, bpair, idesc);
        } else {
            uint32_t ha = hb;
#pragma unroll 1
            for (int tap = 0; tap < kTaps; tap++) {
                if (!(ok = mbar_wait(C.bar(C.wfull + w.slot), w.phase))) break;
                *C.w_waited = i * kTaps + tap + 1;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                issue_tap<kPairs>(acc, ha, (C.wbase + w.slot * wtap) >> 4, bpair, idesc, tap ? 1u : 0u);
                commit(C.bar(C.wfree + w.slot));
                w.next();
                ha += tap == 2 || tap == 5 ? (kRowBytes >> 4) - 2 : 1;
            }
            if (!ok) break;
        }
        commit(C.bar(C.hfree + h.slot));
        commit(C.bar(C.afull + a.slot));
        h.next(), a.next();
    }
    if (!ok) *C.abort_flag = 1;
    // everything this thread issued completes before TMEM is freed
    commit(C.bar(C.dbar));
    mbar_wait(C.bar(C.dbar), 0);
}

// One convolution. A persistent, warp-specialised CTA owns a chunk of the
// output channels (blockIdx.y) and walks tiles blockIdx.x, blockIdx.x +
// gridDim.x, ...:
//   warp 0 (one thread) loads weights, either all nine taps once or, where
//     they do not fit beside the halos, tap after tap through a ring of
//     wstages slots for every tile; and tile i's halo into slot i % ring once
//     the MMAs of tile i - ring have released it;
//   warp 1 (one thread) waits for the halo, for accumulator i % acc_slots to be
//     drained and for each tap's weights, issues the tile's MMAs and commits
//     them to the slots' "released" and the accumulator's "full" barriers;
//   the other warps, groups of four (one TMEM lane quadrant each), drain the
//     accumulators of the tiles in turn to global memory and release them.
// So loads, MMAs and epilogues of consecutive tiles overlap inside a CTA, and
// one or two CTAs per SM suffice: more of them would start up one after
// another (their tensor memory is allocated under a lock), 8 us before the
// last of eight per SM had loaded its first tile. Every wait
// is bounded; a timeout sets a shared abort flag that ends every role's
// loop, and the copies and MMAs in flight are waited for (bounded) before
// the shared memory and TMEM are released.
template <int kMode>
__global__ void __launch_bounds__(kConvThreads, 2) k_conv_tc(const __grid_constant__ CUtensorMap xmap,
                                                             const __grid_constant__ CUtensorMap wmap, TcArgs P) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int H = P.ring, S = P.wstages, A = P.acc_slots;
    const bool resident = S == kTaps;
    const int nchunk = P.cin >> 3;
    float *bias = reinterpret_cast<float *>(smem + P.bias_off);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + P.bar_off);
    ConvCta C;
    C.halo0 = smem_u32(smem), C.wbase = C.halo0 + P.w_off, C.bars = smem_u32(bars);
    C.hfull = 0, C.hfree = H, C.afull = 2 * H, C.afree = C.afull + A, C.wfull = C.afree + A, C.wfree = C.wfull + S,
    C.dbar = C.wfree + S;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + C.dbar + 1);
    C.abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    // loads issued by warp 0 and waited for by warp 1: halos, weights
    C.h_issued = C.abort_flag + 1, C.h_waited = C.abort_flag + 2, C.w_issued = C.abort_flag + 3,
    C.w_waited = C.abort_flag + 4;
    const int n0 = (int)blockIdx.y * P.npad;
    const int first = (int)blockIdx.x, step = (int)gridDim.x;
    const int items = (P.n * P.tiles_x * P.tiles_y - 1 - first) / step + 1;
    C.items = items;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(P.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&xmap)) : "memory");
        for (int i = 0; i < C.dbar + 1; i++) mbar_init_count(C.bar(i), i >= C.afree && i < C.wfull ? 128 : 1);
        *C.abort_flag = 0, *C.h_issued = 0, *C.h_waited = 0, *C.w_issued = 0, *C.w_waited = 0;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    constexpr bool kGrad = kMode == kEpiGradMask || kMode == kEpiGradCat || kMode == kEpiGradUnpool;
    // forward: the chunk's bias; backward: each epilogue warp's bias-gradient sums
    for (int i = tid - 64; i >= 0 && i < (kGrad ? kEpiWarps * P.npad : P.npad); i += kConvThreads - 64)
        bias[i] = !kGrad && n0 + i < P.cout ? __ldg(P.bias + n0 + i) : 0.f;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    C.tmem = *tmem_slot;

    if (warp == 0) {
        if (elect_one()) {
            const uint32_t wtap = (uint32_t)P.cin * P.npad * 2;  // bytes of a tap's weights
            // taps k and k + 1 ... k + n - 1 to consecutive slots from slot s
            auto copy_taps = [&](int s, int tap, int n, uint32_t b) {
                mbar_expect_tx(b, n * wtap);
                if (P.nsplit == 1)
                    bulk_copy(C.wbase + s * wtap, P.w + (size_t)tap * P.cin * P.npad, n * wtap, b);
                else
                    for (int t = 0; t < n; t++) tma_w(C.wbase + (s + t) * wtap, &wmap, b, n0, (tap + t) * nchunk);
            };
            Ring w(S), h(H);
            TileWalk t(first, step, P.tiles_x, P.tiles_y);
            int k = 0, next_tap = 0;  // taps and halos loaded so far, the next tap
            int halos = 0;
            auto load_tap = [&]() {
                if (k >= S && !mbar_wait(C.bar(C.wfree + w.slot), w.phase ^ 1u)) return false;
                copy_taps(w.slot, next_tap, 1, C.bar(C.wfull + w.slot));
                *C.w_issued = ++k;
                if (++next_tap == kTaps) next_tap = 0;
                w.next();
                return true;
            };
            auto load_halo = [&]() {
                if (halos >= H && !mbar_wait(C.bar(C.hfree + h.slot), h.phase ^ 1u)) return false;
                const uint32_t b = C.bar(C.hfull + h.slot);
                mbar_expect_tx(b, (uint32_t)nchunk * kPlaneBytes);
                tma_tile(C.halo0 + (uint32_t)h.slot * P.halo_stride, &xmap, b, t.x0() - 1, t.y0() - 1, t.img);
                *C.h_issued = ++halos;
                h.next(), t.next();
                return true;
            };
            // the weights do not depend on the previous kernel; the input does
            if (resident) copy_taps(0, 0, kTaps, C.bar(C.wfull)), *C.w_issued = 1;
            else
                while (k < S) load_tap();
            grid_dependency_wait();
            bool ok = load_halo();
            for (int i = 0; i < items && ok && !*C.abort_flag; i++) {
                // the next tile's halo before the rest of this one's weights
                if (H > 1 && i + 1 < items) ok = load_halo();
                if (!resident)
                    while (ok && k < kTaps * (i + 1)) ok = load_tap();
                if (H == 1 && i + 1 < items && ok) ok = load_halo();
            }
            if (!ok) *C.abort_flag = 1;
        }
    } else if (warp == 1) {
        if (elect_one()) {
            switch (nchunk / 2) {  // the network's channel counts
            case 1: conv_mma<1>(P, C); break;
            case 2: conv_mma<2>(P, C); break;
            case 3: conv_mma<3>(P, C); break;
            case 4: conv_mma<4>(P, C); break;
            case 5: conv_mma<5>(P, C); break;
            case 6: conv_mma<6>(P, C); break;
            case 7: conv_mma<7>(P, C); break;
            case 8: conv_mma<8>(P, C); break;
            case 10: conv_mma<10>(P, C); break;
            case 14: conv_mma<14>(P, C); break;
            default: *C.abort_flag = 1;
            }
        }
    } else {
        const int quad = warp & 3;  // the warp's TMEM lane quadrant
        // every decision warp-uniform: the TMEM loads below are warp-collective
        // No more groups than accumulators: a group that waits for tile i has
        // seen tile i - groups done, so the slot's previous tile i - A is done
        // too and its barrier is in the phase just before the one waited for
        // (with fewer accumulators the wait could be met by the phase before
        // that, whose parity is the same).
        const int group = (warp - 2) >> 2, groups = A < kEpiGroups ? A : kEpiGroups;
        TileWalk t(first + group * step, groups * step, P.tiles_x, P.tiles_y);
        Ring acc(A);
        for (int i = 0; i < group; i++) acc.next();
        for (int i = group < groups ? group : items; i < items; i += groups, t.next()) {
            if (__any_sync(0xFFFFFFFFu, *C.abort_flag != 0)) break;
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(C.bar(C.afull + acc.slot), acc.phase))) {
                if (lane == 0) *C.abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            epilogue<kMode>(P, C.tmem + (uint32_t)(acc.slot * P.acc_stride), t.img, t.y0(), t.x0(), quad, n0, bias,
                            bias + (warp - 2) * P.npad);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(C.bar(C.afree + acc.slot));
            for (int k = 0; k < groups; k++) acc.next();
        }
    }
    __syncthreads();
    if (tid == 0 && *C.abort_flag) {
        atomicExch(P.err, 1);
        // copies still in flight (bounded) before the shared memory goes away
        for (int j = *C.h_waited; j < *C.h_issued; j++) mbar_wait(C.bar(C.hfull + j % H), (uint32_t)(j / H) & 1u);
        for (int j = *C.w_waited; j < *C.w_issued; j++) mbar_wait(C.bar(C.wfull + j % S), (uint32_t)(j / S) & 1u);
    }
    if (kGrad) {  // the warps' sums in warp order (the roles have met above)
        const int channels = kMode == kEpiGradCat ? P.f.low_c : P.cout;
        for (int i = tid; i < P.npad && n0 + i < channels; i += kConvThreads) {
            float sum = 0.f;
            for (int k = 0; k < kEpiWarps; k++) sum += bias[k * P.npad + i];
            P.f.bias_part[(size_t)blockIdx.x * channels + n0 + i] = sum;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(C.tmem), "r"(P.tmem_cols)
                     : "memory");
    }
}

// ---- weight gradient ---------------------------------------------------------
//
// dw[co][tap][ci] = sum_p g[p][co] x[p + offset(tap)][ci]: per tap a GEMM with
// M = co (64 or 128 rows: the output-gradient channels, zero rows above cout),
// N = ci (cin_pad), K = pixels. Both operands come straight from the
// channel-planar tiles TMA writes ([8-channel plane][pixel][8 channels], 16
// bytes per pixel), read as MN-major matrices (the 8 channels of a pixel
// contiguous, pixels along K):
//   A: the tile's output gradient, one 2,048-byte plane per 8 channels
//      (16 x 8 pixels); core matrices 128 bytes apart along K (8 pixels = one
//      tile row) and one plane apart along M;
//   B: the input halo (18 x 10 pixels per plane, as in the forward pass);
//      for tap (dy, dx) the K-step covering tile rows 2k and 2k + 1 starts at
//      halo pixel (2k + dy, dx), core matrices one halo row (160 bytes) apart
//      along K and one plane apart along N.
// So every tap reads the same halo, shifted by whole 16-byte pixels, as in
// the forward pass. An item is a group of tiles and of taps of one
// convolution (tensor memory holds taps_per_pass x cin_pad FP32 columns, half
// of it, so that two CTAs share an SM and one's epilogue runs beside the
// other's MMAs); all convolutions' items are one grid, the longest first, so
// that the deep levels' few tiles fill the SMs that the wide levels leave (one
// launch per convolution: 8 to 34 us each, 340 us and 130 us of finalizing
// for a batch of 8 x 128^2). One thread loads the
// tiles through up to four shared-memory stages and issues the MMAs. The sums
// of the output channels below cout go to out[group][tap][co][ci]. Every wait
// is bounded (error flag, drain, TMEM freed).
constexpr uint32_t kGradPlaneBytes = kTileW * kTileH * 16;  // 2,048

struct WgArgs {
    TcWgradPlan p;
    int *err;
};

// MN-major A and B: transpose bits of the kind::f16 instruction descriptor
__host__ __device__ constexpr uint32_t inst_desc_mn(int m, int n) { return inst_desc(m, n) | (1u << 15) | (1u << 16); }

__global__ void __launch_bounds__(128, 2) k_wgrad_tc(const __grid_constant__ WgArgs A) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5;
    int ji = 0;
    while (ji + 1 < A.p.jobs && A.p.job[ji + 1].first_item <= (int)blockIdx.x) ji++;
    const TcWgradJob &P = A.p.job[ji];
    const int S = P.stages;
    const uint32_t base = smem_u32(smem);
    // bars[s] stage s loaded, bars[4 + s] MMAs reading stage s done, bars[8] drain
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + A.p.bar_off);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 9);
    int *okflag = reinterpret_cast<int *>(tmem_slot + 1);
    const int gplanes = P.cout_pad >> 3, xplanes = P.cin_pad >> 3;
    const int item = (int)blockIdx.x - P.first_item, group = item / P.passes, pass = item - group * P.passes;
    const int tap0 = pass * P.taps_per_pass, ntaps = min(9 - tap0, P.taps_per_pass);
    const int t_begin = group * P.tiles_per_cta, n = min(P.tiles, t_begin + P.tiles_per_cta) - t_begin;
    auto bar = [&](int i) { return smem_u32(&bars[i]); };

    // the rows of A above cout_pad stay zero, in every stage
    for (int st = 0; st < S; st++)
        for (uint32_t i = (uint32_t)gplanes * kGradPlaneBytes / 16 + tid; i < P.b_off / 16; i += 128)
            reinterpret_cast<uint4 *>(smem + (size_t)st * P.stage_bytes)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(A.p.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < 9; i++) mbar_init(bar(i));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the zero rows, for the tensor cores
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (tid == 0) {
        grid_dependency_wait();
        const CUtensorMap *gmap = reinterpret_cast<const CUtensorMap *>(P.gmap);
        const CUtensorMap *xmap = reinterpret_cast<const CUtensorMap *>(P.xmap);
        const uint32_t idesc = inst_desc_mn(P.rows, P.cin_pad);
        const uint32_t bytes = (uint32_t)gplanes * kGradPlaneBytes + (uint32_t)xplanes * kPlaneBytes;
        TileWalk t(t_begin, 1, P.tiles_x, P.tiles_y);
        Ring in(S), out(S);  // stages loaded, stages consumed
        int issued = 0, waited = 0;
        auto load = [&]() {
            const uint32_t a = base + (uint32_t)in.slot * P.stage_bytes, b = bar(in.slot);
            mbar_expect_tx(b, bytes);
            tma_tile(a, gmap, b, t.x0(), t.y0(), t.img);
            tma_tile(a + P.b_off, xmap, b, t.x0() - 1, t.y0() - 1, t.img);
            in.next(), t.next();
            issued++;
        };
        bool ok = true;
        while (issued < S && issued < n) load();
        for (int i = 0; i < n; i++) {
            if (!(ok = mbar_wait(bar(out.slot), out.phase))) break;
            waited = i + 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = base + (uint32_t)out.slot * P.stage_bytes, b = a + P.b_off;
            const uint64_t ad = smem_desc(a, 128u, kGradPlaneBytes);
            for (int q = 0; q < ntaps; q++) {
                const int tap = tap0 + q, dy = tap / 3, dx = tap - 3 * dy;
                const uint32_t d = tmem + (uint32_t)(q * P.cin_pad);
                const uint64_t bd = smem_desc(b + (uint32_t)(dy * kHaloW + dx) * 16u, kRowBytes, kPlaneBytes);
#pragma unroll
                for (int k = 0; k < kTileH / 2; k++)  // two tile rows per step
                    mma(d, ad + k * (256u >> 4), bd + k * (2 * kRowBytes >> 4), idesc, (i == 0 && k == 0) ? 0u : 1u);
            }
            commit(bar(4 + out.slot));
            // refill the stage of the tile before this one, whose MMAs end
            // while this one's run (one stage: this one's own)
            const int prev = S == 1 ? i : i - 1;
            if (prev >= 0 && issued < n) {
                const int slot = S == 1 ? out.slot : (out.slot ? out.slot : S) - 1;
                const uint32_t phase = S == 1 || out.slot ? out.phase : out.phase ^ 1u;
                if (!(ok = mbar_wait(bar(4 + slot), phase))) break;
                load();
            }
            out.next();
        }
        // everything issued completes before the epilogue reads and TMEM is freed
        commit(bar(8));
        ok = mbar_wait(bar(8), 0) && ok;
        *okflag = ok ? 1 : 0;
        if (!ok) {
            // copies still in flight (bounded)
            Ring r(S);
            for (int i = 0; i < issued; i++, r.next())
                if (i >= waited) mbar_wait(bar(r.slot), r.phase);
        }
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool ok = *okflag != 0;
    if (!ok && tid == 0) atomicExch(A.err, 1);
    // epilogue: warp q reads TMEM lanes 32q..32q+31, all columns. With M = 128
    // these are rows (co) 32q..32q+31, with M = 64 the first 16 lanes are rows
    // 16q..16q+15; rows from cout on are zero padding and are not stored
    const int lane = tid & 31, co = P.rows == 64 ? (lane < 16 ? warp * 16 + lane : P.cout) : warp * 32 + lane;
    const bool direct = P.out == P.dw;  // [co][tap][ci]
    for (int q = 0; ok && q < ntaps && warp * (P.rows >> 2) < P.cout; q++) {
        float *dst = direct ? P.out + ((size_t)co * 9 + tap0 + q) * P.cin_pad
                            : P.out + (((size_t)group * 9 + tap0 + q) * P.cout + co) * P.cin_pad;
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(q * P.cin_pad);
        for (int c0 = 0; c0 < P.cin_pad; c0 += 16) {
            uint32_t r[16];
            load_tmem<1>(taddr + c0, r);
            if (co >= P.cout) continue;
            float4 *o = reinterpret_cast<float4 *>(dst + c0);
#pragma unroll
            for (int k = 0; k < 4; k++)
                o[k] = make_float4(__uint_as_float(r[4 * k]), __uint_as_float(r[4 * k + 1]),
                                   __uint_as_float(r[4 * k + 2]), __uint_as_float(r[4 * k + 3]));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(A.p.tmem_cols)
                     : "memory");
    }
}

// The end of a backward pass, one grid of 256-thread blocks:
//   weight gradients: four consecutive input channels per thread; of more
//     than kFinSlices groups, a warp's 32 such elements x 8 slices (slice s
//     adds groups s, s + 8, ..., and the slice sums are added in order), else
//     256 elements, each thread all groups;
//   bias gradients: a block per channel, thread t adds rows t, t + 256, ...,
//     then a fixed tree;
//   the loss (the last block): the same over the loss kernel's block sums.
// The same order on every run.
constexpr int kFinSlices = 8;
struct FinishArgs {
    struct Weights {
        const float *partial;
        float *dw;
        int groups, cout, cin, cin_pad, sliced, first_block;
    } w[kMaxWgrad];
    BiasJob bias[kMaxWgrad];
    int bias_first[kMaxWgrad];
    int nw, nbias;
    const float *l1;
    float *loss;
    float inv;
    int l1_n;
};

__global__ void __launch_bounds__(256) k_grad_finish(const __grid_constant__ FinishArgs A) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float sm[256];
    __shared__ float4 sm4[kFinSlices][32];
    const int tid = (int)threadIdx.x, b = (int)blockIdx.x;
    if (b >= A.bias_first[0]) {
        int j = 0;
        while (j + 1 < A.nbias && A.bias_first[j + 1] <= b) j++;
        const int k = b - A.bias_first[j];
        const bool loss = k >= A.bias[j].c;  // (past the last bias job)
        const int rows = loss ? A.l1_n : A.bias[j].rows;
        float s = 0.f;
        for (int r = tid; r < rows; r += 256) s += loss ? A.l1[r] : A.bias[j].part[(size_t)r * A.bias[j].c + k];
        sm[tid] = s;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (tid < o) sm[tid] += sm[tid + o];
            __syncthreads();
        }
        if (tid == 0) {
            if (loss) A.loss[0] = sm[0] * A.inv;
            else A.bias[j].db[k] = sm[0];
        }
        return;
    }
    int j = 0;
    while (j + 1 < A.nw && A.w[j + 1].first_block <= b) j++;
    const FinishArgs::Weights &W = A.w[j];
    const int lane = tid & 31, slice = W.sliced ? tid >> 5 : 0, step = W.sliced ? kFinSlices : 1;
    const int i = (b - W.first_block) * (W.sliced ? 32 : 256) + (W.sliced ? lane : tid);
    const int quads = W.cin_pad >> 2, total = W.cout * 9 * quads;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [](float4 &a, const float4 &x) { a.x += x.x, a.y += x.y, a.z += x.z, a.w += x.w; };
    const int ci = 4 * (i % quads), rest = i / quads, co = rest % W.cout, tap = rest / W.cout;
    if (i < total) {
        // [group][tap][co][ci]
        const float4 *src = reinterpret_cast<const float4 *>(W.partial) + i;
        for (int g = slice; g < W.groups; g += step) add(v, src[(size_t)g * total]);
    }
    if (W.sliced) {
        sm4[slice][lane] = v;
        __syncthreads();
        if (slice) return;
        for (int k = 1; k < kFinSlices; k++) add(v, sm4[k][lane]);
    }
    if (i < total) {
        float *d = W.dw + ((size_t)co * 9 + tap) * W.cin + ci;
        const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (ci + k < W.cin) d[k] = f[k];
    }
}

// Forward weights: out[tap][chunk][row][8] from w[cout][9][cin] (zero rows and
// channels pad). The backward-data convolution's (bwd), in the same order: the
// input gradient of a 3x3 convolution is a 3x3 convolution of the output
// gradient with the weights transposed (output channel ci, input channel co)
// and the taps mirrored: out[tap][chunk][ci][8] = w[co][8 - tap][ci].
// A thread packs one row of 8 channels (16 bytes) with 32-bit index
// arithmetic. Bound by latency (12 MB at 1,016,419 weights, both ways): one
// element per thread with 64-bit divisions took 22.7 us, this 10.6 us.
__global__ void __launch_bounds__(256) k_pack_all(const TcPackJob *jobs, int njobs, uint32_t rows) {
    __shared__ TcPackJob sj[64];
    for (int i = (int)threadIdx.x; i < njobs; i += (int)blockDim.x) sj[i] = jobs[i];
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows) return;
    int lo = 0, hi = njobs - 1;  // the last job that begins at or before row i
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if ((uint32_t)(sj[mid].begin / 8) <= i) lo = mid;
        else hi = mid - 1;
    }
    const TcPackJob &J = sj[lo];
    const uint32_t row = i - (uint32_t)(J.begin / 8), npad = (uint32_t)J.npad, nchunk = (uint32_t)J.cin_pad / 8;
    const uint32_t ct = row / npad, tap = ct / nchunk;
    const int r = (int)(row - ct * npad), c0 = (int)(ct - tap * nchunk) * 8;
    __nv_bfloat162 v[4];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const int c = c0 + e;
        float f;
        if (!J.bwd)  // row r = output channel, c = input channel
            f = (r < J.cout_f && c < J.cin_f) ? J.w[((size_t)r * 9 + tap) * J.cin_f + c] : 0.f;
        else  // transposed, taps mirrored: row r = input channel, c = output channel
            f = (r < J.cin_f && c < J.cout_f) ? J.w[((size_t)c * 9 + (8 - tap)) * J.cin_f + r] : 0.f;
        if (e & 1) v[e >> 1].y = __float2bfloat16(f);
        else v[e >> 1].x = __float2bfloat16(f);
    }
    uint4 q;
    memcpy(&q, v, 16);
    *reinterpret_cast<uint4 *>(J.out + (size_t)row * 8) = q;
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    }
    return fn;
}

// Tensor map of a planar tensor (n images of h x w, c channels, a multiple of
// 8) for boxes of bw x bh pixels and every chunk: dimensions (8 w, h, c / 8, n).
cudaError_t tile_map(void *out, const __nv_bfloat16 *x, int n, int h, int w, int c, int bw, int bh) {
    EncodeTiled enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    const cuuint64_t px = (cuuint64_t)h * w, chunks = (cuuint64_t)c / 8;
    const cuuint64_t dims[4] = {(cuuint64_t)w * 8, (cuuint64_t)h, chunks, (cuuint64_t)n};
    const cuuint64_t strides[3] = {(cuuint64_t)w * 16, px * 16, px * chunks * 16};
    const cuuint32_t box[4] = {(cuuint32_t)bw * 8, (cuuint32_t)bh, (cuuint32_t)chunks, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = enc(static_cast<CUtensorMap *>(out), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4,
                           const_cast<__nv_bfloat16 *>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace

size_t tc_packed_weight_elems(int cin_pad, int cout) { return (size_t)9 * cin_pad * ((cout + 15) / 16 * 16); }

cudaError_t tc_pack_all(const TcPackJob *jobs_dev, int njobs, size_t total, cudaStream_t st) {
    if (njobs <= 0 || njobs > 64 || total % 8 || total / 8 > 0xFFFFFFFFull - 255) return cudaErrorInvalidValue;
    const uint32_t rows = (uint32_t)(total / 8);
    k_pack_all<<<(rows + 255) / 256, 256, 0, st>>>(jobs_dev, njobs, rows);
    return cudaGetLastError();
}

cudaError_t tc_wgrad_plan(TcWgradPlan &p, const TcWgradConv *convs, int count, int sm_count) {
    std::memset(&p, 0, sizeof(p));
    if (count <= 0 || count > kMaxWgrad) return cudaErrorInvalidValue;
    // two CTAs per SM: half of the shared memory and of the tensor memory each
    constexpr int kCols = 256;
    const size_t budget = kSmemPerSm / 2 - 1024 - 128;
    // clocks of a tile's MMAs of one tap (operands at 128 bytes per clock)
    auto tap_clk = [](const TcWgradJob &j) { return 8.0 * (32 * j.rows + 32 * j.cin_pad) / 128; };
    double total = 0;
    for (int i = 0; i < count; i++) {
        TcWgradJob &j = p.job[i];
        const TcWgradConv &c = convs[i];
        const TcConvPlan &f = *c.fwd;
        j.n = f.n, j.cin = c.cin, j.cin_pad = f.cin, j.cout = c.cout, j.cout_pad = (c.cout + 15) / 16 * 16;
        if (!c.g || !c.dw || c.cin <= 0 || c.cin > j.cin_pad || (j.cin_pad & 15) || j.cin_pad > kCols || c.cout <= 0 ||
            c.cout > 128)
            return cudaErrorInvalidValue;
        j.dw = c.dw;
        j.tiles_x = f.tiles_x, j.tiles_y = f.tiles_y, j.tiles = f.tiles;
        // 64 rows where they suffice: half the operand bytes of A, which bound
        // the MMAs of few input channels
        j.rows = j.cout <= 64 ? 64 : 128;
        // a stage: the rows of A (8 per plane), then the halo planes of B
        j.b_off = (uint32_t)j.rows / 8 * kGradPlaneBytes;
        j.stage_bytes = (j.b_off + (uint32_t)(j.cin_pad / 8) * kPlaneBytes + 1023) & ~1023u;
        if (j.stage_bytes > budget) return cudaErrorInvalidValue;
        j.stages = (int)std::min<size_t>(4, budget / j.stage_bytes);
        std::memcpy(j.xmap, f.tmap, sizeof(j.xmap));
        const cudaError_t e = tile_map(j.gmap, c.g, f.n, f.h, f.w, j.cout_pad, kTileW, kTileH);
        if (e != cudaSuccess) return e;
        total += j.tiles * 9.0 * tap_clk(j);
    }
    // Each convolution's groups of tiles and of taps: the cheapest split, an
    // item costing its MMAs, its copies (64 bytes per clock and 2,600 clocks of
    // latency, beside the MMAs where there is more than one stage), its stores
    // (32 bytes per clock) and about 3,000 clocks to start up and end; items
    // longer than about an SM's share of all MMAs are penalised (the longest
    // one ends the launch). A group has at most seven tiles, or, of more than
    // seven per SM, the tiles that one SM of a launch of its own would get with
    // all of tensor memory: the FP32 sums run over its pixels one after
    // another, and longer chains round worse (257 tiles per group moved the
    // gradients of 8 x 128^2 by 6e-5, relative).
    const double cap = std::max(0.6 * total / sm_count + 4000, 9000.0);
    double cost[kMaxWgrad];
    for (int i = 0; i < count; i++) {
        TcWgradJob &j = p.job[i];
        const double tile_load = (j.cout_pad / 8 * (double)kGradPlaneBytes + j.cin_pad / 8 * (double)kPlaneBytes) / 64;
        double best = -1;
        const int taps512 = std::min(9, 512 / j.cin_pad), passes512 = (9 + taps512 - 1) / taps512;
        const long long chain = std::max(7LL, ((long long)j.tiles * passes512 + sm_count - 1) / sm_count);
        for (int t = 1; t <= 9 && t * j.cin_pad <= kCols; t++)
            for (long long q = 1; q <= chain && q <= j.tiles; q = q < 16 ? q + 1 : q + q / 8) {
                const double m = t * tap_clk(j);
                const double tile =
                    j.stages > 1 ? std::max({m, tile_load, 2600.0 / j.stages}) : m + tile_load + 1600;
                const double item = q * tile + 4.0 * t * j.cin_pad * j.cout / 32 + 3000;
                const int passes = (9 + t - 1) / t, groups = (int)((j.tiles + q - 1) / q);
                // (too long an item counts as if it alone kept its SM)
                const double c = (double)passes * groups * item + std::max(0.0, item - cap) * sm_count +
                                 (groups > 1 ? groups * 9.0 * j.cout * j.cin_pad / 128 : 0.0);
                if (best < 0 || c < best) {
                    best = c, cost[i] = item;
                    j.taps_per_pass = t, j.passes = passes, j.tiles_per_cta = (int)q, j.groups = groups;
                }
            }
    }
    // the longest items first
    for (int i = 1; i < count; i++)
        for (int k = i; k > 0 && cost[k] > cost[k - 1]; k--)
            std::swap(cost[k], cost[k - 1]), std::swap(p.job[k], p.job[k - 1]);
    p.jobs = count;
    int cols = 32;
    for (int i = 0; i < count; i++) {
        TcWgradJob &j = p.job[i];
        j.first_item = p.items;
        p.items += j.passes * j.groups;
        p.bar_off = std::max(p.bar_off, (uint32_t)j.stages * j.stage_bytes);
        while (cols < j.taps_per_pass * j.cin_pad) cols <<= 1;
        j.partial_off = p.partial_floats;
        if (j.groups > 1 || j.cin != j.cin_pad) p.partial_floats += (size_t)j.groups * 9 * j.cout * j.cin_pad;
    }
    p.tmem_cols = cols;
    p.smem = p.bar_off + 9 * 8 + 16;
    // (no more CTAs per SM than TMEM has columns for)
    const size_t max_ctas = 512 / cols;
    if (kSmemPerSm / (p.smem + 1024) > max_ctas) p.smem = kSmemPerSm / max_ctas - 1024 + 16;
    if (p.smem > kSmemMax) p.smem = kSmemMax;
    return cudaSuccess;
}

void tc_wgrad_place(TcWgradPlan &p, float *partial) {
    for (int i = 0; i < p.jobs; i++) {
        TcWgradJob &j = p.job[i];
        j.out = j.groups > 1 || j.cin != j.cin_pad ? partial + j.partial_off : j.dw;
    }
}

namespace {

// Launches with programmatic stream serialisation: the kernel's prologue may
// overlap the previous kernel, which it waits for itself.
template <class Kernel, class Args>
cudaError_t launch_overlapped(Kernel kernel, unsigned grid, unsigned block, size_t smem, cudaStream_t st, const Args &a) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(grid), cfg.blockDim = dim3(block), cfg.dynamicSmemBytes = smem, cfg.stream = st;
    cfg.attrs = attr, cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace

cudaError_t wgrad_all_tc(const TcWgradPlan &p, int *err, cudaStream_t st) {
    if (p.jobs <= 0 || !p.job[0].out) return cudaErrorInvalidValue;
    static std::atomic<uint64_t> attr_set{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (!bit || !(attr_set.load() & bit)) {
        e = cudaFuncSetAttribute(k_wgrad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
        if (e != cudaSuccess) return e;
        attr_set.fetch_or(bit);
    }
    WgArgs a;
    a.p = p;
    a.err = err;
    return launch_overlapped(k_wgrad_tc, (unsigned)p.items, 128, p.smem, st, a);
}

cudaError_t grad_finish(const TcWgradPlan &p, const BiasJob *bias, int nbias, const float *l1, int l1_n, float *loss,
                        float inv, cudaStream_t st) {
    if (nbias <= 0 || nbias > kMaxWgrad) return cudaErrorInvalidValue;
    FinishArgs a;
    std::memset(&a, 0, sizeof(a));
    int blocks = 0;
    for (int i = 0; i < p.jobs; i++) {
        const TcWgradJob &j = p.job[i];
        if (j.out == j.dw) continue;
        FinishArgs::Weights &w = a.w[a.nw++];
        w.partial = j.out, w.dw = j.dw;
        w.groups = j.groups, w.cout = j.cout, w.cin = j.cin, w.cin_pad = j.cin_pad;
        w.sliced = j.groups > kFinSlices ? 1 : 0;
        w.first_block = blocks;
        const int per_block = w.sliced ? 32 : 256;
        blocks += (j.cout * 9 * (j.cin_pad / 4) + per_block - 1) / per_block;
    }
    for (int i = 0; i < nbias; i++) {
        a.bias[i] = bias[i];
        a.bias_first[i] = blocks;
        blocks += bias[i].c;
    }
    a.nbias = nbias;
    a.l1 = l1, a.l1_n = l1_n, a.loss = loss, a.inv = inv;
    return launch_overlapped(k_grad_finish, (unsigned)blocks + 1, 256, 0, st, a);
}

cudaError_t tc_conv_plan(TcConvPlan &p, const __nv_bfloat16 *x, int n, int h, int w, int cin, int cout, bool relu,
                         int sm_count, bool grad) {
    std::memset(&p, 0, sizeof(p));
    if (n <= 0 || h <= 0 || w <= 0 || cin <= 0 || (cin & 15) || cout <= 0 ||
        !(cin <= 128 || cin == 160 || cin == 224))  // (the pair counts that issue() unrolls)
        return cudaErrorInvalidValue;
    p.x = x, p.n = n, p.h = h, p.w = w, p.cin = cin, p.cout = cout, p.relu = relu ? 1 : 0;
    p.npad = (cout + 15) / 16 * 16;
    if (p.npad > 256) return cudaErrorInvalidValue;
    p.tiles_x = (w + kTileW - 1) / kTileW;
    p.tiles_y = (h + kTileH - 1) / kTileH;
    const long long tiles = (long long)n * p.tiles_x * p.tiles_y;
    if (tiles > 0x7FFFFFFFLL) return cudaErrorInvalidValue;
    p.tiles = (int)tiles;
    p.npad_full = p.npad;
    // The split: a chunk width cw of the output channels (every CTA loads whole
    // halos, so narrower chunks cost loads, and an MMA below N = 32 is no
    // faster), one or two CTAs per SM, the weights resident or streamed. Taken
    // is the one with the shortest estimate in clocks: per tile the larger of
    // the SM's MMAs (operands at 128 bytes per clock, N / 2 clocks at least), its
    // copies at 64 bytes per clock and its epilogue (kEpiClk), for the tiles that fall to one SM, plus the
    // first tile's copies.
    const int pairs = cin / 16;
    constexpr double kEpiClk = 14.0;   // clocks per channel of a tile for one CTA's epilogue warps
    constexpr double kRoleClk = 450.0; // what a CTA's MMA thread spends per tile besides the MMAs
    const size_t halo = ((size_t)(cin / 8) * kPlaneBytes + 127) & ~(size_t)127;  // TMA destinations: 128-byte aligned
    double best = 0;
    for (int cw = 16; cw <= p.npad_full; cw += 16) {
        if (p.npad_full % cw) continue;
        const int nsplit = p.npad_full / cw;
        const size_t wtap = (size_t)cin * cw * 2;
        const int stride = (cw + 31) & ~31;
        for (int per_sm = 1; per_sm <= 2; per_sm++) {
            const long long slots = (long long)sm_count * per_sm / nsplit;
            if (slots < 1) continue;
            const long long ctas = tiles < slots ? tiles : slots, items = (tiles + ctas - 1) / ctas;
            int acc = items > 2 ? 4 : items > 1 ? 2 : 1, cols = 32;
            while (acc > 1 && acc * stride * per_sm > 512) acc--;
            while (cols < acc * stride) cols <<= 1;
            if (cols * per_sm > 512) continue;
            const size_t budget = per_sm == 2 ? kSmemPerSm / 2 - 1024 : kSmemMax;
            const size_t misc = 4 * (size_t)cw * (grad ? kEpiWarps : 1) + 8 * (2 * 4 + 2 * 4 + 2 * kTaps + 1) + 64;
            for (int wst = kTaps; wst >= 3; wst--) {
                const size_t rest = misc + wst * wtap;
                if (rest + halo > budget) continue;
                long long ring = (long long)((budget - rest) / halo);
                if (ring > items) ring = items;
                if (ring > 4) ring = 4;
                const double mma = kTaps * pairs * (cw / 4 + 32 > cw / 2 ? cw / 4 + 32 : cw / 2);
                const double load = ((double)halo + (wst < kTaps ? kTaps * wtap : 0)) / 64, epi = cw * kEpiClk;
                double on_sm = (double)(ctas * nsplit + sm_count - 1) / sm_count;  // CTAs of the busiest SM
                if (on_sm > per_sm) on_sm = per_sm;
                double tile = std::max(on_sm * std::max(mma, load), std::max(mma + kRoleClk, epi));
                if (ring == 1 && items > 1) tile += load / 2 + 600;  // nothing loaded beside the MMAs
                double cost = items * tile + (halo + wst * wtap) / 64.0;
                // small enough for the next kernel's CTAs to start up beside this one's
                if (rest + ring * halo > kSmemPerSm / 2 - 1024) cost += 600;
                if (best == 0 || cost < best) {
                    best = cost;
                    p.npad = cw, p.nsplit = nsplit, p.grid = (int)ctas, p.wstages = wst, p.ring = (int)ring;
                    p.acc_slots = acc, p.acc_stride = stride, p.tmem_cols = cols;
                }
                break;  // fewer weight slots never help
            }
        }
    }
    if (best == 0) return cudaErrorInvalidValue;
    const size_t wtap = (size_t)cin * p.npad * 2;
    p.halo_stride = (uint32_t)halo;
    p.w_off = (uint32_t)(p.ring * halo);
    p.bias_off = (uint32_t)(p.w_off + p.wstages * wtap);
    p.bar_off = (p.bias_off + 4 * (uint32_t)p.npad * (grad ? kEpiWarps : 1) + 15) & ~15u;
    p.grad = grad ? 1 : 0;
    p.smem = p.bar_off + 8 * (2 * (size_t)p.ring + 2 * (size_t)p.acc_slots + 2 * (size_t)p.wstages + 1) + 32;
    // no more CTAs per SM than TMEM has columns for (tcgen05.alloc would wait)
    const size_t max_ctas = 512 / p.tmem_cols;
    if (kSmemPerSm / (p.smem + 1024) > max_ctas) p.smem = kSmemPerSm / max_ctas - 1024 + 16;
    if (p.smem > kSmemMax) p.smem = kSmemMax;
    return tile_map(p.tmap, x, n, h, w, cin, kHaloW, kHaloH);
}

cudaError_t conv3x3_forward_tc(const TcConvPlan &p, const __nv_bfloat16 *wpacked, const float *bias,
                               __nv_bfloat16 *y, float *y32, int *err, cudaStream_t st, const TcFuse *fuse,
                               bool overlap_prologue) {
    if (y && (p.cout & 15)) return cudaErrorInvalidValue;
    if (!bias && !(fuse && fuse->grad != kGradNone)) return cudaErrorInvalidValue;
    if (fuse) {
        if ((fuse->pool || fuse->cat) && (p.cout & 15)) return cudaErrorInvalidValue;
        if (fuse->cat && (fuse->cat_c & 7 || fuse->cat_off & 7 || fuse->cat_off + p.cout > fuse->cat_c))
            return cudaErrorInvalidValue;
        // one of: pooling with the copy into a concatenation, upsampling, FP32
        if ((fuse->pool != nullptr) != (fuse->cat && !fuse->cat_up)) return cudaErrorInvalidValue;
        if ((y32 || fuse->rad) && (y || fuse->cat)) return cudaErrorInvalidValue;
        if (fuse->grad != kGradNone) {
            if (!p.grad || y || y32 || fuse->cat || fuse->rad || (p.cout & 15) || !fuse->mask || !fuse->g ||
                !fuse->bias_part || (fuse->grad != kGradMask && !fuse->skip))
                return cudaErrorInvalidValue;
            if (fuse->grad == kGradCat && ((fuse->low_c & 15) || fuse->low_c > p.cout || ((p.h | p.w) & 1)))
                return cudaErrorInvalidValue;
        }
        if (fuse->res && (p.cout > 4 || (!y32 && !fuse->rad))) return cudaErrorInvalidValue;
        if (fuse->rad && (p.cout != 3 || !fuse->feat)) return cudaErrorInvalidValue;
    }
    // the shared-memory opt-in is a per-device setting of each kernel: once per device
    static std::atomic<uint64_t> attr_set{0};
    int dev = 0;
    cudaError_t e0 = cudaGetDevice(&dev);
    if (e0 != cudaSuccess) return e0;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (!bit || !(attr_set.load() & bit)) {
        for (auto k : {k_conv_tc<kEpiY>, k_conv_tc<kEpiPool>, k_conv_tc<kEpiUp>, k_conv_tc<kEpiF32>,
                       k_conv_tc<kEpiGradMask>, k_conv_tc<kEpiGradCat>, k_conv_tc<kEpiGradUnpool>}) {
            const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
            if (e != cudaSuccess) return e;
        }
        attr_set.fetch_or(bit);
    }
    TcArgs a;
    a.w = wpacked, a.bias = bias;
    a.y = y, a.y32 = y32;
    a.n = p.n, a.h = p.h, a.wd = p.w, a.cin = p.cin, a.cout = p.cout, a.npad = p.npad, a.relu = p.relu;
    a.tiles_x = p.tiles_x, a.tiles_y = p.tiles_y;
    a.ring = p.ring, a.wstages = p.wstages, a.nsplit = p.nsplit;
    a.acc_slots = p.acc_slots, a.acc_stride = p.acc_stride, a.tmem_cols = p.tmem_cols;
    a.halo_stride = p.halo_stride, a.w_off = p.w_off, a.bias_off = p.bias_off, a.bar_off = p.bar_off;
    a.err = err;
    if (fuse) a.f = *fuse;
    CUtensorMap map, wmap;
    std::memcpy(&map, p.tmap, sizeof(map));
    std::memset(&wmap, 0, sizeof(wmap));
    if (p.nsplit > 1) {
        // the packed weights [tap][chunk][npad_full rows][8] as a 3-D map:
        // (8 channels, rows, tap x chunk); each CTA loads rows n0..n0+npad
        EncodeTiled enc = encode_fn();
        if (!enc) return cudaErrorNotSupported;
        const cuuint64_t dims[3] = {8, (cuuint64_t)p.npad_full, (cuuint64_t)9 * (p.cin / 8)};
        const cuuint64_t strides[2] = {16, (cuuint64_t)p.npad_full * 16};
        const cuuint32_t box[3] = {8, (cuuint32_t)p.npad, (cuuint32_t)(p.cin / 8)};  // one tap
        const cuuint32_t estr[3] = {1, 1, 1};
        const CUresult r = enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16 *>(wpacked), dims,
                               strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cfg.attrs = overlap_prologue ? attr : nullptr;
    cfg.numAttrs = overlap_prologue ? 1 : 0;
    cfg.gridDim = dim3((unsigned)p.grid, (unsigned)p.nsplit), cfg.blockDim = dim3(kConvThreads);
    const bool f32 = y32 || (fuse && fuse->rad), pool = fuse && fuse->pool, cat = fuse && fuse->cat;
    const int grad = fuse ? fuse->grad : kGradNone;
    const cudaError_t e = cudaLaunchKernelEx(
        &cfg,
        grad == kGradMask     ? k_conv_tc<kEpiGradMask>
        : grad == kGradCat    ? k_conv_tc<kEpiGradCat>
        : grad == kGradUnpool ? k_conv_tc<kEpiGradUnpool>
        : f32 ? k_conv_tc<kEpiF32> : pool ? k_conv_tc<kEpiPool> : cat ? k_conv_tc<kEpiUp> : k_conv_tc<kEpiY>, map,
        wmap, a);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace dn
}  // namespace pray_gpu
