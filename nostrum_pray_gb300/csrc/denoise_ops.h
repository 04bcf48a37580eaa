// Denoiser layer launchers (denoise_ops.cu). NHWC tensors; n images of
// h x w pixels. Gradient outputs: conv3x3_backward writes dx and adds into
// dw / db; avgpool_backward and split_add add into gx; upsample_backward
// writes gx.
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace pray_gpu {
namespace dn {

// tcgen05 tensor-core version (denoise_tc.cu). Its BF16 tensors are planar in
// 8-channel chunks: [image][channel / 8][y][x][8] (the CUDA-core kernels'
// tensors are channels last). A plan holds the input's TMA tensor map (the
// input buffer is fixed) and the launch shape; Cin must be a multiple of 16
// (pack_input pads the network input), the weights packed by tc_pack_all
// (cin_pad = Cin of the plan). *err is set to 1 if one of the kernel's bounded
// mbarrier waits ran out.
struct TcConvPlan {
    alignas(64) unsigned char tmap[128];  // CUtensorMap of x: (8 W, H, C / 8, N), box (80, 18, C / 8, 1)
    const __nv_bfloat16 *x;
    int n, h, w, cin, cout, npad, relu;
    int tiles_x, tiles_y, tiles;
    int nsplit, npad_full;        // output-channel chunks of npad channels each, of npad_full
    int grid;                     // persistent CTAs of each chunk
    int ring, wstages;            // halo slots; weight slots of a tap each (9: all resident)
    int acc_slots, acc_stride, tmem_cols;
    int grad;                     // planned for TcFuse::grad
    uint32_t halo_stride, w_off, bias_off, bar_off;
    size_t smem;
};
cudaError_t tc_conv_plan(TcConvPlan &p, const __nv_bfloat16 *x, int n, int h, int w, int cin, int cout, bool relu,
                         int sm_count, bool grad = false);
size_t tc_packed_weight_elems(int cin_pad, int cout);
// Every packing of a network's weights in one launch: job j packs w (the
// FP32 [cout_f][9][cin_f] weights of one convolution) into out, for the
// forward convolution (bwd 0: cin_pad = cin_f rounded up to 16, npad = cout_f
// rounded up) or for its backward-data convolution (bwd 1: cin_pad = cout_f
// rounded up, npad = cin_f rounded up): a plan with cin = cout_f rounded up to
// 16 and cout = cin_f that runs on the output gradient (BF16, planar) and
// gives the input gradient. Its 9 x cin_pad x npad elements start at `begin`
// of the concatenated range, jobs in increasing begin (at most 64).
struct TcPackJob {
    const float *w;
    __nv_bfloat16 *out;
    unsigned long long begin;
    int cin_f, cout_f, cin_pad, npad, bwd;
};
cudaError_t tc_pack_all(const TcPackJob *jobs_dev, int njobs, size_t total, cudaStream_t st);
// Extra stores of a forward convolution's epilogue, so that the network's
// pooling, upsampling + concatenation, residual and output transform need no
// kernels of their own. Each takes the values exactly as the separate kernel
// would (the BF16-rounded outputs; the FP32 output plus the residual), so the
// results are the same bits.
//   pool: the 2 x 2 average of the BF16 outputs, (h / 2) x (w / 2) x cout;
//   cat:  the BF16 outputs also into channels [cat_off, cat_off + cout) of a
//         cat_c-channel tensor, at the same pixel (cat_up 0) or, nearest 2x
//         upsampling, at the 2 x 2 block of a 2h x 2w tensor (cat_up 1);
//   res:  FP32 output += res[pixel * res_c + channel] (BF16);
//   rad:  (cout 3) rad = expm1(FP32 output) * (max(albedo, 0) + kDemodFloor),
//         the albedo from feat (7 halves per pixel);
//   grad: for a backward-data convolution, whose FP32 output is the gradient
//         of the forward convolution's input tensor: what the next one down
//         the chain reads, the gradient masked by the ReLU of that tensor
//         (mask: its BF16 values, planar) and rounded to BF16 (g, planar), with
//         per-CTA sums of the masked FP32 values (bias_part: grid x channels of
//         g, for the bias gradient).
//         kGradMask: the input is itself a convolution's output;
//         kGradCat: it is a concatenation; of channels [0, low_c) the sums over
//         2 x 2 blocks (mask, g: h / 2 x w / 2, low_c channels), the others as
//         they are into skip (FP32, planar);
//         kGradUnpool: it is the 2 x 2 average of a tensor whose other share of
//         the gradient is skip (mask, g, skip: 2h x 2w): skip + output / 4.
// pool and cat need cout a multiple of 16; pool comes with cat at the same
// pixel; res (cout at most 4) goes with rad or the FP32 output, which take no
// other store.
struct TcFuse {
    __nv_bfloat16 *pool = nullptr;
    __nv_bfloat16 *cat = nullptr;
    int cat_c = 0, cat_off = 0, cat_up = 0;
    const __nv_bfloat16 *res = nullptr;
    int res_c = 0;
    float *rad = nullptr;
    const __half *feat = nullptr;
    int grad = 0;
    const __nv_bfloat16 *mask = nullptr;
    __nv_bfloat16 *g = nullptr;
    float *skip = nullptr, *bias_part = nullptr;
    int low_c = 0;
};
enum { kGradNone = 0, kGradMask, kGradCat, kGradUnpool };
cudaError_t conv3x3_forward_tc(const TcConvPlan &p, const __nv_bfloat16 *wpacked, const float *bias,
                               __nv_bfloat16 *y, float *y32, int *err, cudaStream_t st,
                               const TcFuse *fuse = nullptr, bool overlap_prologue = false);
// y: the BF16 output (planar, cout a multiple of 16), y32: the FP32 output
// (channels last); either may be NULL.
// overlap_prologue: launch with programmatic stream serialisation, so that the
// kernel's prologue (barriers, tensor memory, weight copies) overlaps the
// previous kernel of the stream; its input copies wait for that kernel to
// complete. The previous kernel must not write the weights or the bias.
// Weight gradients of a network's 3x3 convolutions on the tensor cores:
// dw[co][tap][ci] = sum over pixels p of g[p][co] * x[p + offset(tap)][ci],
// per tap a GEMM with M = output channels (padded to 64 or 128), N = input channels,
// K = pixels. g: the output gradient as BF16 with cout rounded up to 16
// channels (planar); x: the convolution's input, read through a forward
// plan's tensor map. One launch serves every convolution: its CTAs are items
// (convolution, group of tiles, group of taps); an item's sums go to `partial`
// per group of tiles, or, where one group holds every tile, straight to dw.
// grad_finish adds the groups in order, sums the bias gradients' rows and
// makes the loss, in one launch.
constexpr int kMaxWgrad = 24;
struct TcWgradJob {
    alignas(64) unsigned char gmap[128];  // CUtensorMap of g: (8 W, H, cout_pad / 8, N), box (64, 16, cout_pad / 8, 1)
    alignas(64) unsigned char xmap[128];  // the forward plan's
    float *dw, *out;                      // out: partial sums [group][9][cout][cin_pad], or dw (one group)
    int n, cin, cin_pad, cout, cout_pad, rows, tiles_x, tiles_y, tiles;  // rows: M
    int tiles_per_cta, groups, taps_per_pass, passes, stages, first_item;
    uint32_t b_off, stage_bytes;
    size_t partial_off;
};
struct TcWgradPlan {
    TcWgradJob job[kMaxWgrad];  // in the order of their items
    int jobs, items, tmem_cols;
    uint32_t bar_off;
    size_t smem, partial_floats;
};
// One convolution of a plan to be made.
struct TcWgradConv {
    const __nv_bfloat16 *g;
    const TcConvPlan *fwd;  // a plan over x with cin = cin_pad
    int cin, cout;
    float *dw;
};
cudaError_t tc_wgrad_plan(TcWgradPlan &p, const TcWgradConv *convs, int count, int sm_count);
// Places the partial sums (partial_floats floats).
void tc_wgrad_place(TcWgradPlan &p, float *partial);
cudaError_t wgrad_all_tc(const TcWgradPlan &p, int *err, cudaStream_t st);
// Bias gradient: db[k] = the sum over rows of part[row * c + k].
struct BiasJob {
    const float *part;
    float *db;
    int rows, c;
};
// After wgrad_all_tc: the group sums, the bias gradients, and the loss as inv
// times the sum of l1[0..l1_n).
cudaError_t grad_finish(const TcWgradPlan &p, const BiasJob *bias, int nbias, const float *l1, int l1_n, float *loss,
                        float inv, cudaStream_t st);
cudaError_t conv3x3_forward(const __nv_bfloat16 *x, const __nv_bfloat16 *w, const float *b, __nv_bfloat16 *y,
                            float *y32, int n, int h, int wd, int cin, int cout, bool relu, cudaStream_t st);
// gpre: output gradient after the ReLU mask (FP32, n*h*w*cout); dx may be NULL
cudaError_t conv3x3_backward(const __nv_bfloat16 *x, const __nv_bfloat16 *w, const float *gpre, float *dx, float *dw,
                             float *db, int n, int h, int wd, int cin, int cout, cudaStream_t st);
cudaError_t relu_mask(const __nv_bfloat16 *y, const float *g, float *out, size_t n, cudaStream_t st);
cudaError_t avgpool(const __nv_bfloat16 *x, __nv_bfloat16 *y, int n, int h, int w, int c, cudaStream_t st);
cudaError_t avgpool_backward(const float *gy, float *gx, int n, int h, int w, int c, cudaStream_t st);
cudaError_t upsample_backward(const float *gy, float *gx, int n, int h, int w, int c, int cy, cudaStream_t st);
cudaError_t split_add(const float *gy, float *gx, size_t pixels, int c, int cy, int off, cudaStream_t st);
// Radiance is demodulated by the first-hit albedo: divided by
// max(albedo, 0) + kDemodFloor (per channel) on the way in and in the loss's
// target, multiplied back on the way out.
constexpr float kDemodFloor = 0.05f;
// x (may be NULL): 10 channels; x16 (may be NULL): the same padded to 16
// channels, planar (images of px pixels)
cudaError_t pack_input(const float *rad, const __half *feat, __nv_bfloat16 *x, __nv_bfloat16 *x16, size_t pixels,
                       size_t px, cudaStream_t st);
// cat = [nearest 2x upsampling of low (c channels, h x w), skip (cs channels)]
cudaError_t upsample_concat(const __nv_bfloat16 *low, const __nv_bfloat16 *skip, __nv_bfloat16 *cat, int n, int h,
                            int w, int c, int cs, cudaStream_t st);
// L1 loss (mean over the n values, into loss[0]) and its gradient; part:
// scratch of kL1Parts floats (per-block sums, added in a fixed order)
constexpr int kL1Parts = 152 * 32;
cudaError_t l1_loss(const float *out, const float *target, const __half *feat, float *g, float *loss, float *part,
                    size_t n, cudaStream_t st);
// The same for the tensor-core backward: the gradient of each pixel's three
// values as BF16, planar, padded to 16 channels (images of px pixels); per
// block the sum of the |differences| in part[block] and of the three gradients
// in part[kL1Blocks + 3 block + k] (part: 4 kL1Blocks floats, l1_blocks(pixels)
// blocks); grad_finish adds them.
constexpr int kL1Blocks = 608;
int l1_blocks(size_t pixels);
cudaError_t l1_loss_tc(const float *out, const float *target, const __half *feat, __nv_bfloat16 *g, float *part,
                       size_t pixels, size_t px, cudaStream_t st);
// out (3 channels) += the first 3 of x0's x0_c channels (the input's log radiance)
cudaError_t add_input(float *out, const __nv_bfloat16 *x0, int x0_c, size_t pixels, cudaStream_t st);
cudaError_t expm1_out(const float *out, const __half *feat, float *rad, size_t n, cudaStream_t st);
cudaError_t adam(float *w, const float *g, float *m, float *v, __nv_bfloat16 *wb, size_t n, float lr, float b1,
                 float b2, float eps, int step, cudaStream_t st);
cudaError_t to_bf16(const float *a, __nv_bfloat16 *b, size_t n, cudaStream_t st);

}  // namespace dn
}  // namespace pray_gpu
