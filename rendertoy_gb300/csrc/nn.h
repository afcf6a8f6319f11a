// nn.h — the denoiser's device operators (NHWC BF16 tensors, channel counts
// padded to multiples of 8; convolutions on the tcgen05 tensor cores).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace rtx {
namespace nn {

using bf16 = __nv_bfloat16;

// Network input and output records.
//   raw input, FP32 per pixel: radiance 3 (linear), albedo 3, normal 3 (as the
//   normal pass encodes it), depth 1, and the radiance's samples per pixel 1
//   (the same value over a frame; it tells the network how noisy the
//   radiance is).
//   prediction, FP32 per pixel: kKpTaps filter logits (padded to kPredCh).
//   The denoised radiance is the softmax of the logits applied to the
//   kKpWidth x kKpWidth neighbourhood of the input radiance (taps clamped to
//   the frame): a kernel-predicting output (Bako et al., SIGGRAPH 2017),
//   which can only average input pixels and so approaches its input as the
//   input's noise vanishes.
constexpr int kRawCh = 11;
constexpr int kKpWidth = 5;
constexpr int kKpTaps = kKpWidth * kKpWidth;
constexpr int kPredCh = 32;
// Loss: relative squared error with the prediction (not differentiated) in
// the denominator, (o - t)^2 / (o^2 + kRelEps): its minimiser over noisy
// targets is their mean, so unbiased targets of any noise level train it
// toward the clean image.
constexpr float kRelEps = 1e-2f;

// One input of a convolution: C channels; `up` = stored at half resolution
// and read upsampled (nearest) to the convolution's resolution.
struct Src {
  const bf16* ptr;
  int C;
  int up;
};

struct ConvFwd {
  Src s1, s2;        // s2.ptr == nullptr: single source
  int N, H, W;       // convolution (output) resolution
  int Cin;           // s1.C + s2.C
  int Cout;          // multiple of 16, <= 256
  const bf16* w;     // [Cout][9][Cin]
  const float* bias; // [Cout] or nullptr
  int relu;
  bf16* out;         // [P][Cout] or nullptr
  float* out_f32;    // [P][Cout] or nullptr
  int* err;
  // [P / 4][Cout] or nullptr: the output's 2 x 2 averages, written beside it
  // (tile kernels, a full-resolution source, even H and W)
  bf16* pool = nullptr;
};

// The kernel-predicting output layer together with what its logits are for:
// the filtered radiance (out), or the loss and its gradient (dpred, loss).
struct KpHead {
  const float* rad;     // radiance of frames stored Hs x Ws, rad_px floats per pixel (RGB first)
  int rad_px, Hs, Ws;
  int Hc, Wc;           // frame the taps are clamped to (out: [N][Hc][Wc][3])
  float* out;
  const float* target;  // [N][H][W][3]; H = Hc, W = Wc
  bf16* dpred;          // [P][kPredCh]
  double* loss;         // += the summed loss
  float inv;            // 1 / (3 P)
};

struct ConvDgrad {
  const bf16* dout;  // [P][Cout]
  int Cout;
  const bf16* wt;    // [Cin][9][Cout]
  int N, H, W, Cin;  // Cin multiple of 16
  Src s1, s2;        // the sources (read for the ReLU mask)
  int mask_relu;
  bf16* din;         // [P][Cin] (s1's channels upsampled when s1.up)
  int* err;
  // Both given (tile kernels, s1 upsampled and s2 a skip source): instead of din, s1's
  // channels go to dlow [P / 4][C1], summed over each 2 x 2 block (nearest
  // upsampling's gradient), and s2's to dskip [P][C2].
  bf16 *dlow = nullptr, *dskip = nullptr;
};

struct ConvWgrad {
  const bf16* dout;  // [P][Cout]
  int Cout;
  Src s1, s2;
  int N, H, W, Cin;
  float* dw;         // [Cout][9][Cin], accumulated
  int* err;
  float* db = nullptr;  // [Cout] or nullptr: the bias gradient, accumulated
};

cudaError_t conv_fwd(const ConvFwd& a, cudaStream_t st);
// The output layer with its head in one launch; false: not a shape it takes
// (rows of at least 64 pixels), nothing launched.
bool conv_head(const ConvFwd& a, const KpHead& h, cudaStream_t st, cudaError_t* e);
cudaError_t conv_dgrad(const ConvDgrad& a, cudaStream_t st);
cudaError_t conv_wgrad(const ConvWgrad& a, cudaStream_t st);

}  // namespace nn
}  // namespace rtx
