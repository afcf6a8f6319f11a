// nn_ops.h — launchers of the denoiser's memory-bound operators (nn_ops.cu).
#pragma once
#include "nn.h"

namespace rtx {
namespace nn {

cudaError_t encode_input(const float* raw, bf16* x, long long P, cudaStream_t st);
cudaError_t pool_grad_acc(const bf16* dpool, const bf16* skip, bf16* dskip, int N, int H, int W, int C,
                          cudaStream_t st);
// loss of the kernel-predicting output of N frames of H x W (see nn.h);
// adds the summed per-pixel, per-channel loss to *loss
cudaError_t kp_loss(const float* pred, const float* raw, const float* target, bf16* dpred, int N, int H,
                    int W, double* loss, cudaStream_t st);
cudaError_t adam(float* p, const float* g, float* m, float* v, long long n, float lr, int step,
                 cudaStream_t st);
cudaError_t weights_bf16(const float* master, bf16* w, bf16* wt, int Cout, int Cin, cudaStream_t st);
// Several layers' BF16 weights w [Cout][9][Cin] and transposes wt [Cin][9][Cout]
// from their FP32 masters in one launch
struct WeightLayouts {
  static constexpr int kMax = 16;
  int n = 0;
  const float* master[kMax];
  bf16* w[kMax];
  bf16* wt[kMax];
  int Cout[kMax], Cin[kMax];
};
cudaError_t weights_bf16_all(const WeightLayouts& layers, cudaStream_t st);
// out [N][Hc][Wc][3] = the predicted filters applied to the input radiance of
// frames stored as Hs x Ws pixels (pred and raw share that layout)
cudaError_t kp_apply(const float* pred, const float* raw, float* out, int N, int Hc, int Wc, int Hs, int Ws,
                     cudaStream_t st);
// the same for one W x H frame given as its radiance pass; pred rows are Wp
// pixels apart
cudaError_t kp_apply_passes(const float* pred, const float* rad, float* out, int W, int H, int Wp, cudaStream_t st);
// the renderer's passes (W x H RGB FP32 each) and their samples per pixel ->
// the encoded input [Hp][Wp][16], that of a zero record outside the frame
cudaError_t encode_passes(const float* rad, const float* alb, const float* nrm, const float* dep, float spp, bf16* x,
                          int W, int H, int Wp, int Hp, cudaStream_t st);

}  // namespace nn
}  // namespace rtx
