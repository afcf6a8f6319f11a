// nn_ops.cu — the denoiser's memory-bound operators: input encoding, 2 x 2
// average pooling and its gradient, the gradient of nearest upsampling and of
// channel concatenation, the kernel-predicting output with its relative-L2
// loss, bias gradients, Adam and the BF16 weight layouts the convolutions
// read.  One thread per 8 channels of a pixel (16-byte BF16 accesses) unless
// noted.
#include <algorithm>

#include "nn.h"
#include "nn_ops.h"

namespace rtx {
namespace nn {

namespace {

__device__ __forceinline__ void ld8(const bf16* p, float* f) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ void st8(bf16* p, const float* f) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}

unsigned blocks(long long n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// A radiance value made safe to filter and to learn from: NaN and negative
// values (the renderer's rare NaN pixels) read 0, +inf reads the BF16 range.
__device__ __forceinline__ float sane(float v) { return fminf(fmaxf(v, 0.0f), 65504.0f); }

// Pixel (n, y, x) of frames of Hs x Ws stored pixels, RGB of its raw record
template <int kPx = kRawCh>
__device__ __forceinline__ void raw_rgb(const float* raw, long long pix, float* c) {
  const float* r = raw + (long long)kPx * pix;
  c[0] = sane(r[0]);
  c[1] = sane(r[1]);
  c[2] = sane(r[2]);
}

// Softmax of the pixel's kKpTaps logits (max subtracted first); the logits
// are read as seven 16-byte loads (the record is kPredCh = 32 floats, 128-byte
// aligned).
__device__ __forceinline__ void kp_weights(const float* __restrict__ logits_g, float* w) {
  static_assert(kPredCh % 4 == 0 && kKpTaps <= 28 && kPredCh >= 28, "seven float4 of logits");
  float logits[28];
  const float4* l4 = reinterpret_cast<const float4*>(logits_g);
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    const float4 v = __ldg(l4 + i);
    logits[4 * i] = v.x;
    logits[4 * i + 1] = v.y;
    logits[4 * i + 2] = v.z;
    logits[4 * i + 3] = v.w;
  }
  float m = logits[0];
#pragma unroll
  for (int k = 1; k < kKpTaps; ++k) m = fmaxf(m, logits[k]);
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < kKpTaps; ++k) {
    w[k] = expf(logits[k] - m);
    s += w[k];
  }
  const float inv = 1.0f / s;
#pragma unroll
  for (int k = 0; k < kKpTaps; ++k) w[k] *= inv;
}

// Tap k of pixel (x, y) of an Hc x Wc frame stored with row stride Ws:
// offset (k / kKpWidth - r, k % kKpWidth - r), clamped to the frame.
__device__ __forceinline__ long long kp_tap(long long frame0, int x, int y, int k, int Wc, int Hc, int Ws) {
  constexpr int r = kKpWidth / 2;
  const int ty = min(max(y + k / kKpWidth - r, 0), Hc - 1);
  const int tx = min(max(x + k % kKpWidth - r, 0), Wc - 1);
  return frame0 + (long long)ty * Ws + tx;
}

}  // namespace

// One pixel's encoded input: radiance as log(1 + x), albedo, normal and depth
// as they are, the samples per pixel as log2(spp) / 16, channels 11..15 zero
__device__ __forceinline__ void encode_px(const float* r, bf16* x) {
  float f[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) f[i] = 0.0f;
#pragma unroll
  for (int i = 0; i < 3; ++i) f[i] = log1pf(sane(r[i]));
#pragma unroll
  for (int i = 3; i < 10; ++i) f[i] = r[i];
  f[10] = log2f(fmaxf(r[10], 1.0f)) * (1.0f / 16.0f);
  st8(x, f);
  st8(x + 8, f + 8);
}

// raw [P][kRawCh] -> [P][16] BF16
__global__ void k_encode_input(const float* __restrict__ raw, bf16* __restrict__ x, long long P) {
  long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= P) return;
  const float* r = raw + (long long)kRawCh * p;
  float f[kRawCh];
#pragma unroll
  for (int i = 0; i < kRawCh; ++i) f[i] = r[i];
  encode_px(f, x + 16 * p);
}

// The same from the renderer's passes, without the 44-byte records in between
// (1920 x 1080: 87 us of packing and 25 of encoding -> 27 us; its 168 MB take
// 25 us).
__global__ void k_encode_passes(const float* __restrict__ rad, const float* __restrict__ alb,
                                const float* __restrict__ nrm, const float* __restrict__ dep, float spp,
                                bf16* __restrict__ x, int W, int H, int Wp) {
  const int px = blockIdx.x * blockDim.x + threadIdx.x, py = blockIdx.y;
  if (px >= Wp) return;
  float f[kRawCh];
#pragma unroll
  for (int k = 0; k < kRawCh; ++k) f[k] = 0.0f;
  if (px < W && py < H) {
    const long long s = ((long long)py * W + px) * 3;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      f[k] = __ldg(rad + s + k);
      f[3 + k] = __ldg(alb + s + k);
      f[6 + k] = __ldg(nrm + s + k);
    }
    f[9] = __ldg(dep + s);
    f[10] = spp;
  }
  encode_px(f, x + 16 * ((long long)py * Wp + px));
}

// dskip[p, c] += (skip[p, c] > 0) * 0.25 * dpool[p / 2, c]: the pooled path's
// gradient reaching a ReLU output
__global__ void k_pool_grad_acc(const bf16* __restrict__ dpool, const bf16* __restrict__ skip,
                                bf16* __restrict__ dskip, int N, int H, int W, int C) {
  int c8 = C >> 3;
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long total = (long long)N * H * W * c8;
  if (i >= total) return;
  int c = (int)(i % c8) * 8;
  long long p = i / c8;
  int x = (int)(p % W);
  long long r = p / W;
  int y = (int)(r % H);
  int n = (int)(r / H);
  float d[8], s[8], g[8];
  ld8(dpool + (((size_t)n * (H >> 1) + (y >> 1)) * (W >> 1) + (x >> 1)) * C + c, d);
  ld8(skip + p * C + c, s);
  ld8(dskip + p * C + c, g);
#pragma unroll
  for (int k = 0; k < 8; ++k) g[k] += s[k] > 0.0f ? 0.25f * d[k] : 0.0f;
  st8(dskip + p * C + c, g);
}

// L1 on log(1 + target): pred [P][16] FP32 (channels 0..2), target [P][3];
// d_pred = sign(pred - log1p(target)) / (3P) as BF16 [P][16]; loss summed
// into *loss (FP64)
// The loss of the kernel-predicting output, per pixel p of N frames of H x W:
// o = sum_k w_k r(tap k), loss = sum_c (o_c - t_c)^2 / (o_c^2 + kRelEps),
// with the denominator held constant; the gradient of the mean over pixels
// and channels is taken through the filter and the softmax to the logits
// (dl_k = w_k (dw_k - sum_j w_j dw_j), dw_k = sum_c g_c r_c(tap k)), stored
// as BF16 [P][kPredCh] (zero beyond the taps).
// kTile (W a multiple of the 256-pixel block, so a block is one run of one
// image row): the block first stages the RGB of its kKpWidth clamped rows x
// (256 + kKpWidth - 1) clamped columns in shared memory, once, instead of
// every pixel reading its 25 taps twice through L1.
constexpr int kKpBlock = 256, kKpTileW = kKpBlock + kKpWidth - 1;

template <bool kTile>
__global__ void __launch_bounds__(kKpBlock) k_kp_loss(const float* __restrict__ pred, const float* __restrict__ raw,
                                                      const float* __restrict__ target, bf16* __restrict__ dpred,
                                                      int N, int H, int W, double* loss) {
  __shared__ float tile[kTile ? kKpWidth : 1][kTile ? kKpTileW : 1][3];
  const long long P = (long long)N * H * W;
  long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (kTile) {
    constexpr int r = kKpWidth / 2;
    const long long pb = blockIdx.x * (long long)blockDim.x;
    const int x0 = (int)(pb % W);
    const long long qb = pb / W;
    const int yb = (int)(qb % H);
    const long long fb = (qb / H) * (long long)H * W;
    for (int e = threadIdx.x; e < kKpWidth * kKpTileW; e += blockDim.x) {
      const int rr = e / kKpTileW, cc = e - rr * kKpTileW;
      const int ty = min(max(yb + rr - r, 0), H - 1), tx = min(max(x0 + cc - r, 0), W - 1);
      raw_rgb(raw, fb + (long long)ty * W + tx, tile[rr][cc]);
    }
    __syncthreads();
  }
  // tap k of this pixel: from the staged tile, or through kp_tap
  auto tap = [&](long long frame0, int x, int y, int k, float* c) {
    if (kTile) {
      const float* t = tile[k / kKpWidth][threadIdx.x + k % kKpWidth];
      c[0] = t[0];
      c[1] = t[1];
      c[2] = t[2];
    } else {
      raw_rgb(raw, kp_tap(frame0, x, y, k, W, H, W), c);
    }
  };
  float part = 0.0f;
  if (p < P) {
    const int x = (int)(p % W);
    const long long q = p / W;
    const int y = (int)(q % H);
    const long long frame0 = (q / H) * (long long)H * W;
    float w[kKpTaps];
    kp_weights(pred + (long long)kPredCh * p, w);
    float o[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < kKpTaps; ++k) {
      float c[3];
      tap(frame0, x, y, k, c);
      o[0] += w[k] * c[0];
      o[1] += w[k] * c[1];
      o[2] += w[k] * c[2];
    }
    const float inv = 1.0f / (3.0f * (float)P);
    float g[3];
    for (int i = 0; i < 3; ++i) {
      const float d = o[i] - sane(target[3 * p + i]);
      const float den = o[i] * o[i] + kRelEps;
      part += d * d / den;
      g[i] = 2.0f * d / den * inv;
    }
    float dw[kKpTaps], s = 0.0f;
#pragma unroll
    for (int k = 0; k < kKpTaps; ++k) {
      float c[3];
      tap(frame0, x, y, k, c);
      dw[k] = g[0] * c[0] + g[1] * c[1] + g[2] * c[2];
      s += w[k] * dw[k];
    }
    float dl[kPredCh];
#pragma unroll
    for (int k = 0; k < kPredCh; ++k) dl[k] = k < kKpTaps ? w[k] * (dw[k] - s) : 0.0f;
#pragma unroll
    for (int k = 0; k < kPredCh; k += 8) st8(dpred + (long long)kPredCh * p + k, dl + k);
  }
  for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, (double)part);
}

// Adam (Kingma & Ba) on the FP32 master parameters
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, long long n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float gi = g[i];
  float mi = b1 * m[i] + (1.0f - b1) * gi;
  float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// master [Cout][9][Cin] FP32 -> w [Cout][9][Cin] and wt [Cin][9][Cout] BF16
__device__ __forceinline__ void weight_bf16(const float* __restrict__ master, bf16* __restrict__ w,
                                            bf16* __restrict__ wt, int Cout, int Cin, long long i) {
  long long n = (long long)Cout * 9 * Cin;
  if (i >= n) return;
  int c = (int)(i % Cin);
  long long r = i / Cin;
  int t = (int)(r % 9);
  int o = (int)(r / 9);
  bf16 b = __float2bfloat16_rn(master[i]);
  w[i] = b;
  if (wt) wt[((size_t)c * 9 + t) * Cout + o] = b;
}

__global__ void k_weights_bf16(const float* __restrict__ master, bf16* __restrict__ w, bf16* __restrict__ wt,
                               int Cout, int Cin) {
  weight_bf16(master, w, wt, Cout, Cin, blockIdx.x * (long long)blockDim.x + threadIdx.x);
}

// Every layer's BF16 weights and transposes in one launch (blockIdx.y = layer)
__global__ void k_weights_bf16_all(WeightLayouts j) {
  const int l = blockIdx.y;
  weight_bf16(j.master[l], j.w[l], j.wt[l], j.Cout[l], j.Cin[l], blockIdx.x * (long long)blockDim.x + threadIdx.x);
}

// The denoised radiance: the predicted filter applied to the input radiance,
// for N frames of Hc x Wc pixels stored as Hs x Ws (the frame is the top-left
// corner; taps are clamped to it); out [N][Hc][Wc][3].
// kPx: floats per pixel of `raw` (a record, or the radiance pass itself, whose
// rows are Wr pixels while pred's are Ws).
template <int kPx>
__global__ void k_kp_apply(const float* __restrict__ pred, const float* __restrict__ raw, float* __restrict__ out,
                           int N, int Hc, int Wc, int Hs, int Ws, int Hr, int Wr) {
  const long long P = (long long)N * Hc * Wc;
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= P) return;
  const int x = (int)(i % Wc);
  const long long q = i / Wc;
  const int y = (int)(q % Hc);
  const long long n = q / Hc, frame0 = n * Hr * Wr;
  const long long p = n * Hs * Ws + (long long)y * Ws + x;
  float w[kKpTaps];
  kp_weights(pred + (long long)kPredCh * p, w);
  float o[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int k = 0; k < kKpTaps; ++k) {
    float c[3];
    raw_rgb<kPx>(raw, kp_tap(frame0, x, y, k, Wc, Hc, Wr), c);
    o[0] += w[k] * c[0];
    o[1] += w[k] * c[1];
    o[2] += w[k] * c[2];
  }
  out[3 * i] = o[0];
  out[3 * i + 1] = o[1];
  out[3 * i + 2] = o[2];
}

// ---- launchers ------------------------------------------------------------
cudaError_t encode_input(const float* raw, bf16* x, long long P, cudaStream_t st) {
  k_encode_input<<<blocks(P), 256, 0, st>>>(raw, x, P);
  return cudaGetLastError();
}
cudaError_t pool_grad_acc(const bf16* dpool, const bf16* skip, bf16* dskip, int N, int H, int W, int C,
                          cudaStream_t st) {
  long long n = (long long)N * H * W * (C / 8);
  k_pool_grad_acc<<<blocks(n), 256, 0, st>>>(dpool, skip, dskip, N, H, W, C);
  return cudaGetLastError();
}
cudaError_t kp_loss(const float* pred, const float* raw, const float* target, bf16* dpred, int N, int H,
                    int W, double* loss, cudaStream_t st) {
  if (W % kKpBlock == 0)
    k_kp_loss<true><<<blocks((long long)N * H * W), kKpBlock, 0, st>>>(pred, raw, target, dpred, N, H, W, loss);
  else
    k_kp_loss<false><<<blocks((long long)N * H * W), kKpBlock, 0, st>>>(pred, raw, target, dpred, N, H, W, loss);
  return cudaGetLastError();
}
cudaError_t adam(float* p, const float* g, float* m, float* v, long long n, float lr, int step,
                 cudaStream_t st) {
  const float b1 = 0.9f, b2 = 0.999f;
  float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  k_adam<<<blocks(n), 256, 0, st>>>(p, g, m, v, n, lr, b1, b2, 1e-8f, c1, c2);
  return cudaGetLastError();
}
cudaError_t weights_bf16(const float* master, bf16* w, bf16* wt, int Cout, int Cin, cudaStream_t st) {
  k_weights_bf16<<<blocks((long long)Cout * 9 * Cin), 256, 0, st>>>(master, w, wt, Cout, Cin);
  return cudaGetLastError();
}
cudaError_t weights_bf16_all(const WeightLayouts& j, cudaStream_t st) {
  if (j.n <= 0 || j.n > WeightLayouts::kMax) return cudaErrorInvalidValue;
  long long nmax = 1;
  for (int l = 0; l < j.n; ++l) nmax = std::max(nmax, (long long)j.Cout[l] * 9 * j.Cin[l]);
  k_weights_bf16_all<<<dim3(blocks(nmax), (unsigned)j.n), 256, 0, st>>>(j);
  return cudaGetLastError();
}
cudaError_t kp_apply(const float* pred, const float* raw, float* out, int N, int Hc, int Wc, int Hs, int Ws,
                     cudaStream_t st) {
  k_kp_apply<kRawCh><<<blocks((long long)N * Hc * Wc), 256, 0, st>>>(pred, raw, out, N, Hc, Wc, Hs, Ws, Hs, Ws);
  return cudaGetLastError();
}

cudaError_t kp_apply_passes(const float* pred, const float* rad, float* out, int W, int H, int Wp, cudaStream_t st) {
  k_kp_apply<3><<<blocks((long long)W * H), 256, 0, st>>>(pred, rad, out, 1, H, W, H, Wp, H, W);
  return cudaGetLastError();
}

cudaError_t encode_passes(const float* rad, const float* alb, const float* nrm, const float* dep, float spp, bf16* x,
                          int W, int H, int Wp, int Hp, cudaStream_t st) {
  // grid.y is at most 65,535 rows: taller frames in slices
  for (int y0 = 0; y0 < Hp; y0 += 65535) {
    const int rows = std::min(65535, Hp - y0);
    const long long o = 3LL * W * y0;
    k_encode_passes<<<dim3((Wp + 127) / 128, rows), 128, 0, st>>>(rad + o, alb + o, nrm + o, dep + o, spp,
                                                                 x + 16LL * Wp * y0, W, H - y0, Wp);
  }
  return cudaGetLastError();
}

}  // namespace nn
}  // namespace rtx
