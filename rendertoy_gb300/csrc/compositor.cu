// compositor.cu — RenderToy's Image filters on the GPU
// (include/RenderToy/compositor.h:107-178, src/compositor.cpp:42-77).
//
// Every output pixel sums its taps in the reference's order (row of the
// kernel, then column; products rounded before each addition: the file is
// built with --fmad=false), so results equal the reference bit for bit.
// Edge taps use the reference's reflect mapping (compositor.h:25-39), in
// which index == size maps to itself; a tap whose linear index falls outside
// the image reads zero (the reference reads past its buffer there).
//
// Separable passes (GaussianBlur = 1 x size then size x 1) stage a row
// segment / column strip with its halo in shared memory (cp.async, one wait
// per tile), so each input pixel is read from HBM once per pass; bloom's
// extraction is fused into the first pass and its final addition into the
// second.  The separable passes and the 3 x 3 / 5 x 5 convolutions are
// register-blocked (a thread computes 8 or 4 outputs along one axis and
// reuses every staged pixel for all of them) and run two outputs per packed
// FP32 instruction; each output's taps are still summed one by one in the
// reference's order with the same roundings.  They are FP32-issue bound: a
// size-49 pass is 49 x 3 multiplies and adds per pixel for 24 bytes of HBM.
#include <algorithm>

#include "device_math.cuh"
#include "rtx_internal.h"

namespace rtx {

enum ConvFlags { kAbs = 1, kLength = 2, kNormalize = 4 };

RTX_DEV long long reflect_index(long long row, long long col, long long W, long long H) {
  if (row < 0) row = -row;
  if (col < 0) col = -col;
  if (col >= W) col = 2 * W - col;
  if (row >= H) row = 2 * H - row;
  long long idx = row * W + col;
  return (idx < 0 || idx >= W * H) ? -1 : idx;
}

RTX_DEV F3 load_px(const float* __restrict__ in, long long idx) {
  if (idx < 0) return f3s(0.0f);
  return f3(__ldg(in + 3 * idx), __ldg(in + 3 * idx + 1), __ldg(in + 3 * idx + 2));
}

// Stage pixel idx (or zeros for idx < 0) into shared memory at s with three
// 4-byte cp.async copies: a tile's fill issues all its loads before waiting
// once (cp_wait_all), instead of one DRAM round trip per loop iteration.
RTX_DEV void stage_px(float* s, const float* __restrict__ in, long long idx) {
  if (idx < 0) {
    s[0] = 0.0f;
    s[1] = 0.0f;
    s[2] = 0.0f;
    return;
  }
  const unsigned d = (unsigned)__cvta_generic_to_shared(s);
  const float* g = in + 3 * idx;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(g) : "memory");
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4), "l"(g + 1) : "memory");
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 8), "l"(g + 2) : "memory");
}
RTX_DEV void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Image::Extract(Luma > threshold) (compositor.cpp:51-59, 69-71)
RTX_DEV F3 extract(F3 p, float thr) { return luma(p) > thr ? p : f3s(0.0f); }

// General kr x kc convolution, one pixel per thread (Image::Convolute)
__global__ void k_convolve(const float* __restrict__ in, float* __restrict__ out, int W, int H,
                           const float* __restrict__ k, int kr, int kc, int flags) {
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  if (x >= W) return;
  long long r2 = kr >> 1, c2 = kc >> 1;
  F3 acc = f3s(0.0f);
  for (int ii = 0; ii < kr; ++ii)
    for (int jj = 0; jj < kc; ++jj) {
      long long idx = reflect_index(y - r2 + ii, x - c2 + jj, W, H);
      acc = acc + load_px(in, idx) * __ldg(k + ii * kc + jj);
    }
  if (flags & kAbs) acc = f3(fabsf(acc.x), fabsf(acc.y), fabsf(acc.z));
  if (flags & kLength) acc = f3s(length(acc));
  if (flags & kNormalize) acc = normalized(acc);
  float* o = out + 3 * ((size_t)y * W + x);
  o[0] = acc.x;
  o[1] = acc.y;
  o[2] = acc.z;
}

// The same convolution from a shared-memory tile: a block fills its 32 x 8
// pixels plus the kernel's halo once (every element through reflect_index,
// so RenderToy's reflection, including its row wrap, is kept), then each
// thread sums its taps in the same order as k_convolve.
constexpr int kConvTX = 32, kConvTY = 8;

__global__ void __launch_bounds__(kConvTX * kConvTY) k_convolve_tiled(const float* __restrict__ in,
                                                                     float* __restrict__ out, int W, int H,
                                                                     const float* __restrict__ k, int kr,
                                                                     int kc, int flags) {
  extern __shared__ float sm[];
  float* wsm = sm;            // kr * kc weights
  float* tile = sm + kr * kc; // (kConvTY + kr - 1) x (kConvTX + kc - 1) pixels
  const int tid = threadIdx.x;
  const int x0 = blockIdx.x * kConvTX, y0 = blockIdx.y * kConvTY;
  const int r2 = kr >> 1, c2 = kc >> 1, tw = kConvTX + kc - 1, th = kConvTY + kr - 1;
  for (int i = tid; i < kr * kc; i += blockDim.x) wsm[i] = k[i];
  for (int i = tid; i < tw * th; i += blockDim.x) {
    const int ty = i / tw, tx = i - ty * tw;
    F3 p = load_px(in, reflect_index((long long)y0 - r2 + ty, (long long)x0 - c2 + tx, W, H));
    tile[3 * i] = p.x;
    tile[3 * i + 1] = p.y;
    tile[3 * i + 2] = p.z;
  }
  __syncthreads();
  const int lx = tid % kConvTX, ly = tid / kConvTX;
  const int x = x0 + lx, y = y0 + ly;
  if (x >= W || y >= H) return;
  F3 acc = f3s(0.0f);
  for (int ii = 0; ii < kr; ++ii)
    for (int jj = 0; jj < kc; ++jj) {
      const float* q = tile + 3 * ((ly + ii) * tw + lx + jj);
      acc = acc + f3(q[0], q[1], q[2]) * wsm[ii * kc + jj];
    }
  if (flags & kAbs) acc = f3(fabsf(acc.x), fabsf(acc.y), fabsf(acc.z));
  if (flags & kLength) acc = f3s(length(acc));
  if (flags & kNormalize) acc = normalized(acc);
  float* o = out + 3 * ((size_t)y * W + x);
  o[0] = acc.x;
  o[1] = acc.y;
  o[2] = acc.z;
}

// acc + p * w with the product rounded before the addition, exactly as the
// scalar multiply and add.  ptxas contracts a packed multiply followed by a
// packed add into one fused operation even under --fmad=false, so the
// product is formed as fma(p, w, nz) with nz = -0.0 passed in at run time
// (unknown to the compiler): that rounds p * w once, as a multiply does
// (x + -0 == x, also for x = +0 and -0), and leaves nothing to contract.
RTX_DEV f2_t f2_mul_add(f2_t acc, f2_t p, f2_t w, f2_t nz) { return f2_add(acc, f2_fma(p, w, nz)); }
// One tap into an accumulator pair: RenderToy's rounding (kFma = false) or one
// fused multiply-add per tap (kFma = true: RTX_OPT_COMPOSITOR_FMA), which
// halves the FP32 work of the register-blocked filters.
template <bool kFma>
RTX_DEV f2_t f2_tap(f2_t acc, f2_t p, f2_t w, f2_t nz) {
  return kFma ? f2_fma(p, w, acc) : f2_mul_add(acc, p, w, nz);
}
template <bool kFma>
RTX_DEV float f_tap(float acc, float p, float w) {
  return kFma ? __fmaf_rn(p, w, acc) : acc + p * w;
}
RTX_DEV float f3c(F3 p, int c) { return c == 0 ? p.x : (c == 1 ? p.y : p.z); }

// Small 2-D kernels (3 x 3, 5 x 5), register-blocked: a thread computes
// kConvR vertically adjacent outputs of one column, with the weights in
// registers.  It walks the staged rows of its window in order and output r
// takes staged row yy as kernel row yy - r, so each output still sums its
// taps row by row, column by column, as the reference does.
constexpr int kConvR = 4, kConvRegThreads = 256, kConvRegW = 32,
              kConvRegH = (kConvRegThreads / kConvRegW) * kConvR;

template <int KR, int KC, bool kFma>
__global__ void __launch_bounds__(kConvRegThreads, 4) k_convolve_reg(const float* __restrict__ in,
                                                                  float* __restrict__ out, int W, int H,
                                                                  const float* __restrict__ k, int flags,
                                                                  float negzero) {
  constexpr int tw = kConvRegW + KC - 1, th = kConvRegH + KR - 1;
  __shared__ float tile[3 * tw * th];
  const int tid = threadIdx.x;
  const int x0 = blockIdx.x * kConvRegW, y0 = blockIdx.y * kConvRegH;
  for (int i = tid; i < tw * th; i += kConvRegThreads) {
    const int ty = i / tw, tx = i - ty * tw;
    stage_px(tile + 3 * i, in, reflect_index((long long)y0 - KR / 2 + ty, (long long)x0 - KC / 2 + tx, W, H));
  }
  float wk[KR * KC];
#pragma unroll
  for (int i = 0; i < KR * KC; ++i) wk[i] = __ldg(k + i);
  cp_wait_all();
  __syncthreads();
  const int lx = tid % kConvRegW, g = tid / kConvRegW;
  const int x = x0 + lx, yb = y0 + kConvR * g;
  if (x >= W || yb >= H) return;
  const f2_t nz = f2_pack(negzero, negzero);
  f2_t acc[3][kConvR / 2];  // [channel][output pair (rows 2q, 2q + 1)]
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int q = 0; q < kConvR / 2; ++q) acc[c][q] = f2_pack(0.0f, 0.0f);
#pragma unroll
  for (int yy = 0; yy < kConvR + KR - 1; ++yy)
#pragma unroll
    for (int jj = 0; jj < KC; ++jj) {
      const float* t = tile + 3 * ((kConvR * g + yy) * tw + lx + jj);
      const F3 p = f3(t[0], t[1], t[2]);
      const f2_t pp[3] = {f2_pack(p.x, p.x), f2_pack(p.y, p.y), f2_pack(p.z, p.z)};
#pragma unroll
      for (int q = 0; q < kConvR / 2; ++q) {
        const int i0 = yy - 2 * q, i1 = i0 - 1;  // kernel rows of outputs 2q, 2q + 1
        const bool v0 = i0 >= 0 && i0 < KR, v1 = i1 >= 0 && i1 < KR;
        if (v0 && v1) {
          const f2_t ww = f2_pack(wk[i0 * KC + jj], wk[i1 * KC + jj]);
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[c][q] = f2_tap<kFma>(acc[c][q], pp[c], ww, nz);
        } else if (v0 || v1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            float a, b;
            f2_unpack(acc[c][q], a, b);
            if (v0) a = f_tap<kFma>(a, f3c(p, c), wk[i0 * KC + jj]);
            if (v1) b = f_tap<kFma>(b, f3c(p, c), wk[i1 * KC + jj]);
            acc[c][q] = f2_pack(a, b);
          }
        }
      }
    }
#pragma unroll
  for (int r = 0; r < kConvR; ++r) {
    const int y = yb + r;
    if (y >= H) break;
    float lo[3], hi[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) f2_unpack(acc[c][r >> 1], lo[c], hi[c]);
    F3 v = (r & 1) ? f3(hi[0], hi[1], hi[2]) : f3(lo[0], lo[1], lo[2]);
    if (flags & kAbs) v = f3(fabsf(v.x), fabsf(v.y), fabsf(v.z));
    if (flags & kLength) v = f3s(length(v));
    if (flags & kNormalize) v = normalized(v);
    float* o = out + 3 * ((size_t)y * W + x);
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
  }
}

// Separable passes, register-blocked: a thread computes kSepR consecutive
// outputs along the filter direction.  It walks its window of
// kSepR + size - 1 staged pixels once and adds each pixel into every output
// whose taps cover it (output o takes window pixel j as tap j - o).  j only
// grows, so each output still sums its taps in the order 0 .. size - 1 with
// the same roundings as one output per thread (products rounded, then
// added), while shared-memory loads drop kSepR-fold and every weight is
// loaded once per chunk of kSepR pixels.  Outputs 2q and 2q + 1 of a channel
// share one packed accumulator, so one f32x2 multiply and one f32x2 add
// serve two taps.
constexpr int kSepR = 8, kSepQ = kSepR / 2;

struct SepAcc {
  f2_t v[3][kSepQ];  // [channel][output pair]
  RTX_DEV F3 out(int o) const {
    float a[3], b[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) f2_unpack(v[c][o >> 1], a[c], b[c]);
    return (o & 1) ? f3(b[0], b[1], b[2]) : f3(a[0], a[1], a[2]);
  }
};

// A window starts kLead pixels before its first tap, so that its first pixel is
// kSepR m / 2 (a multiple of four) pixels before the first output and the
// windows' chunks of kSepR pixels number m + 1.  Window<k>: sizes with
// kLead = k % 4; k >= 4: even ones, whose last tap is missing on the right.
template <int k>
struct Window {
  static constexpr int kLead = k & 3, kTail = kLead + (k >> 2);
};
static int window_kind(int size) { return (4 - (size >> 1) % 4) % 4 + (size % 2 == 0 ? 4 : 0); }
RTX_DEV int window_chunks(int size, int lead) { return ((size | 1) + 2 * lead) >> 3; }  // m

// Add window pixels j0 .. j0 + kSepR - 1 into the accumulators; output o takes
// pixel j0 + s as tap j0 + s - o - kLead.  Which (pixel, output) pairs of a
// chunk are taps is known at compile time: those with kLo <= s - o <= kHi.
// (Run-time tests of the edge chunks took 58 % of the horizontal pass's ALU.)
template <int kLo_, int kHi_, int kLead_>
struct Taps {
  static constexpr int kLo = kLo_, kHi = kHi_, kLead = kLead_;
  static constexpr bool kAll = kLo <= 1 - kSepR && kHi >= kSepR - 1;
  static RTX_DEV constexpr bool in(int s, int o) { return s - o >= kLo && s - o <= kHi; }
};

template <class T>
RTX_DEV void tap_weights(float (&wv)[2 * kSepR - 1], const float* __restrict__ wsm, int size, int j0) {
#pragma unroll
  for (int k = 0; k < 2 * kSepR - 1; ++k) {  // wv[k]: the weight of s - o = k - (kSepR - 1)
    const int ii = j0 - (kSepR - 1) + k - T::kLead;
    wv[k] = wsm[T::kAll ? ii : min(max(ii, 0), size - 1)];
  }
}

template <class T, bool kFma, class Px>
RTX_DEV void sep_chunk(SepAcc& A, const float* __restrict__ wsm, int size, int j0, f2_t nz, Px px) {
  float wv[2 * kSepR - 1];
  tap_weights<T>(wv, wsm, size, j0);
  f2_t wp[2 * kSepR - 1];  // wp[k] = (wv[k], wv[k - 1]): the taps of an output pair
#pragma unroll
  for (int k = 1; k < 2 * kSepR - 1; ++k) wp[k] = f2_pack(wv[k], wv[k - 1]);
#pragma unroll
  for (int s = 0; s < kSepR; ++s) {
    const F3 p = px(j0 + s);
    const f2_t pp[3] = {f2_pack(p.x, p.x), f2_pack(p.y, p.y), f2_pack(p.z, p.z)};
#pragma unroll
    for (int q = 0; q < kSepQ; ++q) {
      const int o0 = 2 * q, o1 = 2 * q + 1, k0 = s - o0 + kSepR - 1;
      const bool v0 = T::in(s, o0);
      const bool v1 = T::in(s, o1);
      if (v0 && v1) {
#pragma unroll
        for (int c = 0; c < 3; ++c) A.v[c][q] = f2_tap<kFma>(A.v[c][q], pp[c], wp[k0], nz);
      } else if (v0 || v1) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float a, b;
          f2_unpack(A.v[c][q], a, b);
          const float pc = f3c(p, c);
          if (v0) a = f_tap<kFma>(a, pc, wv[k0]);
          if (v1) b = f_tap<kFma>(b, pc, wv[k0 - 1]);
          A.v[c][q] = f2_pack(a, b);
        }
      }
    }
  }
}

// The taps of chunk c of Window<k>'s chunks 0 .. m.
template <int k, class Fn>
RTX_DEV void chunk_taps(int c, int m, Fn f) {
  constexpr int kN = kSepR, kLead = Window<k>::kLead, kTail = Window<k>::kTail;
  if (c == 0) {
    if (k == 0 && m == 0)
      f(Taps<0, 0, 0>());
    else if (m == 1)
      f(Taps<kLead, kN - kTail, kLead>());
    else
      f(Taps<kLead, kN - 1, kLead>());
  } else if (c == m) {
    if (m == 1)
      f(Taps<kLead - kN, -kTail, kLead>());
    else
      f(Taps<1 - kN, -kTail, kLead>());
  } else if ((kLead < 2 || c > 1) && (kTail < 2 || c < m - 1)) {
    f(Taps<1 - kN, kN - 1, kLead>());
  } else if (c > 1) {
    f(Taps<1 - kN, kN - kTail, kLead>());
  } else if (c < m - 1) {
    f(Taps<kLead - kN, kN - 1, kLead>());
  } else {
    f(Taps<kLead - kN, kN - kTail, kLead>());
  }
}

template <int k, bool kFma, class Px>
RTX_DEV void sep_window(SepAcc& A, const float* __restrict__ wsm, int size, float negzero, Px px) {
  const f2_t nz = f2_pack(negzero, negzero);
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int q = 0; q < kSepQ; ++q) A.v[c][q] = f2_pack(0.0f, 0.0f);
  const int m = window_chunks(size, Window<k>::kLead);
  for (int c = 0; c <= m; ++c)
    chunk_taps<k>(c, m, [&](auto taps) { sep_chunk<decltype(taps), kFma>(A, wsm, size, kSepR * c, nz, px); });
}

// Horizontal pass (1 x size kernel): a block computes kRowTile pixels of one
// row.  The row segment and its halo sit in shared memory as RGB triples with
// one spare triple after every kSepR pixels, so the kSepR-pixel strides of a
// warp's lanes (27 words apart) fall in distinct banks.  Only pixels that are
// taps are staged (size - 1 beyond the outputs; the window's kLead before them
// have no slot), so that the segment fits up to 12,493 taps.
constexpr int kRowThreads = 128, kRowTile = kRowThreads * kSepR;
RTX_DEV int row_slot(int i) { return 3 * (i + i / kSepR); }

template <int k, bool kFma>
__global__ void __launch_bounds__(kRowThreads, 7) k_gauss_x(const float* __restrict__ in,
                                                         float* __restrict__ out, int W, int H,
                                                         const float* __restrict__ w, int size,
                                                         int extract_mode, float thr, float negzero) {
  extern __shared__ float sm[];
  float* wsm = sm;                       // size weights
  float* tile = sm + ((size + 3) & ~3);
  constexpr int kLead = Window<k>::kLead;
  auto slot = [&](int i) { return tile + row_slot(i) - row_slot(kLead); };  // of window pixel i >= kLead
  const int y = blockIdx.y, x0 = blockIdx.x * kRowTile, r = size >> 1, tid = threadIdx.x;
  const int n_out = min(kRowTile, W - x0);
  const int span = n_out + size - 1, cap = kRowTile + size - 1;
  for (int j = tid; j < size; j += kRowThreads) wsm[j] = w[j];
  for (int j = tid; j < cap; j += kRowThreads)
    stage_px(slot(kLead + j), in, j < span ? reflect_index(y, (long long)x0 - r + j, W, H) : -1);
  cp_wait_all();
  if (extract_mode) {  // bloom: Extract applied to the staged pixels
    for (int j = tid; j < span; j += kRowThreads) {
      float* s = slot(kLead + j);
      const F3 p = extract(f3(s[0], s[1], s[2]), thr);
      s[0] = p.x;
      s[1] = p.y;
      s[2] = p.z;
    }
  }
  __syncthreads();
  SepAcc acc;
  const int b = kSepR * tid;
  if (b < n_out) {
    sep_window<k, kFma>(acc, wsm, size, negzero, [&](int j) {
      const float* s = slot(b + j);
      return f3(s[0], s[1], s[2]);
    });
  }
  __syncthreads();  // the tile now holds the outputs
  if (b < n_out) {
#pragma unroll
    for (int o = 0; o < kSepR; ++o) {
      float* s = tile + row_slot(b + o);
      const F3 v = acc.out(o);
      s[0] = v.x;
      s[1] = v.y;
      s[2] = v.z;
    }
  }
  __syncthreads();
  float* orow = out + 3 * ((size_t)y * W + x0);
  for (int f = tid; f < 3 * n_out; f += kRowThreads) {
    const int q = f / 3;
    orow[f] = tile[row_slot(q) + (f - 3 * q)];
  }
}

// Vertical pass (size x 1 kernel): a block computes kColW columns x kColH
// rows; lanes take neighbouring columns, each thread kSepR consecutive rows,
// from a shared-memory strip of kColH + size - 1 rows (those that are taps; the
// window's kLead rows before them are not staged): up to 568 taps.
// Registers for five blocks per SM: at seven (72) the compile-time windows
// spilled or were scheduled with loads late, which showed where strips leave few
// blocks on an SM (1,024^2: 520 taps 375 -> 342 us, 568 taps 408 -> 371; run-time
// windows took 362, 390) and at small sizes too (513 x 511: 49 taps 26.7 -> 25.1).
constexpr int kColW = 32, kColThreads = 128, kColH = (kColThreads / kColW) * kSepR;

template <int k, bool kFma>
__global__ void __launch_bounds__(kColThreads, 5) k_gauss_y(const float* __restrict__ in,
                                                         const float* __restrict__ orig,
                                                         float* __restrict__ out, int W, int H,
                                                         const float* __restrict__ w, int size,
                                                         float negzero) {
  extern __shared__ float sm[];
  float* wsm = sm;
  float* strip = sm + ((size + 3) & ~3);  // rows x kColW x 3
  const int x0 = blockIdx.x * kColW, y0 = blockIdx.y * kColH, r = size >> 1, tid = threadIdx.x;
  for (int j = tid; j < size; j += kColThreads) wsm[j] = w[j];
  const int rows = kColH + size - 1;
  for (int e = tid; e < rows * kColW; e += kColThreads) {
    const int rr = e / kColW, cc = e - rr * kColW;
    const int x = x0 + cc;
    stage_px(strip + 3 * e, in, x < W ? reflect_index((long long)y0 - r + rr, x, W, H) : -1);
  }
  cp_wait_all();
  __syncthreads();
  const int cc = tid % kColW, g = tid / kColW;
  const int x = x0 + cc, yb = y0 + kSepR * g;
  if (x >= W || yb >= H) return;
  SepAcc acc;
  sep_window<k, kFma>(acc, wsm, size, negzero, [&](int j) {
    const float* s = strip + 3 * ((kSepR * g + j - Window<k>::kLead) * kColW + cc);
    return f3(s[0], s[1], s[2]);
  });
#pragma unroll
  for (int o = 0; o < kSepR; ++o) {
    const int y = yb + o;
    if (y < H) {
      const size_t p = (size_t)y * W + x;
      F3 v = acc.out(o);
      if (orig) v = f3(__ldg(orig + 3 * p), __ldg(orig + 3 * p + 1), __ldg(orig + 3 * p + 2)) + v;
      out[3 * p] = v.x;
      out[3 * p + 1] = v.y;
      out[3 * p + 2] = v.z;
    }
  }
}

// ---------------------------------------------------------------------------
// The separable passes on 16-byte accesses: images whose rows are a multiple
// of four pixels (48 bytes).  Same taps in the same order with the same
// roundings; what differs is how pixels reach the registers.  The passes are FP32-issue bound (7.7 us each for 49
// taps at 1,024^2); the 4-byte staging copies with their 64-bit reflection
// arithmetic, three scalar shared loads and six register moves per pixel, and
// loads that all finished before any arithmetic began cost as much again.
// Both passes together, 49 taps at 1,024^2: 31.8 -> 22.4 us per call; 1920 x 1080
// bloom 65 -> 45.5 us.
// ---------------------------------------------------------------------------
RTX_DEV void cp16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
RTX_DEV void st_row(float* p, const float* v, bool wide) {  // 24 floats
  if (wide) {
#pragma unroll
    for (int k = 0; k < 24; k += 8)
      asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p + k), "f"(v[k]), "f"(v[k + 1]),
                   "f"(v[k + 2]), "f"(v[k + 3]), "f"(v[k + 4]), "f"(v[k + 5]), "f"(v[k + 6]), "f"(v[k + 7])
                   : "memory");
  } else {
#pragma unroll
    for (int k = 0; k < 24; k += 4) *reinterpret_cast<float4*>(p + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
  }
}

// Horizontal: staged pixels sit in groups of eight (24 floats) 28 floats apart,
// so that a window chunk is six 16-byte loads and eight neighbouring threads'
// loads fall in distinct banks.  Eight outputs are 96 contiguous bytes.  The
// window starts at a pixel that is a multiple of four, kLead pixels before its
// first tap.
constexpr int kRowGroup = 28;

template <int k, bool kFma>
__global__ void __launch_bounds__(kRowThreads, 7) k_gauss_x16(const float* __restrict__ in, float* __restrict__ out,
                                                             int W, int H, const float* __restrict__ w, int size,
                                                             int extract_mode, float thr, float negzero, int wide) {
  extern __shared__ __align__(16) float sm[];
  float* wsm = sm;
  float* tile = sm + ((size + 3) & ~3);
  const int y = blockIdx.y, x0 = blockIdx.x * kRowTile, tid = threadIdx.x;
  const int r = (size >> 1) + Window<k>::kLead;
  const int m = window_chunks(size, Window<k>::kLead), n_out = min(kRowTile, W - x0), groups = (n_out + 7) / 8 + m;
  for (int j = tid; j < size; j += kRowThreads) wsm[j] = w[j];
  // chunk c: floats 4 c .. 4 c + 3 from pixel x0 - r on; the row's ends fall on
  // chunk boundaries
  const float* row = in + 3 * (size_t)W * y;
  const int f0 = 3 * (x0 - r), f1 = 3 * W;
  const unsigned td = (unsigned)__cvta_generic_to_shared(tile);
  for (int c = tid; c < 6 * groups; c += kRowThreads) {
    const int f = f0 + 4 * c, d = (c / 6) * kRowGroup + (c % 6) * 4;
    if (f >= 0 && f < f1) {
      cp16(td + 4 * d, row + f);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int g = f + e + 3 * (size + 3), x = g / 3 - (size + 3);  // floor for negative f
        const long long idx = reflect_index(y, x, W, H);
        tile[d + e] = idx < 0 ? 0.0f : __ldg(in + 3 * idx + (g - 3 * (g / 3)));
      }
    }
  }
  cp_wait_all();
  __syncthreads();
  if (extract_mode) {  // bloom: Extract applied to the staged pixels
    for (int j = tid; j < 8 * groups; j += kRowThreads) {
      float* s = tile + (j >> 3) * kRowGroup + 3 * (j & 7);
      const F3 p = extract(f3(s[0], s[1], s[2]), thr);
      s[0] = p.x;
      s[1] = p.y;
      s[2] = p.z;
    }
    __syncthreads();
  }
  const int b = kSepR * tid;
  if (b >= n_out) return;
  const f2_t nz = f2_pack(negzero, negzero);
  SepAcc A;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int q = 0; q < kSepQ; ++q) A.v[c][q] = f2_pack(0.0f, 0.0f);
  for (int c = 0; c <= m; ++c) {
    const float4* s = reinterpret_cast<const float4*>(tile + (tid + c) * kRowGroup);
    float px[24];
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      const float4 v = s[e];
      px[4 * e] = v.x;
      px[4 * e + 1] = v.y;
      px[4 * e + 2] = v.z;
      px[4 * e + 3] = v.w;
    }
    const int j0 = kSepR * c;
    chunk_taps<k>(c, m, [&](auto taps) {
      sep_chunk<decltype(taps), kFma>(A, wsm, size, j0, nz, [&](int j) {
        return f3(px[3 * (j - j0)], px[3 * (j - j0) + 1], px[3 * (j - j0) + 2]);
      });
    });
  }
  float* o = out + 3 * ((size_t)y * W + x0 + b);
  float v[24];
#pragma unroll
  for (int e = 0; e < kSepR; ++e) {
    const F3 p = A.out(e);
    v[3 * e] = p.x;
    v[3 * e + 1] = p.y;
    v[3 * e + 2] = p.z;
  }
  if (b + kSepR <= n_out) {
    st_row(o, v, wide != 0);
  } else {  // n_out is a multiple of four pixels
#pragma unroll
    for (int e = 0; e < 12; e += 4) *reinterpret_cast<float4*>(o + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
  }
}

// Vertical: the image as rows of 3 W floats.  A thread computes kSepR rows of
// four neighbouring floats; the two floats of a packed operand share a weight,
// so a staged row is one 16-byte load and no moves.  A warp's rows arrive in
// chunks of kSepR (one cp.async group each) and its arithmetic starts with the
// first ones.
constexpr int kColQ = 32, kCol16Threads = 128, kCol16Groups = kCol16Threads / kColQ, kCol16H = kCol16Groups * kSepR;

template <class T, bool kFma>
RTX_DEV void col_chunk(f2_t (&acc)[2][kSepR], const float* __restrict__ wsm, int size, int j0, f2_t nz,
                       const float4* s) {
  float wv[2 * kSepR - 1];
  tap_weights<T>(wv, wsm, size, j0);
#pragma unroll
  for (int k = 0; k < kSepR; ++k) {
    const float4 v = s[k * kColQ];
    const f2_t a = f2_pack(v.x, v.y), b = f2_pack(v.z, v.w);
#pragma unroll
    for (int o = 0; o < kSepR; ++o) {
      if (T::in(k, o)) {
        const float ww = wv[k - o + kSepR - 1];
        const f2_t w2 = f2_pack(ww, ww);
        acc[0][o] = f2_tap<kFma>(acc[0][o], a, w2, nz);
        acc[1][o] = f2_tap<kFma>(acc[1][o], b, w2, nz);
      }
    }
  }
}

// The image bloom adds back is fetched into staged rows no warp reads any
// more, two chunks before it is needed.
template <int k, bool kFma>
__global__ void __launch_bounds__(kCol16Threads, 5) k_gauss_y16(const float* __restrict__ in,
                                                               const float* __restrict__ orig, float* __restrict__ out,
                                                               int W, int H, const float* __restrict__ w, int size,
                                                               float negzero) {
  extern __shared__ __align__(16) float sm[];
  float4* strip = reinterpret_cast<float4*>(sm);  // chunks * kSepR rows x kColQ
  const int nc = window_chunks(size, Window<k>::kLead) + 1;
  const int chunks = nc + kCol16Groups - 1;
  float* wsm = sm + 4 * (size_t)chunks * kSepR * kColQ;
  const int tid = threadIdx.x, q = tid % kColQ, g = tid / kColQ;
  const int nq = 3 * W / 4, q0 = blockIdx.x * kColQ, y0 = blockIdx.y * kCol16H, r = (size >> 1) + Window<k>::kLead;
  for (int j = tid; j < size; j += kCol16Threads) wsm[j] = w[j];
  const bool live = q0 + q < nq;
  const unsigned sd = (unsigned)__cvta_generic_to_shared(strip);
  const float4* col = reinterpret_cast<const float4*>(in) + q0 + q;
  auto stage = [&](int c) {  // rows 8 c .. 8 c + 7; warp g takes two of them
    if (c < chunks)
#pragma unroll
      for (int e = g; e < kSepR; e += kCol16Groups) {
        int yy = abs(y0 - r + kSepR * c + e);
        if (yy >= H) yy = 2 * H - yy;
        if (live && yy >= 0 && yy < H)
          cp16(sd + 16 * ((kSepR * c + e) * kColQ + q), col + (size_t)yy * nq);
        else
          strip[(kSepR * c + e) * kColQ + q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // chunk c of the window needs staged chunks 0 .. c + kCol16Groups - 1; kAhead
  // more are in flight
  constexpr int kAhead = 3;
  for (int c = 0; c < kCol16Groups + kAhead - 1; ++c) stage(c);
  const f2_t nz = f2_pack(negzero, negzero);
  f2_t acc[2][kSepR];
#pragma unroll
  for (int o = 0; o < kSepR; ++o) acc[0][o] = acc[1][o] = f2_pack(0.0f, 0.0f);
  // after chunk c's barrier no warp reads rows below kSepR * c
  const int c_orig = orig && nc - 1 >= kCol16Groups ? max(kCol16Groups, nc - 2) : -1;
  for (int c = 0; c < nc; ++c) {
    stage(c + kCol16Groups + kAhead - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kAhead) : "memory");
    __syncthreads();
    if (c == c_orig && live) {
#pragma unroll
      for (int o = 0; o < kSepR; ++o) {
        const int y = y0 + kSepR * g + o;
        if (y < H)
          cp16(sd + 16 * ((kSepR * g + o) * kColQ + q), reinterpret_cast<const float4*>(orig) + (size_t)y * nq + q0 + q);
      }
    }
    const int j0 = c * kSepR;
    const float4* s = strip + (size_t)(kSepR * (g + c)) * kColQ + q;
    chunk_taps<k>(c, nc - 1, [&](auto taps) { col_chunk<decltype(taps), kFma>(acc, wsm, size, j0, nz, s); });
  }
  cp_wait_all();
  if (!live) return;
#pragma unroll
  for (int o = 0; o < kSepR; ++o) {
    const int y = y0 + kSepR * g + o;
    if (y >= H) break;
    const size_t p = (size_t)y * nq + q0 + q;
    float4 v;
    f2_unpack(acc[0][o], v.x, v.y);
    f2_unpack(acc[1][o], v.z, v.w);
    if (orig) {
      const float4 i = c_orig >= 0 ? strip[(kSepR * g + o) * kColQ + q] : __ldg(reinterpret_cast<const float4*>(orig) + p);
      v = make_float4(i.x + v.x, i.y + v.y, i.z + v.z, i.w + v.w);
    }
    reinterpret_cast<float4*>(out)[p] = v;
  }
}

// EdgeDetection<All> (compositor.h:153-178): Sobel-X and Sobel-Y sums of the
// 3 x 3 neighbourhood, each in the reference's tap order, then |gy + gx|.
__global__ void k_edge(const float* __restrict__ in, float* __restrict__ out, int W, int H) {
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  if (x >= W) return;
  const float sx[9] = {-1.f, 0.f, 1.f, -2.f, 0.f, 2.f, -1.f, 0.f, 1.f};
  const float sy[9] = {1.f, 2.f, 1.f, 0.f, 0.f, 0.f, -1.f, -2.f, -1.f};
  F3 gx = f3s(0.0f), gy = f3s(0.0f);
#pragma unroll
  for (int ii = 0; ii < 3; ++ii)
#pragma unroll
    for (int jj = 0; jj < 3; ++jj) {
      F3 p = load_px(in, reflect_index(y - 1 + ii, x - 1 + jj, W, H));
      gx = gx + p * sx[ii * 3 + jj];
      gy = gy + p * sy[ii * 3 + jj];
    }
  float l = length(gy + gx);
  float* o = out + 3 * ((size_t)y * W + x);
  o[0] = l;
  o[1] = l;
  o[2] = l;
}

__global__ void k_extract(const float* __restrict__ in, float* __restrict__ out, size_t n, float thr) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  F3 p = extract(f3(in[3 * i], in[3 * i + 1], in[3 * i + 2]), thr);
  out[3 * i] = p.x;
  out[3 * i + 1] = p.y;
  out[3 * i + 2] = p.z;
}

// Image::operator+ (compositor.cpp:102-115): out = a + b
__global__ void k_add(const float* __restrict__ a, const float* __restrict__ b,
                      float* __restrict__ out, size_t n) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = a[i] + b[i];
}

cudaError_t launch_convolve(const float* in, float* out, int W, int H, const float* d_k, int kr,
                            int kc, int flags, bool fma, cudaStream_t st, int* launches) {
  const size_t smem = sizeof(float) * ((size_t)kr * kc + 3 * (size_t)(kConvTY + kr - 1) * (kConvTX + kc - 1));
  const dim3 rgrid((W + kConvRegW - 1) / kConvRegW, (H + kConvRegH - 1) / kConvRegH);
  if (kr == 5 && kc == 5) {
    if (fma)
      k_convolve_reg<5, 5, true><<<rgrid, kConvRegThreads, 0, st>>>(in, out, W, H, d_k, flags, -0.0f);
    else
      k_convolve_reg<5, 5, false><<<rgrid, kConvRegThreads, 0, st>>>(in, out, W, H, d_k, flags, -0.0f);
  } else if (kr == 3 && kc == 3) {
    if (fma)
      k_convolve_reg<3, 3, true><<<rgrid, kConvRegThreads, 0, st>>>(in, out, W, H, d_k, flags, -0.0f);
    else
      k_convolve_reg<3, 3, false><<<rgrid, kConvRegThreads, 0, st>>>(in, out, W, H, d_k, flags, -0.0f);
  } else if (smem <= 48 * 1024) {
    dim3 grid((W + kConvTX - 1) / kConvTX, (H + kConvTY - 1) / kConvTY);
    k_convolve_tiled<<<grid, kConvTX * kConvTY, smem, st>>>(in, out, W, H, d_k, kr, kc, flags);
  } else {
    dim3 grid((W + 127) / 128, H);
    k_convolve<<<grid, 128, 0, st>>>(in, out, W, H, d_k, kr, kc, flags);
  }
  ++*launches;
  return cudaGetLastError();
}

// pixels of a window beyond its first output's: kSepR m
static size_t window_halo(int size) { return (size_t)((size | 1) + 2 * (window_kind(size) & 3)) / 8 * 8; }
static size_t smem_x(int size) {
  const size_t cap = (size_t)kRowTile + size - 1, lead = window_kind(size) & 3;
  return sizeof(float) * (((size_t)size + 3 & ~(size_t)3) + 3 * (cap + (lead + cap - 1) / kSepR));
}
static size_t smem_y(int size) {
  return sizeof(float) * (((size_t)size + 3 & ~(size_t)3) + 3 * ((size_t)kColH + size - 1) * kColW);
}

// A separable pass' instance for a size.
#define RTX_BY_SIZE(name, kernel)                               \
  static decltype(&kernel<0, false>) name(int size, bool fma) { \
    switch (window_kind(size)) {                                \
      case 0: return fma ? kernel<0, true> : kernel<0, false>;  \
      case 1: return fma ? kernel<1, true> : kernel<1, false>;  \
      case 2: return fma ? kernel<2, true> : kernel<2, false>;  \
      case 3: return fma ? kernel<3, true> : kernel<3, false>;  \
      case 4: return fma ? kernel<4, true> : kernel<4, false>;  \
      case 5: return fma ? kernel<5, true> : kernel<5, false>;  \
      case 6: return fma ? kernel<6, true> : kernel<6, false>;  \
      default: return fma ? kernel<7, true> : kernel<7, false>; \
    }                                                           \
  }
RTX_BY_SIZE(gauss_x, k_gauss_x)
RTX_BY_SIZE(gauss_y, k_gauss_y)
RTX_BY_SIZE(gauss_x16, k_gauss_x16)
RTX_BY_SIZE(gauss_y16, k_gauss_y16)
#undef RTX_BY_SIZE

// GaussianBlur(size) on `in` (extract_mode: bloom's Extract fused into the
// first pass, and the second pass adds `in` back: Image::Bloom).
// Kernels too large for a shared-memory strip take the direct path, with
// extraction and the final addition as separate elementwise passes (tmp2 is
// then required).
cudaError_t launch_gaussian(const float* in, float* tmp, float* tmp2, float* out, int W, int H,
                            const float* d_w, int size, int extract_mode, float threshold, bool fma,
                            cudaStream_t st, int* launches) {
  cudaError_t e;
  const size_t sx = smem_x(size), sy = smem_y(size);
  const size_t kMaxSmem = 227 * 1024;
  size_t n = (size_t)W * H;
  if (extract_mode && (sx > kMaxSmem || sy > kMaxSmem)) {
    if (!tmp2) return cudaErrorInvalidValue;
    k_extract<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, tmp2, n, threshold);
    k_convolve<<<dim3((W + 127) / 128, H), 128, 0, st>>>(tmp2, tmp, W, H, d_w, 1, size, 0);
    k_convolve<<<dim3((W + 127) / 128, H), 128, 0, st>>>(tmp, tmp2, W, H, d_w, size, 1, 0);
    k_add<<<(unsigned)((3 * n + 255) / 256), 256, 0, st>>>(in, tmp2, out, 3 * n);
    *launches += 4;
    return cudaGetLastError();
  }
  // 16-byte forms: rows of a multiple of four pixels, 16-byte aligned images
  // (size 3 at 64^2: 17.8 -> 15.8 us per call, 49 at 1,024^2: 31 -> 22.4).
  // Down the columns their strips are a third larger: where only one fits an
  // SM but two of the 4-byte form's do (194 to 267 taps), that form is
  // faster (512^2: 201 taps 52.0 -> 45.2 us, 261 taps 63.9 -> 55.4; 1,024^2:
  // 129 -> 121, 166 -> 156; 1920 x 1080: 238 -> 229, 307 -> 299).
  auto al = [](const void* p, uintptr_t m) { return (reinterpret_cast<uintptr_t>(p) & (m - 1)) == 0; };
  const bool quads = W % 4 == 0 && al(in, 16) && al(tmp, 16) && al(out, 16);
  const size_t ws16 = (size_t)size + 3 & ~(size_t)3;
  const size_t sx16 = sizeof(float) * (ws16 + kRowGroup * ((size_t)kRowTile + window_halo(size)) / 8);
  const size_t sy16 = sizeof(float) * (ws16 + 4 * (size_t)kColQ * (kCol16H + window_halo(size)));
  if (quads && sx16 <= kMaxSmem) {
    auto kx = gauss_x16(size, fma);
    if (sx16 > 48 * 1024 && (e = cudaFuncSetAttribute(kx, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx16)))
      return e;
    kx<<<dim3((W + kRowTile - 1) / kRowTile, H), kRowThreads, sx16, st>>>(in, tmp, W, H, d_w, size, extract_mode,
                                                                         threshold, -0.0f, W % 8 == 0 && al(tmp, 32));
  } else if (sx <= kMaxSmem) {
    auto kx = gauss_x(size, fma);
    if (sx > 48 * 1024 && (e = cudaFuncSetAttribute(kx, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx)))
      return e;
    kx<<<dim3((W + kRowTile - 1) / kRowTile, H), kRowThreads, sx, st>>>(in, tmp, W, H, d_w, size, extract_mode,
                                                                       threshold, -0.0f);
  } else {
    k_convolve<<<dim3((W + 127) / 128, H), 128, 0, st>>>(in, tmp, W, H, d_w, 1, size, 0);
  }
  ++*launches;
  const size_t kHalfSmem = 113 * 1024;  // two blocks on an SM, 1 KB each reserved
  if (quads && sy16 <= kMaxSmem && (sy16 <= kHalfSmem || sy > kHalfSmem)) {
    auto ky = gauss_y16(size, fma);
    if (sy16 > 48 * 1024 && (e = cudaFuncSetAttribute(ky, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sy16)))
      return e;
    ky<<<dim3((3 * W / 4 + kColQ - 1) / kColQ, (H + kCol16H - 1) / kCol16H), kCol16Threads, sy16, st>>>(
        tmp, extract_mode ? in : nullptr, out, W, H, d_w, size, -0.0f);
  } else if (sy <= kMaxSmem) {
    auto ky = gauss_y(size, fma);
    if (sy > 48 * 1024 && (e = cudaFuncSetAttribute(ky, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sy)))
      return e;
    ky<<<dim3((W + kColW - 1) / kColW, (H + kColH - 1) / kColH), kColThreads, sy, st>>>(
        tmp, extract_mode ? in : nullptr, out, W, H, d_w, size, -0.0f);
  } else {
    k_convolve<<<dim3((W + 127) / 128, H), 128, 0, st>>>(tmp, out, W, H, d_w, size, 1, 0);
  }
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_edge(const float* in, float* out, int W, int H, cudaStream_t st, int* launches) {
  k_edge<<<dim3((W + 127) / 128, H), 128, 0, st>>>(in, out, W, H);
  ++*launches;
  return cudaGetLastError();
}

}  // namespace rtx
