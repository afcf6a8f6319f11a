// nn_conv.cu — 3 x 3 convolutions of the denoiser as implicit GEMMs on the
// tcgen05 tensor cores (BF16 operands, FP32 accumulation in TMEM): the choice
// of kernel, and the kernels for channel counts the tiles do not take.
//
// Tensors are NHWC BF16 with channel counts padded to multiples of 8.  A
// convolution reads one or two sources: s1 (optionally at half resolution,
// upsampled by nearest neighbour on the fly) and s2 (a skip connection,
// concatenated after s1's channels); neither the upsampled nor the
// concatenated tensor is ever materialised.
//
//   forward : out[p, o]  = relu?(bias[o] + sum_{t, c} src[p + off(t), c] w[o, t, c])
//             GEMM M = pixels (128 per CTA), N = Cout (<= 256), K = 9 * Cin
//   dgrad   : din[p, c]  = mask(p, c) * sum_{t, o} dout[p - off(t), o] w[o, t, c]
//             GEMM M = pixels, N = Cin (tiles of <= 256), K = 9 * Cout, with
//             the weights re-laid out as wt[c, t, o]; mask = (src > 0) when
//             the source is a ReLU output
//   wgrad   : dw[o, t, c] += sum_p dout[p, o] src[p + off(t), c], all of it in
//             nn_wgrad_tile.cu
// off(t) = (t / 3 - 1, t % 3 - 1).  Out-of-image taps read zero ("same"
// zero padding).
//
// Channel counts that are multiples of 16 run as tiles (nn_conv_tile.cu,
// nn_wgrad_tile.cu).  The gather kernels here: the K range is cut into slices of
// 64; every thread copies its 16-byte chunks of a slice straight
// into shared memory with cp.async (zero-filled where the tap falls outside
// the image), S - 1 slices ahead, into a ring of S stages.  Thread 0 issues the
// slice's MMAs and commits them to the stage's mbarrier; a stage is refilled
// once the MMAs that read it have completed.
#include <algorithm>

#include "nn.h"
#include "nn_tile.h"
#include "tc_core.cuh"

namespace rtx {
namespace nn {

namespace {

constexpr int kSlice = 64;    // K per shared-memory slice
constexpr int kThreads = 256;  // 8 warps: all gather, warps w and w + 4 share accumulator lanes

struct Pix {
  int n, y, x;
};

__device__ __forceinline__ Pix pix_of(long long p, int H, int W) {
  Pix r;
  int hw = H * W;
  r.n = (int)(p / hw);
  int rem = (int)(p - (long long)r.n * hw);
  r.y = rem / W;
  r.x = rem - r.y * W;
  return r;
}

// 8 channels [c, c + 8) of the (virtually concatenated, upsampled) source at
// pixel (n, y, x) of the full-resolution grid; zero outside the image.
__device__ __forceinline__ uint4 src_chunk(const Src& s1, const Src& s2, int N, int H, int W, int n,
                                           int y, int x, int c) {
  uint4 v = make_uint4(0, 0, 0, 0);
  if (y < 0 || y >= H || x < 0 || x >= W) return v;
  if (c < s1.C) {
    if (s1.up) {
      size_t off = (((size_t)n * (H >> 1) + (y >> 1)) * (W >> 1) + (x >> 1)) * s1.C + c;
      v = *reinterpret_cast<const uint4*>(s1.ptr + off);
    } else {
      v = *reinterpret_cast<const uint4*>(s1.ptr + (((size_t)n * H + y) * W + x) * s1.C + c);
    }
  } else if (s2.ptr) {
    int cc = c - s1.C;
    v = *reinterpret_cast<const uint4*>(s2.ptr + (((size_t)n * H + y) * W + x) * s2.C + cc);
  }
  return v;
}

__device__ __forceinline__ void bf16x8_to_f32(uint4 u, float* f) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ uint4 f32_to_bf16x8(const float* f) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// Address of 8 channels [c, c + 8) of the (virtually concatenated,
// upsampled) source at pixel (n, y, x), or nullptr outside the image.
__device__ __forceinline__ const bf16* src_ptr(const Src& s1, const Src& s2, int H, int W, int n, int y, int x,
                                               int c) {
  if (y < 0 || y >= H || x < 0 || x >= W) return nullptr;
  if (c < s1.C) {
    if (s1.up) return s1.ptr + (((size_t)n * (H >> 1) + (y >> 1)) * (W >> 1) + (x >> 1)) * s1.C + c;
    return s1.ptr + (((size_t)n * H + y) * W + x) * s1.C + c;
  }
  if (s2.ptr) return s2.ptr + (((size_t)n * H + y) * W + x) * s2.C + (c - s1.C);
  return nullptr;
}

// 16 bytes from p into shared address dst, zeros when p is null (`base` is a
// valid address the zero-fill form names but does not read)
__device__ __forceinline__ void chunk_async(uint32_t dst, const void* p, const void* base) {
  tc::cp_async16(dst, p ? p : base, p ? 16u : 0u);
}

// Shared set-up of a tensor-core CTA: TMEM columns and S MMA barriers.
__device__ __forceinline__ void tc_begin(uint32_t* tmem_slot, uint64_t* bars, int nbar, uint32_t ncols) {
  if ((threadIdx.x >> 5) == 0) tc::tmem_alloc(tmem_slot, ncols);
  if (threadIdx.x == 0) {
    for (int i = 0; i < nbar; ++i) tc::mbar_init(&bars[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
}

__device__ __forceinline__ void tc_end(uint32_t tmem, uint32_t ncols) {
  tc::fence_before();
  __syncthreads();
  if ((threadIdx.x >> 5) == 0) tc::tmem_dealloc(tmem, ncols);
}

// The S-stage ring over n slices (see the file comment).  load(slice, stage)
// issues this thread's copies of a slice (nothing for slice >= n); mma(stage,
// first) is run by thread 0.  Returns false, uniformly across the CTA, when
// an MMA barrier wait ran out (error flag set); copies are drained either way.
// `done(it)` runs on every thread once slice it's MMAs (and all earlier
// ones) have completed, after the copies of slice it + S - 1 were issued and
// while slice it + 1's MMAs run: the persistent kernels read a finished
// accumulator there.
template <int S, class Load, class Mma, class Done>
__device__ __forceinline__ bool conv_ring(int n, uint64_t* bars, Load&& load, Mma&& mma, Done&& done, int* err) {
  uint32_t parity = 0;
#pragma unroll
  for (int s = 0; s < S - 1; ++s) {
    load(s, s);
    tc::cp_async_commit();
  }
  bool wok = true, ok = true;
  for (int it = 0; it < n; ++it) {
    const int st = it % S;
    tc::cp_async_wait<S - 2>();  // this thread's copies of slice `it` landed
    tc::fence_proxy_async();
    tc::fence_before();  // order the previous done()'s TMEM reads before the barrier
    if (!__syncthreads_and(wok)) {
      ok = false;
      break;
    }
    if (threadIdx.x == 0) {
      tc::fence_after();
      mma(it, st, it == 0);
      tc::mma_commit(&bars[st]);
    }
    if (it > 0) {  // the previous slice's MMAs free its stage for slice it + S - 1
      const int ps = (it - 1) % S;
      wok = tc::mbar_wait(&bars[ps], (parity >> ps) & 1u);
      parity ^= 1u << ps;
    }
    load(it + S - 1, (it + S - 1) % S);
    tc::cp_async_commit();
    if (it > 0 && wok) {
      tc::fence_after();
      done(it - 1);
    }
  }
  if (ok && n > 0) {
    const int ls = (n - 1) % S;
    const bool w = wok && tc::mbar_wait(&bars[ls], (parity >> ls) & 1u);
    ok = __syncthreads_and(w);
    if (ok) {
      tc::fence_after();
      done(n - 1);
    }
  }
  if (!ok && (threadIdx.x & 31) == 0) atomicOr(err, tc::kErrMbarTimeout);
  tc::cp_async_wait_all();
  return ok;
}

// Warp-specialised rings (no CTA-wide barrier per slice).  Thread 0 issues
// the MMAs; producer warp 1 + p (p < S <= 7) owns ring stage p and copies
// units p, p + S, p + 2S, ...: it waits for the stage to be free (empty: the
// MMA commit of the unit S before), issues its 32 lanes' cp.async copies,
// waits for them, fences them to the async proxy and arrives on full (32
// arrivals).  Up to S units are in flight, each warp blocking only on its own
// copies; the MMA thread consumes units in order.  Because a warp's units on
// its stage are exactly one lap apart, every parity wait targets the
// barrier's current or next phase, never one two laps away.
// load(unit, stage, lane) copies with item stride kLoadStride.
constexpr int kProducerWarps = 7;
constexpr int kLoadStride = 32;

// pre(pw, lane) issues copies every MMA needs (resident weights, split over
// the producer warps); the warp waits for them and its 32 lanes arrive on
// wbar (kProducerWarps * 32 arrivals; null: none) before its first unit, so
// that arrival never waits on MMA progress.
template <int S, class Pre, class Load>
__device__ __forceinline__ bool produce(int n, uint64_t* full, uint64_t* empty, uint64_t* wbar, Pre&& pre,
                                        Load&& load) {
  static_assert(S >= 1 && S <= kProducerWarps, "one producer warp per stage");
  const int pw = (threadIdx.x >> 5) - 1, lane = threadIdx.x & 31;
  if (wbar) {
    pre(pw, lane);
    tc::cp_async_commit();
    tc::cp_async_wait<0>();
    tc::fence_proxy_async();
    tc::mbar_arrive(wbar);
  }
  if (pw >= S) return true;
  for (int u = pw; u < n; u += S) {
    if (u >= S && !tc::mbar_wait(&empty[pw], (uint32_t)(u / S - 1) & 1u)) return false;
    load(u, pw, lane);
    tc::cp_async_commit();
    tc::cp_async_wait<0>();
    tc::fence_proxy_async();
    tc::mbar_arrive(&full[pw]);
  }
  return true;
}

// Persistent tiles (kTileThreads = 12 warps): thread 0 issues MMAs, warps
// 1 .. 7 produce, warps 8 .. 11 run the epilogue, warp 8 + q reading
// accumulator lanes 32 q .. 32 q + 31.  A CTA walks n_tiles output tiles of
// nsl slices each; tile i accumulates in TMEM buffer i & 1, so tile i's
// epilogue overlaps tile i + 1's copies and MMAs.  accf[b]: MMA commit after
// a tile's last slice (buffer b complete); acce[b]: the 128 epilogue threads'
// arrivals once they have read buffer b.  mma(unit, stage, buffer, slice)
// and epi(tile, buffer) are the kernel's.
constexpr int kTileThreads = 384;
constexpr int kEpilogue = 128;
constexpr int kMaxStages = 8;

struct TileBars {
  uint64_t full[kMaxStages], empty[kMaxStages], accf[2], acce[2], wbar;
};

template <int S>
__device__ __forceinline__ void tile_bars_init(TileBars& b) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < S; ++i) {
      tc::mbar_init(&b.full[i], kLoadStride);
      tc::mbar_init(&b.empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&b.accf[i], 1);
      tc::mbar_init(&b.acce[i], kEpilogue);
    }
    tc::mbar_init(&b.wbar, kProducerWarps * 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
}

template <int S, class Pre, class Load, class Mma, class Epi>
__device__ __forceinline__ bool ws_tiles(int n_tiles, int nsl, TileBars& b, Pre&& pre, Load&& load, Mma&& mma,
                                         Epi&& epi, int* err) {
  const int tid = threadIdx.x, warp = tid >> 5;
  const int n = n_tiles * nsl;
  bool ok = true;
  if (warp == 0) {
    if (tid == 0) {
      if (n > 0) ok = tc::mbar_wait(&b.wbar, 0u);
      for (int u = 0; u < n && ok; ++u) {
        const int i = u / nsl, s = u - i * nsl, st = u % S, buf = i & 1;
        if (s == 0 && i >= 2) ok = tc::mbar_wait(&b.acce[buf], (uint32_t)((i >> 1) - 1) & 1u);
        if (ok) ok = tc::mbar_wait(&b.full[st], (uint32_t)(u / S) & 1u);
        if (!ok) break;
        tc::fence_after();
        mma(u, st, buf, s);
        tc::mma_commit(&b.empty[st]);
        if (s == nsl - 1) tc::mma_commit(&b.accf[buf]);
      }
    }
  } else if (warp <= kProducerWarps) {
    ok = produce<S>(n, b.full, b.empty, &b.wbar, pre, load);
  } else {
    for (int i = 0; i < n_tiles; ++i) {
      const int buf = i & 1;
      if (!tc::mbar_wait(&b.accf[buf], (uint32_t)(i >> 1) & 1u)) {
        ok = false;
        break;
      }
      tc::fence_after();
      epi(i, buf);
      tc::fence_before();
      tc::mbar_arrive(&b.acce[buf]);
    }
  }
  ok = __syncthreads_and(ok);
  if (!ok && (tid & 31) == 0) atomicOr(err, tc::kErrMbarTimeout);
  return ok;
}

template <int S, class Load, class Mma>
__device__ __forceinline__ bool conv_pipeline(int n, uint64_t* bars, Load&& load, Mma&& mma, int* err) {
  return conv_ring<S>(
      n, bars, load, [&](int, int st, bool first) { mma(st, first); }, [](int) {}, err);
}

}  // namespace

// ---------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------
template <int S>
__global__ void __launch_bounds__(kThreads, 2) k_conv_fwd(ConvFwd a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[S];
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long P = (long long)a.N * a.H * a.W;
  const long long m0 = (long long)blockIdx.x * 128;
  const uint32_t ncols = a.Cout <= 32 ? 32 : (a.Cout <= 64 ? 64 : (a.Cout <= 128 ? 128 : 256));
  const uint32_t a_bytes = 128 * kSlice * 2, stage = a_bytes + (uint32_t)a.Cout * kSlice * 2;
  tc_begin(&tmem_slot, bars, S, ncols);
  const uint32_t tmem = tmem_slot;
  const uint32_t idesc = tc::make_idesc_bf16(128, a.Cout);
  const uint32_t s0 = tc::smem_u32(smem);
  const int K = 9 * a.Cin;
  const int n_slices = (K + kSlice - 1) / kSlice;
  // this thread's 4 tile rows (tid >> 3) + 32 i and its chunk column tid & 7
  const int kc = tid & 7;
  Pix px[4];
  bool pv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    long long p = m0 + (tid >> 3) + 32 * i;
    pv[i] = p < P;
    px[i] = pix_of(pv[i] ? p : 0, a.H, a.W);
  }
  auto load = [&](int slice, int st) {
    if (slice >= n_slices) return;
    const uint32_t sa = s0 + st * stage, sb = sa + a_bytes;
    const int k0 = slice * kSlice, k = k0 + kc * 8;
    const bool kv = k < K;
    const int t = kv ? k / a.Cin : 0, c = k - t * a.Cin;
    const int dy = t / 3 - 1, dx = t % 3 - 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = (tid >> 3) + 32 * i;
      const bf16* p = (pv[i] && kv) ? src_ptr(a.s1, a.s2, a.H, a.W, px[i].n, px[i].y + dy, px[i].x + dx, c) : nullptr;
      chunk_async(sa + tc::tile_offset(row, kc * 8, kSlice), p, a.s1.ptr);
    }
    for (int ch = tid; ch < a.Cout * 8; ch += kThreads) {
      const int row = ch >> 3, kk = (ch & 7) * 8;
      const bf16* p = k0 + kk < K ? a.w + (size_t)row * K + k0 + kk : nullptr;
      chunk_async(sb + tc::tile_offset(row, kk, kSlice), p, a.w);
    }
  };
  auto mma = [&](int st, bool first) {
    const uint32_t a0 = s0 + st * stage, b0 = a0 + a_bytes;
    // consecutive K steps are 256 B apart: +16 in the descriptors' address field
    const uint64_t ad = tc::make_desc(a0, 128, kSlice * 16), bd = tc::make_desc(b0, 128, kSlice * 16);
#pragma unroll
    for (int s = 0; s < kSlice / 16; ++s) tc::mma_bf16(tmem, ad + 16 * s, bd + 16 * s, idesc, !first || s > 0);
  };
  const bool ok = conv_pipeline<S>(n_slices, bars, load, mma, a.err);
  tc::fence_after();
  if (ok) {
    // warp w reads accumulator lanes 32 (w % 4) .. + 31, half w / 4 of the columns
    const int lw = warp & 3, half = a.Cout >> 1;
    const long long p = m0 + lw * 32 + lane;
    const uint32_t taddr = tmem + ((uint32_t)(lw * 32) << 16);
    for (int c0 = (warp >> 2) * half; c0 < (warp >> 2) * half + half; c0 += 8) {
      float v[8];
      tc::tmem_ld8(taddr + c0, v);
      if (p < P) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (a.bias) v[i] += a.bias[c0 + i];
          if (a.relu) v[i] = fmaxf(v[i], 0.0f);
        }
        if (a.out) *reinterpret_cast<uint4*>(a.out + (size_t)p * a.Cout + c0) = f32_to_bf16x8(v);
        if (a.out_f32)
#pragma unroll
          for (int i = 0; i < 8; ++i) a.out_f32[(size_t)p * a.Cout + c0 + i] = v[i];
      }
    }
  }
  tc_end(tmem, ncols);
}

// ---------------------------------------------------------------------------
// forward, row tiles: a tile is 128 consecutive pixels of one image row.  Per
// slice of 16 input channels the producers copy the tile's 3-row halo (pixels
// x0 - 1 .. x0 + 128, 2 chunks of 8 channels each) once; the nine taps are
// the same halo read through descriptors shifted by whole pixels (rows of the
// K-major layout are 16 B apart and the two channel chunks one halo row
// apart, so every shift is a legal start address): one third of the gather
// traffic of k_conv_fwd, one address per copied pixel chunk.  Persistent and
// warp-specialised (ws_tiles): a CTA walks tiles blockIdx.x, + gridDim.x, ...;
// with kRes the whole weight tensor stays in shared memory ([slice][tap]
// tiles of Cout x 16, K-major), otherwise each stage carries its slice's nine
// weight tiles.
// ---------------------------------------------------------------------------
constexpr int kHalo = 130;                                  // pixels x0 - 1 .. x0 + 128
constexpr uint32_t kHaloBytes = 3 * 2 * kHalo * 16;          // rows x chunks x pixels x 16 B

// smem byte offset of chunk c (of 2) of halo pixel h in halo row r
__device__ __forceinline__ uint32_t halo_off(int r, int c, int h) { return ((r * 2 + c) * kHalo + h) * 16; }

template <int S, bool kRes>
__global__ void __launch_bounds__(kTileThreads, 1) k_conv_fwd_rows(ConvFwd a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) TileBars bars;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int TR = (a.W + 127) / 128;  // tiles per image row
  const int T = a.N * a.H * TR;
  const int n_tiles = (int)blockIdx.x < T ? (T - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int nsl = a.Cin / 16;
  const uint32_t ncols = a.Cout <= 32 ? 32 : (a.Cout <= 64 ? 64 : (a.Cout <= 128 ? 128 : 256));
  const uint32_t tap_bytes = (uint32_t)a.Cout * 32;
  const uint32_t stage = kRes ? kHaloBytes : kHaloBytes + 9 * tap_bytes;
  if (warp == 0) tc::tmem_alloc(&tmem_slot, 2 * ncols);
  tile_bars_init<S>(bars);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t idesc = tc::make_idesc_bf16(128, a.Cout);
  const uint32_t s0 = tc::smem_u32(smem), sw = s0 + S * stage;  // sw: resident weights
  auto tile_of = [&](int i, int& n, int& y, int& x0) {
    const int j = (int)blockIdx.x + i * (int)gridDim.x;
    const int row = j / TR;
    x0 = (j - row * TR) * 128;
    n = row / a.H;
    y = row - n * a.H;
  };
  auto weight_tile = [&](uint32_t dst, int q) {  // chunk q of one [slice][tap] tile set
    const int kc = q & 1, o = (q >> 1) % a.Cout, st = (q >> 1) / a.Cout, sl = st / 9, t = st - sl * 9;
    chunk_async(dst + st * tap_bytes + tc::tile_offset(o, 8 * kc, 16),
                a.w + ((size_t)o * 9 + t) * a.Cin + sl * 16 + 8 * kc, a.w);
  };
  auto pre = [&](int pw, int lane) {
    if (kRes)
      for (int q = pw * 32 + lane; q < nsl * 9 * a.Cout * 2; q += kProducerWarps * 32) weight_tile(sw, q);
  };
  auto load = [&](int u, int st, int lane) {
    const int i = u / nsl, s = u - i * nsl;
    int n, y, x0;
    tile_of(i, n, y, x0);
    const uint32_t sh = s0 + st * stage;
    const int c0 = s * 16;
    // neighbouring lanes take the two chunks of one pixel (32 B)
    for (int q = lane; q < 3 * kHalo * 2; q += kLoadStride) {
      const int c = q & 1, h = (q >> 1) % kHalo, r = (q >> 1) / kHalo;
      chunk_async(sh + halo_off(r, c, h), src_ptr(a.s1, a.s2, a.H, a.W, n, y + r - 1, x0 + h - 1, c0 + 8 * c),
                  a.s1.ptr);
    }
    if (!kRes)  // slice s's nine tiles: q -> (tap, row, chunk) with the slice fixed
      for (int q = lane; q < 9 * a.Cout * 2; q += kLoadStride) {
        const int kc = q & 1, o = (q >> 1) % a.Cout, t = (q >> 1) / a.Cout;
        chunk_async(sh + kHaloBytes + t * tap_bytes + tc::tile_offset(o, 8 * kc, 16),
                    a.w + ((size_t)o * 9 + t) * a.Cin + c0 + 8 * kc, a.w);
      }
  };
  auto mma = [&](int, int st, int buf, int s) {
    const uint32_t sh = s0 + st * stage;
    const uint32_t sb = kRes ? sw + (uint32_t)s * 9 * tap_bytes : sh + kHaloBytes;
    // A: pixel groups 128 B apart (SBO), channel chunks one halo row apart
    // (LBO); tap t starts (dy + 1) halo rows and 1 + dx pixels in (offsets in
    // the descriptors' 16-byte address units)
    const uint64_t ah = tc::make_desc(sh, kHalo * 16, 128), bw = tc::make_desc(sb, 128, 256);
    const uint32_t d = tmem + buf * ncols;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
      const int dy = t / 3 - 1, dx = t % 3 - 1;
      tc::mma_bf16(d, ah + ((dy + 1) * 2 * kHalo + 1 + dx), bw + t * (tap_bytes >> 4), idesc, s > 0 || t > 0);
    }
  };
  auto epi = [&](int i, int buf) {
    const int q = warp & 3;  // accumulator lanes 32 q .. 32 q + 31 = pixels
    int n, y, x0;
    tile_of(i, n, y, x0);
    const int x = x0 + q * 32 + lane;
    const size_t p = ((size_t)n * a.H + y) * a.W + x;
    const uint32_t taddr = tmem + buf * ncols + ((uint32_t)(q * 32) << 16);
    for (int c0 = 0; c0 < a.Cout; c0 += 8) {
      float v[8];
      tc::tmem_ld8(taddr + c0, v);
      if (x < a.W) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (a.bias) v[k] += a.bias[c0 + k];
          if (a.relu) v[k] = fmaxf(v[k], 0.0f);
        }
        if (a.out) *reinterpret_cast<uint4*>(a.out + p * a.Cout + c0) = f32_to_bf16x8(v);
        if (a.out_f32)
#pragma unroll
          for (int k = 0; k < 8; ++k) a.out_f32[p * a.Cout + c0 + k] = v[k];
      }
    }
  };
  ws_tiles<S>(n_tiles, nsl, bars, pre, load, mma, epi, a.err);
  tc_end(tmem, 2 * ncols);
}

// ---------------------------------------------------------------------------
// data gradient
// ---------------------------------------------------------------------------
template <int S>
__global__ void __launch_bounds__(kThreads, 2) k_conv_dgrad(ConvDgrad a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[S];
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long P = (long long)a.N * a.H * a.W;
  const long long m0 = (long long)blockIdx.x * 128;
  const int n0 = blockIdx.y * 256;
  const int NT = min(256, a.Cin - n0);  // output channels of this CTA
  const uint32_t ncols = NT <= 32 ? 32 : (NT <= 64 ? 64 : (NT <= 128 ? 128 : 256));
  const uint32_t a_bytes = 128 * kSlice * 2, stage = a_bytes + (uint32_t)min(256, a.Cin) * kSlice * 2;
  tc_begin(&tmem_slot, bars, S, ncols);
  const uint32_t tmem = tmem_slot;
  const uint32_t idesc = tc::make_idesc_bf16(128, NT);
  const uint32_t s0 = tc::smem_u32(smem);
  const int K = 9 * a.Cout;
  const int n_slices = (K + kSlice - 1) / kSlice;
  const int kc = tid & 7;
  Pix px[4];
  bool pv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    long long p = m0 + (tid >> 3) + 32 * i;
    pv[i] = p < P;
    px[i] = pix_of(pv[i] ? p : 0, a.H, a.W);
  }
  auto load = [&](int slice, int st) {
    if (slice >= n_slices) return;
    const uint32_t sa = s0 + st * stage, sb = sa + a_bytes;
    const int k0 = slice * kSlice, k = k0 + kc * 8;
    const bool kv = k < K;
    const int t = kv ? k / a.Cout : 0, o = k - t * a.Cout;
    const int dy = t / 3 - 1, dx = t % 3 - 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = (tid >> 3) + 32 * i;
      const int yy = px[i].y - dy, xx = px[i].x - dx;
      const bf16* p = (pv[i] && kv && yy >= 0 && yy < a.H && xx >= 0 && xx < a.W)
                          ? a.dout + (((size_t)px[i].n * a.H + yy) * a.W + xx) * a.Cout + o
                          : nullptr;
      chunk_async(sa + tc::tile_offset(row, kc * 8, kSlice), p, a.dout);
    }
    for (int ch = tid; ch < NT * 8; ch += kThreads) {
      const int row = ch >> 3, kk = (ch & 7) * 8;
      const bf16* p = k0 + kk < K ? a.wt + (size_t)(n0 + row) * K + k0 + kk : nullptr;
      chunk_async(sb + tc::tile_offset(row, kk, kSlice), p, a.wt);
    }
  };
  auto mma = [&](int st, bool first) {
    const uint32_t a0 = s0 + st * stage, b0 = a0 + a_bytes;
    // consecutive K steps are 256 B apart: +16 in the descriptors' address field
    const uint64_t ad = tc::make_desc(a0, 128, kSlice * 16), bd = tc::make_desc(b0, 128, kSlice * 16);
#pragma unroll
    for (int s = 0; s < kSlice / 16; ++s) tc::mma_bf16(tmem, ad + 16 * s, bd + 16 * s, idesc, !first || s > 0);
  };
  const bool ok = conv_pipeline<S>(n_slices, bars, load, mma, a.err);
  tc::fence_after();
  if (ok) {
    const int lw = warp & 3, half = NT >> 1;
    const long long p = m0 + lw * 32 + lane;
    const uint32_t taddr = tmem + ((uint32_t)(lw * 32) << 16);
    Pix q = pix_of(p < P ? p : 0, a.H, a.W);
    for (int c0 = (warp >> 2) * half; c0 < (warp >> 2) * half + half; c0 += 8) {
      float v[8];
      tc::tmem_ld8(taddr + c0, v);
      if (p < P) {
        if (a.mask_relu) {
          float sv[8];
          bf16x8_to_f32(src_chunk(a.s1, a.s2, a.N, a.H, a.W, q.n, q.y, q.x, n0 + c0), sv);
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (!(sv[i] > 0.0f)) v[i] = 0.0f;
        }
        *reinterpret_cast<uint4*>(a.din + (size_t)p * a.Cin + n0 + c0) = f32_to_bf16x8(v);
      }
    }
  }
  tc_end(tmem, ncols);
}

// ---------------------------------------------------------------------------
// Stages of the ring for a B tile of nb rows: 3 stages up to 128 rows, 2
// beyond (72 KB per CTA for nb <= 64, at most 96 KB otherwise).
static int stages_for(int nb) { return nb <= 128 ? 3 : 2; }

// Ring depth of a gather kernel: stages_for(nb), except that a grid of
// fewer CTAs than SMs (the 16- and 32-pixel-wide levels at small batches)
// whose stages are too large for three gets four (one CTA per SM), so that
// more slices' copies are in flight along each CTA's K loop: 160 output
// channels at 16^2 x 8, 44.8 -> 35.4 us (forward) and 64.6 -> 45.8 us (data
// gradient); three -> six stages measured no faster.
static int gather_stages(int nb, dim3 grid, size_t stage_bytes);

template <class K4, class K3, class K2, class Args>
static cudaError_t launch_staged(K4 k4, K3 k3, K2 k2, int stages, dim3 grid, size_t stage_bytes, const Args& a,
                                 cudaStream_t st, size_t extra = 0) {
  size_t smem = stage_bytes * stages + extra;
  cudaError_t e;
  if (stages == 4) {
    if ((e = cudaFuncSetAttribute(k4, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))) return e;
    k4<<<grid, kThreads, smem, st>>>(a);
  } else if (stages == 3) {
    if ((e = cudaFuncSetAttribute(k3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))) return e;
    k3<<<grid, kThreads, smem, st>>>(a);
  } else {
    if ((e = cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))) return e;
    k2<<<grid, kThreads, smem, st>>>(a);
  }
  return cudaGetLastError();
}

static int gather_stages(int nb, dim3 grid, size_t stage_bytes) {
  const int base = stages_for(nb);
  const long long ctas = (long long)grid.x * grid.y * grid.z;
  return (base == 2 && ctas < tile_sm_count() && 4 * stage_bytes <= 200 * 1024) ? 4 : base;
}

// Row tiles pay off once a row holds at least half a tile; they need input
// slices of 16 channels.
static bool use_rows(int W, int Ck) { return W >= 64 && Ck % 16 == 0; }

// Persistent tile kernels (ws_tiles): one CTA per SM, shared memory padded
// past half the SM so that a second CTA never waits on the first one's TMEM
// columns.  Resident weights take a 7-stage halo ring; streamed weights the
// deepest ring (6, 4 or 2 stages) that fits 200 KB.
template <class KR, class K6, class K4, class K2>
static cudaError_t launch_tiles(KR kr, K6 k6, K4 k4, K2 k2, bool res, size_t stage, size_t res_bytes, long long T,
                                const ConvFwd& a, cudaStream_t st) {
  if (T <= 0) return cudaSuccess;
  int S = 7;
  size_t smem = 7 * stage + res_bytes;
  if (!res) {
    S = 6 * stage <= 200 * 1024 ? 6 : (4 * stage <= 200 * 1024 ? 4 : 2);
    smem = S * stage;
  }
  smem = std::max(smem, (size_t)116 * 1024);
  const unsigned grid = (unsigned)std::min<long long>(T, tile_sm_count());
  cudaError_t e;
#define RTX_LAUNCH_TILES(K)                                                                          \
  if ((e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))) return e; \
  K<<<grid, kTileThreads, smem, st>>>(a);
  if (res) {
    RTX_LAUNCH_TILES(kr)
  } else if (S == 6) {
    RTX_LAUNCH_TILES(k6)
  } else if (S == 4) {
    RTX_LAUNCH_TILES(k4)
  } else {
    RTX_LAUNCH_TILES(k2)
  }
#undef RTX_LAUNCH_TILES
  return cudaGetLastError();
}

// weights kept in shared memory by the persistent kernels up to this size
// (128 KB: with 1 KB-aligned tensor-copy halo stages, 7 x 13 KB + 128 KB
// fits the 227 KB of a CTA; measured 0.75 % faster per training step than 96)
constexpr size_t kResidentWeights = 128 * 1024;

cudaError_t conv_fwd(const ConvFwd& a, cudaStream_t st) {
  long long P = (long long)a.N * a.H * a.W;
  if (a.Cout % 16 || a.Cout > 256 || a.Cin % 8) return cudaErrorInvalidValue;
  if (a.pool && (a.s1.up || !a.out || a.H % 2 || a.W % 2)) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  if (conv_tile_fwd(a, use_rows(a.W, a.Cin), st, &e)) return e;
  if (a.pool) return cudaErrorNotSupported;  // only the tile kernels pool
  if (use_rows(a.W, a.Cin)) {
    const size_t wbytes = (size_t)9 * a.Cin * a.Cout * 2;
    const bool res = wbytes <= kResidentWeights;
    const size_t stage = res ? kHaloBytes : kHaloBytes + (size_t)9 * a.Cout * 32;
    const long long T = (long long)a.N * a.H * ((a.W + 127) / 128);
    return launch_tiles(k_conv_fwd_rows<7, true>, k_conv_fwd_rows<6, false>, k_conv_fwd_rows<4, false>,
                        k_conv_fwd_rows<2, false>, res, stage, res ? wbytes : 0, T, a, st);
  }
  size_t stage = 128 * kSlice * 2 + (size_t)a.Cout * kSlice * 2;
  const dim3 grid((unsigned)((P + 127) / 128));
  return launch_staged(k_conv_fwd<4>, k_conv_fwd<3>, k_conv_fwd<2>, gather_stages(a.Cout, grid, stage), grid,
                       stage, a, st);
}

bool conv_head(const ConvFwd& a, const KpHead& h, cudaStream_t st, cudaError_t* e) {
  return use_rows(a.W, a.Cin) && conv_tile_head(a, h, st, e);
}

cudaError_t conv_dgrad(const ConvDgrad& a, cudaStream_t st) {
  long long P = (long long)a.N * a.H * a.W;
  if (a.Cin % 16 || a.Cout % 8) return cudaErrorInvalidValue;
  if (a.dlow && (!a.s1.up || !a.s2.ptr || a.s1.C % 16 || a.H % 2 || a.W % 2)) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  if (conv_tile_dgrad(a, use_rows(a.W, a.Cout), st, &e)) return e;
  if (a.dlow || a.dskip) return cudaErrorNotSupported;  // only the tile kernel splits its output
  int nb = std::min(256, a.Cin);
  size_t stage = 128 * kSlice * 2 + (size_t)nb * kSlice * 2;
  const dim3 grid((unsigned)((P + 127) / 128), (a.Cin + 255) / 256);
  return launch_staged(k_conv_dgrad<4>, k_conv_dgrad<3>, k_conv_dgrad<2>, gather_stages(nb, grid, stage), grid,
                       stage, a, st);
}

cudaError_t conv_wgrad(const ConvWgrad& a, cudaStream_t st) {
  long long P = (long long)a.N * a.H * a.W;
  if (P >= (1LL << 31) || a.Cout % 16 || a.Cout > 256) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  return conv_tile_wgrad(a, st, &e) ? e : cudaErrorNotSupported;  // it takes every shape allowed here
}

}  // namespace nn
}  // namespace rtx
