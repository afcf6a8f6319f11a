// nn_wgrad_tile.cu — 3 x 3 weight gradients on the tcgen05 tensor cores from
// swizzled tensor copies (TMA):
//   dw[o, t, c] += sum over pixels p of dout[p, o] src[p + off(t), c]
//
// A GEMM over the pixels of 8 x TR-pixel tiles, both operands MN-major (a
// shared-memory row is one pixel's KO outputs or CB source channels).  All
// nine taps of a KO x CB block come from one MMA per 16 pixels: the operands'
// "atoms" (groups of KO or CB elements along M or N) may overlap in shared
// memory, so
//   M = 4 atoms of KO outputs, atom i = the dout tile one pixel row further
//       down (rows y - 1 + i): with the source row fixed that is tap dy = 1 - i
//       (i = 3 is padding),
//   N = 3 atoms of CB channels, atom d = the source tile one pixel further
//       right (columns x - 1 + d): tap dx = d - 1.
// dout carries a halo of one row above and below, the source of one column
// left and right; both read zeros outside the image, so every (pixel, tap)
// pair inside it is counted once.  Against M = the output channels and one
// MMA per tap (the row kernels this replaces) a 32 x 32 block costs 56 clocks
// per 16 pixels instead of 9 x 40, and every byte is copied about once.
//
// A source at half resolution (read upsampled) is expanded into the same
// layout by the eight warps that later run the epilogue: 16-byte cp.async
// copies, one unit ahead.
//
// The bias gradient (sums of dout over the pixels) comes from the same tiles:
// the epilogue warps of the last channel column (the one with least to expand)
// add up each unit's dout rows from shared memory (instead of 131 us of reading
// every dout again per step of 32 x 256^2; in the first column, behind the
// expansion, d1's launch grew from 100 to 174 us).
//
// An infinite or NaN source value in an image's first or last row meets dout's
// zero halo rows (in the last column of a width that is not a multiple of
// eight, dout's zero columns): 0 x inf is NaN, in taps that do not read the
// value.  So rows of sums of those taps that are not all finite are left out and
// formed again from memory, over the pixels of dout alone, once the CTA is done;
// while all values are finite nothing is read twice.  The reverse is not made
// good: an infinite dout value in those rows leaves taps that would read the
// padding beside it as they are, where multiplying the padding would give NaN.
//
// A CTA owns one or more groups of CB channels for one or more blocks of
// outputs and keeps their accumulators in TMEM over a run of tiles.  FP32
// accumulation in the tensor core truncates: a run of n MMAs loses about n 2^-26
// of a sum that grows steadily (measured 1.3e-5 after 864 of them), so a CTA's
// range is cut into runs no longer than the earlier kernels' (run_pixels).  The
// epilogue warps add the runs up in registers, or TMEM holds them side by side,
// and a CTA's sums go to dw once, with FP32 atomics: no more partial sums than
// before either.  Runs of at least 512 pixels, added to dw each, had
// made narrow layers less exact (128 -> 512 pixels: 153 -> 502e-9 relative at
// 8 x 32^2, 96 + 64 -> 64; now 152).
#include <algorithm>
#include <cuda.h>

#include "nn.h"
#include "nn_tile.cuh"
#include "nn_tile.h"

namespace rtx {
namespace nn {

namespace {

constexpr int kThreadsW = 320, kMaxSW = 8, kMaxBlocks = 10;
constexpr int kExpanders = 8;     // warps that expand, sum the bias and run the epilogue
constexpr uint32_t kPad = 4096;   // MMA reads of padding atoms past the last stage
constexpr uint32_t kXch = 2 * 16 * 12 * 4;  // bytes an epilogue warp passes rows through

struct WgradArgs {
  int KO, CB, ao, G;        // block sizes; o-blocks and channel groups of a CTA
  int Cout, Cin;            // outputs; dw's channel stride
  int C1, C2, ng1, ng;      // the sources' channels; channel groups of the first, of both
  int up1;                  // the first source is expanded from half resolution
  const bf16 *x1, *x2, *dout;
  int H, W;
  int ngc;                  // CTA columns: sets of G channel groups (x o-block sets)
  int TR, tx, ty;           // tile rows, tiles per image row / column
  int tiles, per;           // all tiles, tiles per CTA
  int run, sets;            // tiles per run; accumulator sets (of all runs, or two that runs alternate between)
  int S;
  uint32_t stage, dbytes, sbytes, src_off;  // ring stage; bytes of one dout / source box (1 KB steps); source offset
  uint32_t ncols;
  float *dw, *db;
  int* err;
};
struct WgradMaps {
  CUtensorMap dout, src[2];
};

__device__ __forceinline__ uint64_t mn_desc(uint32_t addr, uint32_t atom, uint32_t group, int K) {
  const uint64_t layout = K == 32 ? 4 : 6;  // 64- / 32-byte swizzle
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((atom >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((group >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (layout << 61);
}

__device__ __forceinline__ void add4(float* d, float4 v) {
  if ((reinterpret_cast<uintptr_t>(d) & 15) == 0) {
    atomicAdd(reinterpret_cast<float4*>(d), v);
  } else {
    atomicAdd(d, v.x);
    atomicAdd(d + 1, v.y);
    atomicAdd(d + 2, v.z);
    atomicAdd(d + 3, v.w);
  }
}

// Adds a warp's 32 rows x NC columns (v: this lane's row, m0 the first) to dw
// at tap column d, channels c0 .. of the nc left in the source.  A row is one
// (output, tap), 9 Cin floats from the next, so rows pass through shared memory
// (xw, this warp's): an instruction then adds whole 64-byte (NC = 8: 32-byte)
// pieces of 8 (16) rows instead of 16 bytes of 32 rows (32 x 32^2, 128 -> 128:
// 41.0 -> 26.8 us together with the sums held).  xw holds two
// turns' rows, used alternately: one __syncwarp a turn, an even number of turns.
template <int NC>
__device__ __forceinline__ void add_rows(const WgradArgs& a, float* xw, const float* v, int o0, int m0, int d, int c0,
                                         int nc, int lane) {
  constexpr int kRow = NC + 4, kCh = NC / 4, kRows = 32 / kCh;  // floats a row (padded: distinct banks), pieces, rows a turn
#pragma unroll
  for (int p = 0; p < 32 / kRows; ++p) {
    float* const x = xw + (p & 1) * (kXch / 8);
    if (lane / kRows == p)
#pragma unroll
      for (int e = 0; e < kCh; ++e)
        *reinterpret_cast<float4*>(x + (lane % kRows) * kRow + 4 * e) =
            make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
    __syncwarp();
    const int r = lane / kCh, ch = lane % kCh, m = m0 + kRows * p + r;
    const int atom = a.KO == 32 ? m >> 5 : m >> 4, o = o0 + (m & (a.KO - 1));
    if (atom < 3 && 4 * ch < nc)
      add4(a.dw + ((size_t)o * 9 + (2 - atom) * 3 + d) * a.Cin + c0 + 4 * ch,
           *reinterpret_cast<const float4*>(x + r * kRow + 4 * ch));
  }
}

// NC of a lane's accumulator columns at each of the three tap columns, `step` apart
template <int NC>
__device__ __forceinline__ void load3(uint32_t t, uint32_t step, float (&v)[3][16]) {
  uint32_t r[3][NC];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    uint32_t* const q = r[d];
    if constexpr (NC == 16)
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]), "=r"(q[8]),
            "=r"(q[9]), "=r"(q[10]), "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15])
          : "r"(t + d * step)
          : "memory");
    else
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7])
                   : "r"(t + d * step)
                   : "memory");
  }
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 3 * NC; ++k) v[k / NC][k % NC] = __uint_as_float(r[k / NC][k % NC]);
}

__device__ __forceinline__ void prefetch_map(const void* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}

// Walks a CTA's tiles in order
struct Walk {
  int x, y, img;
  __device__ __forceinline__ Walk(const WgradArgs& a, int t) {
    x = t % a.tx;
    t /= a.tx;
    y = t % a.ty;
    img = t / a.ty;
  }
  __device__ __forceinline__ void next(const WgradArgs& a) {
    if (++x == a.tx) {
      x = 0;
      if (++y == a.ty) {
        y = 0;
        ++img;
      }
    }
  }
};

// kHeld: blocks whose sums over the CTA's runs stay in registers (0: every run
// has accumulators of its own)
template <int kHeld>
__global__ void __launch_bounds__(kThreadsW, 1) k_wgrad_tile(const WgradArgs a, const __grid_constant__ WgradMaps tm) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t full[kMaxSW], empty[kMaxSW], done[2], drained[2];
  __shared__ uint32_t tmem_slot;
  __shared__ float sdb[256];
  // rows (outputs and tap rows) of a block's tap column and an epilogue warp
  // whose sums are formed again
  __shared__ uint32_t redo[kMaxBlocks * 3 * kExpanders];
  __shared__ int again;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gc = (int)blockIdx.x % a.ngc, go = (int)blockIdx.x / a.ngc;
  const int g0 = gc * a.G, gn = min(a.G, a.ng - g0);               // channel groups g0 .. g0 + gn - 1
  const int nup = a.up1 ? max(0, min(gn, a.ng1 - g0)) : 0;         // of which expanded (the first ones)
  const int ob0 = go * a.ao, on = min(a.ao, a.Cout / a.KO - ob0);  // o-blocks
  const bool bias = a.db && gc == a.ngc - 1;                       // this CTA sums dout
  const int t0 = (int)blockIdx.y * a.per, n = max(0, min(a.per, a.tiles - t0));
  if (tid == 64) {  // the maps' fetches overlap what follows
    prefetch_map(&tm.dout);
    if (nup < gn) prefetch_map(&tm.src[g0 + nup < a.ng1 ? 0 : 1]);
  }
  if (warp == 0) tc::tmem_alloc(&tmem_slot, a.ncols);
  if (tid == 32) {
    for (int i = 0; i < a.S; ++i) {
      tc::mbar_init(&full[i], 1 + (nup ? kExpanders : 0));
      tc::mbar_init(&empty[i], 1 + (bias ? kExpanders : 0));
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&done[i], 1);
      tc::mbar_init(&drained[i], kExpanders * 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int k = tid; k < 256; k += kThreadsW) {
    sdb[k] = 0.0f;
    if (k < kMaxBlocks * 3 * kExpanders) redo[k] = 0;
  }
  if (tid == 0) again = 0;
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_slot, s0 = tc::smem_u32(smem);
  const uint32_t ncb = 3 * a.CB;  // accumulator columns of a block
  bool ok = true;
  if (warp == 0) {
    const uint32_t idesc = tc::make_idesc_bf16(128, ncb, true, true);
    const uint32_t drow = 8 * a.KO * 2, srow = 10 * a.CB * 2;       // a pixel row of the tile
    const uint32_t dstep = 2 * drow >> 4, sstep = 2 * srow >> 4;    // 16 pixels further
    int st = 0, left = 0, set = a.sets - 1;
    uint32_t ph = 0, set_ph = 0;  // fresh barriers: the phase before reads complete
    for (int u = 0; u < n && ok; ++u) {
      const bool fresh = left == 0;  // first unit of a run
      if (fresh) {
        left = min(a.run, n - u);
        if (++set == a.sets) {
          set = 0;
          set_ph ^= 1u;
        }
        if (kHeld) ok = warp_wait(&drained[set], set_ph);
      }
      const uint32_t set_col = set * a.ao * a.G * ncb;
      --left;
      ok = ok && warp_wait(&full[st], ph);
      if (!ok) break;
      tc::fence_after();
      const uint32_t sd = s0 + st * a.stage, ss = sd + a.src_off;
      if (elect_one()) {
        for (int o = 0; o < on; ++o) {
          const uint64_t ad = mn_desc(sd + o * a.dbytes, drow, drow, a.KO);
          for (int g = 0; g < gn; ++g) {
            const uint64_t bd = mn_desc(ss + g * a.sbytes, a.CB * 2, srow, a.CB);
            const uint32_t d = tmem + set_col + (o * a.G + g) * ncb;
#pragma unroll 4
            for (int ks = 0; ks < a.TR / 2; ++ks)
              tc::mma_bf16(d, ad + (uint64_t)(ks * dstep), bd + (uint64_t)(ks * sstep), idesc, !fresh || ks > 0);
          }
        }
        tc::mma_commit(&empty[st]);
        if (left == 0 && (kHeld || u == n - 1)) tc::mma_commit(&done[kHeld ? set : 0]);
      }
      __syncwarp();
      if (++st == a.S) {
        st = 0;
        ph ^= 1u;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int st = 0, issued = 0;
      uint32_t ph = 1;
      Walk w(a, t0);
      const uint32_t bytes = (uint32_t)on * (uint32_t)((a.TR + 2) * 8 * a.KO * 2) +
                             (uint32_t)(gn - nup) * (uint32_t)(a.TR * 10 * a.CB * 2);
      for (int u = 0; u < n; ++u, w.next(a)) {
        ok = tc::mbar_wait(&empty[st], ph);
        if (!ok) break;
        const uint32_t sd = s0 + st * a.stage;
        tc::mbar_arrive_expect_tx(&full[st], bytes);
        for (int o = 0; o < on; ++o)
          tma4(sd + o * a.dbytes, &tm.dout, (ob0 + o) * a.KO, w.x * 8, w.y * a.TR - 1, w.img, &full[st]);
        for (int g = nup; g < gn; ++g) {
          const bool first = g0 + g < a.ng1;
          tma4(sd + a.src_off + g * a.sbytes, first ? &tm.src[0] : &tm.src[1],
               (g0 + g - (first ? 0 : a.ng1)) * a.CB, w.x * 8 - 1, w.y * a.TR, w.img, &full[st]);
        }
        ++issued;
        if (++st == a.S) {
          st = 0;
          ph ^= 1u;
        }
      }
      if (!ok)
        for (int u = max(0, issued - a.S); u < issued; ++u) tc::mbar_wait(&full[u % a.S], (uint32_t)(u / a.S) & 1u);
    }
  } else {
    // expand the half-resolution groups: thread -> chunk of 8 channels, every
    // pxs-th pixel of the TR x 10 halo
    const int cpp = a.CB >> 3, ch = (tid - 64) % cpp, p0 = (tid - 64) / cpp, pxs = kExpanders * 32 / cpp;
    const int Hl = a.H >> 1, Wl = a.W >> 1;
    // epilogue: two warps per 32 lanes, each half of a group's channels
    const int q = warp & 3, odd = (warp - 2) >> 2;
    const int nc2 = a.CB >> 1;
    const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16) + odd * nc2;
    const bool taps = q * 32 / a.KO < 3;  // some lane of the warp holds one
    float held[kHeld ? kHeld : 1][3][16];
#pragma unroll
    for (int i = 0; i < 3 * 16 * (kHeld ? kHeld : 1); ++i) held[i / 48][i / 16 % 3][i % 16] = 0.0f;
    float* const xw = reinterpret_cast<float*>(smem + (size_t)a.S * a.stage + kPad) + (warp - 2) * (kXch / 4);
    // block b's tap column d
    auto flush = [&](int b, int d, float* v) {
      const int o = b / a.G, g = b % a.G;
      const bool first = g0 + g < a.ng1;
      const int cl = (g0 + g - (first ? 0 : a.ng1)) * a.CB + odd * nc2;  // channel within its source
      const int c0 = (first ? 0 : a.C1) + cl, nc = (first ? a.C1 : a.C2) - cl;
      const int m = q * 32 + lane, atom = a.KO == 32 ? m >> 5 : m >> 4;
      float t = 0.0f;  // 0, or NaN once a sum is not finite
#pragma unroll
      for (int k = 0; k < 16; ++k) t = __fmaf_rn(v[k], 0.0f, t);
      const bool bad = !(t == 0.0f) && atom < 3 && (atom != 1 || (d == 0 && a.W % 8));  // a tap that may have met dout's zeros
      const uint32_t rows = __ballot_sync(0xffffffffu, bad);
      if (rows) {
        if (lane == 0) redo[(b * 3 + d) * kExpanders + warp - 2] = rows, again = 1;
        if (bad)
#pragma unroll
          for (int k = 0; k < 16; ++k) v[k] = 0.0f;
      }
      if (a.CB == 32)
        add_rows<16>(a, xw, v, (ob0 + o) * a.KO, q * 32, d, c0, nc, lane);
      else
        add_rows<8>(a, xw, v, (ob0 + o) * a.KO, q * 32, d, c0, nc, lane);
    };
    int st = 0, set = 1;
    uint32_t ph = 1, set_ph = 1;
    Walk w(a, t0);
    auto arrive = [&](int stage) {
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&full[stage]);
    };
    // bias: thread -> 8 outputs of one pixel out of every `bps`
    const int bch = a.KO >> 3, bcols = on * bch, bc = (tid - 64) % bcols, bp0 = (tid - 64) / bcols,
              bps = kExpanders * 32 / bcols;
    float bsum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    int bst = 0;
    uint32_t bph = 0;
    auto sum_bias = [&] {
      if (!warp_wait(&full[bst], bph)) return false;
      const uint32_t sd = s0 + bst * a.stage + (bc / bch) * a.dbytes;
      if (bp0 < bps)
        for (int h = 8 + bp0; h < 8 + 8 * a.TR; h += bps) {  // the halo's rows 1 .. TR
          const int ch = (bc % bch) ^ (a.KO == 32 ? (h >> 1) & 3 : (h >> 2) & 1);
          uint4 v;
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                       : "r"(sd + h * a.KO * 2 + (ch << 4)));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            bsum[2 * k] += __uint_as_float(w[k] << 16);
            bsum[2 * k + 1] += __uint_as_float(w[k] & 0xffff0000u);
          }
        }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&empty[bst]);
      if (++bst == a.S) {
        bst = 0;
        bph ^= 1u;
      }
      return true;
    };
    const int step = kHeld ? a.run : n, runs = kHeld ? 1 : (n + a.run - 1) / a.run;
    for (int u0 = 0; u0 < n && ok; u0 += step) {
      const int u1 = min(n, u0 + step);
      if (nup) {
        int prev = -1;
        for (int u = u0; u < u1; ++u, w.next(a)) {
          ok = warp_wait(&empty[st], ph);
          if (!ok) break;
          const uint32_t ss = s0 + st * a.stage + a.src_off;
          for (int h = p0; h < 10 * a.TR; h += pxs) {
            const int r = h / 10, X = w.x * 8 - 1 + (h - 10 * r), Y = w.y * a.TR + r;
            const bool in = X >= 0 && X < a.W && Y < a.H;
            const bf16* px = a.x1 + (((size_t)w.img * Hl + (Y >> 1)) * Wl + (X >> 1)) * a.C1;
            // 64- / 32-byte swizzle of 16-byte chunks
            const uint32_t dst = ss + h * a.CB * 2 + ((a.CB == 32 ? ch ^ ((h >> 1) & 3) : ch ^ ((h >> 2) & 1)) << 4);
            for (int g = 0; g < nup; ++g) {
              const int c = (g0 + g) * a.CB + 8 * ch;
              const bool v = in && c < a.C1;
              tc::cp_async16(dst + g * a.sbytes, v ? px + c : a.x1, v ? 16u : 0u);
            }
          }
          tc::cp_async_commit();
          if (prev >= 0) {
            tc::cp_async_wait<1>();
            arrive(prev);
            if (bias && !(ok = sum_bias())) break;
          }
          prev = st;
          if (++st == a.S) {
            st = 0;
            ph ^= 1u;
          }
        }
        tc::cp_async_wait<0>();
        if (ok && prev >= 0) {
          arrive(prev);
          if (bias) ok = sum_bias();
        }
      } else if (bias) {
        for (int u = u0; u < u1 && ok; ++u) ok = sum_bias();
      }
      if (!kHeld || ++set == a.sets) {
        set = 0;
        set_ph ^= 1u;
      }
      ok = ok && warp_wait(&done[set], set_ph);
      tc::fence_after();
      if (ok && taps) {
        const uint32_t cols = a.ao * a.G * ncb, t = lanes + set * cols;
        if constexpr (kHeld > 0) {
#pragma unroll
          for (int b = 0; b < kHeld; ++b)
            if (b / a.G < on && b % a.G < gn)
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                float v[16];
                if (a.CB == 32) {
                  tmem_ld16(t + b * ncb + d * a.CB, v);
#pragma unroll
                  for (int k = 0; k < 16; ++k) held[b][d][k] += v[k];
                } else {
                  tc::tmem_ld8(t + b * ncb + d * a.CB, v);
#pragma unroll
                  for (int k = 0; k < 8; ++k) held[b][d][k] += v[k];
                }
              }
        } else {
          for (int b = 0; b < a.ao * a.G; ++b) {
            if (b / a.G >= on || b % a.G >= gn) continue;
            float v[3][16] = {};
            for (int r = 0; r < runs; ++r) {
              float w[3][16];
              const uint32_t tr = t + r * cols + b * ncb;
              if (a.CB == 32)
                load3<16>(tr, a.CB, w);
              else
                load3<8>(tr, a.CB, w);
#pragma unroll
              for (int k = 0; k < 48; ++k) v[k / 16][k % 16] += k % 16 < nc2 ? w[k / 16][k % 16] : 0.0f;
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) flush(b, d, v[d]);
          }
        }
      }
      tc::fence_before();
      tc::mbar_arrive(&drained[set]);
    }
    if constexpr (kHeld > 0) {
      if (ok && taps)
#pragma unroll
        for (int b = 0; b < kHeld; ++b)
          if (b / a.G < on && b % a.G < gn)
#pragma unroll
            for (int d = 0; d < 3; ++d) flush(b, d, held[b][d]);
    }
    if (bias && bp0 < bps)
#pragma unroll
      for (int k = 0; k < 8; ++k) atomicAdd(&sdb[8 * bc + k], bsum[k]);
  }
  const bool all = __syncthreads_and(ok);
  if (!all && lane == 0) atomicOr(a.err, tc::kErrMbarTimeout);
  // rows to form again: a warp each, pixel by pixel with zeros outside the image
  for (int i = warp; all && again && i < a.ao * a.G * 3 * kExpanders; i += kThreadsW / 32) {
    for (uint32_t rows = redo[i]; rows; rows &= rows - 1) {
      const int ew = i % kExpanders, d = i / kExpanders % 3, b = i / (3 * kExpanders), g = b % a.G;
      const int m = ((ew + 2) & 3) * 32 + __ffs(rows) - 1, atom = m / a.KO;  // epilogue warp ew + 2's row
      const bool first = g0 + g < a.ng1;
      const int c = (g0 + g - (first ? 0 : a.ng1)) * a.CB + (ew >> 2) * (a.CB >> 1), C = first ? a.C1 : a.C2;
      const int o = (ob0 + b / a.G) * a.KO + m % a.KO, dy = 1 - atom, up = first ? a.up1 : 0;
      const bf16* const src = first ? a.x1 : a.x2;
      for (int ck = c; ck < min(C, c + (a.CB >> 1)); ++ck) {
        float s = 0.0f;
        bool nan = false;
        Walk w(a, t0);
        for (int u = 0; u < n && !nan; ++u, w.next(a)) {
          for (int h = lane; h < 8 * a.TR; h += 32) {
            // the tile's pairs: its columns of dout, its rows of the source
            const int x = w.x * 8 + (h & 7), Y = w.y * a.TR + (h >> 3), y = Y - dy, X = x + d - 1;
            if (x < a.W && Y < a.H && y >= 0 && y < a.H) {
              const float v = __bfloat162float(a.dout[(((size_t)w.img * a.H + y) * a.W + x) * a.Cout + o]);
              const size_t p = ((size_t)w.img * (a.H >> up) + (Y >> up)) * (a.W >> up) + (X >> up);
              s += v * (X >= 0 && X < a.W ? __bfloat162float(src[p * C + ck]) : 0.0f);
            }
          }
          nan = __any_sync(0xffffffffu, s != s);  // and stays so
        }
        for (int j = 16; j > 0; j >>= 1) s += __shfl_xor_sync(0xffffffffu, s, j);
        if (lane == 0) atomicAdd(a.dw + ((size_t)o * 9 + (2 - atom) * 3 + d) * a.Cin + (first ? 0 : a.C1) + ck, s);
      }
    }
  }
  if (bias && tid < on * a.KO) atomicAdd(a.db + ob0 * a.KO + tid, sdb[tid]);
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, a.ncols);
}

// Clocks of the split's estimate, from forced splits of 37 layers: a unit costs
// kUnit and an MMA kMma32 (kMma16 with 16-channel groups), adding a block's sums
// to dw kFlush, taking them into registers kHold, a CTA's start kStart.
constexpr double kUnit = 590, kMma32 = 80, kMma16 = 65, kFlush = 3000, kHold = 300, kStart = 6000;
constexpr uint32_t kSmemW = 212 * 1024;  // the ring and kPad; rows in passing and static arrays take the rest of 227 KB
static_assert(kSmemW + kExpanders * kXch + 3072 <= 227 * 1024, "shared memory of a block");

// Pixels an accumulator may sum before it is added to dw (see the file
// comment): no more than a CTA of the kernels before this one summed, so that
// no weight loses more to truncation than it did.  Rows of 64 pixels or more:
// those kernels' row tiles (32, 64 or 128 pixels wide) shared out over one CTA
// per SM and set of channels -- all of up to 128 where outputs are few, else
// the width (48, 32 or 16) that weighed a set's fixed cost against its number
// -- two for 16 channels.  Narrower rows: about eight CTAs per SM, multiples of
// 64 pixels.
long long run_pixels(const ConvWgrad& c) {
  const long long P = (long long)c.N * c.H * c.W;
  int nr = 0, tw = 0, per_sm = 1;
  if (c.W >= 64 && c.Cin % 16 == 0 && 9 * c.Cout <= 512 && c.Cin >= 64) {
    nr = (c.Cin + 127) / 128;
    tw = 32;
  } else if (c.W >= 64 && c.Cin % 16 == 0 && c.Cout <= 128) {
    long long best = -1;
    for (int cr : {48, 32, 16}) {
      const int k = (c.Cin + cr - 1) / cr;
      const long long cost = (long long)k * (cr + c.Cout / 4 + 8);
      if (cr <= c.Cin && (best < 0 || cost < best)) best = cost, nr = k;
    }
    tw = c.W >= 128 ? 128 : 64;
    per_sm = c.Cin <= 16 ? 2 : 1;
  }
  if (!nr) {
    const long long ranges = std::max(1, 8 * 152 / ((9 * c.Cin + 127) / 128)), per = (P + ranges - 1) / ranges;
    return std::max(64LL, (per + 63) / 64 * 64);
  }
  const long long row = (c.W + tw - 1) / tw, npg = std::max(1, tile_sm_count() * per_sm / nr);
  return ((long long)c.N * c.H * row + npg - 1) / npg * c.W / row;
}

}  // namespace

bool conv_tile_wgrad(const ConvWgrad& c, cudaStream_t st, cudaError_t* e) {
  if (c.Cout % 16 || c.Cout > 256 || c.s1.C % 8 || c.s2.C % 8 || c.s2.up) return false;
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (!aligned(c.dout) || !aligned(c.s1.ptr) || !aligned(c.s2.ptr)) return false;
  if (c.s1.up && (c.H % 2 || c.W % 2)) return false;
  WgradArgs a{};
  a.Cout = c.Cout;
  a.Cin = c.Cin;
  a.C1 = c.s1.C;
  a.C2 = c.s2.ptr ? c.s2.C : 0;
  a.up1 = c.s1.up ? 1 : 0;
  a.x1 = c.s1.ptr;
  a.x2 = c.s2.ptr;
  a.dout = c.dout;
  a.H = c.H;
  a.W = c.W;
  a.dw = c.dw;
  a.db = c.db;
  a.err = c.err;
  a.KO = c.Cout % 32 == 0 ? 32 : 16;
  const int at = c.Cout / a.KO;
  a.CB = std::max(a.C1, a.C2) > 16 ? 32 : 16;
  if (at * 3 * a.CB > 512) a.CB = 16;  // the accumulators of all outputs in 512 columns
  a.ng1 = (a.C1 + a.CB - 1) / a.CB;
  a.ng = a.ng1 + (a.C2 + a.CB - 1) / a.CB;
  auto plan = [&](int TR, int G) {
    a.TR = TR;
    a.G = G;
    a.dbytes = up1k((uint32_t)((TR + 2) * 8 * a.KO * 2));
    a.sbytes = up1k((uint32_t)(TR * 10 * a.CB * 2));
    a.src_off = a.ao * a.dbytes;
    a.stage = a.src_off + G * a.sbytes;
    a.S = (int)std::min<uint32_t>(kMaxSW, (kSmemW - kPad) / a.stage);
    return a.S;
  };
  // The split (tile rows TR, channel groups G and output blocks ao of a CTA)
  // with the shortest estimate.  One block of outputs (up to 32) may take
  // several channel groups, so that dout is read once; more take one.  No split
  // whose number of partial sums exceeds the earlier kernels' (their FP32
  // additions round), unless all do.  Every block of outputs in one CTA, and
  // tiles as tall as fit, left small layers to a handful of CTAs with long
  // flushes (1 x 16^2, 128 -> 160: 23.2 -> 16.6 us per enqueued call; 64 + 32 ->
  // 32: 20.6 -> 16.6; 32 x 64^2, 96 -> 96: 51.9 -> 41.2).
  const long long limit = run_pixels(c), P = (long long)c.N * c.H * c.W, most = (P + limit - 1) / limit;
  const int at_max = std::min(at, 512 / (3 * a.CB));
  int G = 1, held = 0;
  // false: not a split
  auto split = [&](int TR, int g, int o, double* cost, bool* over) {
    a.ao = o;
    G = g;
    if (o * g * 3 * a.CB > 512 || (TR > 8 && c.H <= TR / 2) || plan(TR, g) < (TR > 8 ? 3 : 2)) return false;
    const int px = std::min(8, c.W) * std::min(TR, c.H);  // a full tile's
    if (TR > 8 && px > limit) return false;
    a.tx = (c.W + 7) / 8;
    a.ty = (c.H + TR - 1) / TR;
    a.tiles = (int)((long long)c.N * a.tx * a.ty);  // at most the pixels, which are fewer than 2^31
    a.ngc = (a.ng + g - 1) / g;
    const int columns = a.ngc * ((at + o - 1) / o);
    const int ranges = (int)std::min<long long>(std::max(1, tile_sm_count() / columns), most);
    a.per = (a.tiles + ranges - 1) / ranges;
    // a run of a few tiles counts them as full, a longer one as full as they are on average
    long long run = limit / px;
    if (run >= 4) run = limit * a.tx * a.ty / ((long long)c.H * c.W);
    run = std::max(1LL, std::min<long long>(a.per, run));
    const int runs = (int)((a.per + run - 1) / run), used = (a.tiles + a.per - 1) / a.per;
    a.run = (a.per + runs - 1) / runs;  // equal runs
    // several runs: held in registers where a CTA has one or two blocks, else
    // no more than TMEM has accumulators for
    held = runs > 1 && o * g <= 2 ? o * g : 0;
    a.sets = held ? 2 : runs;
    if (a.sets * o * g * 3 * a.CB > 512) return false;
    *over = used > most;
    const double mmas = (TR / 2) * o * g, unit = kUnit + mmas * (a.CB == 32 ? kMma32 : kMma16);
    const double work = a.per * unit, flush = o * g * kFlush;
    const double waves = (columns * used + tile_sm_count() - 1) / tile_sm_count();
    *cost = waves * (kStart + (held ? std::max(work, runs * o * g * kHold) : work) + flush);
    return true;
  };
  double best = 0, cost;
  bool best_over = true, over;
  int pick[3] = {0, 0, 0};
  for (int o = 1; o <= at_max; ++o)
    for (int g = 1; g <= (at == 1 ? a.ng : 1); ++g)
      for (int TR : {32, 16, 8})
        if (split(TR, g, o, &cost, &over) && (!pick[0] || over < best_over || (over == best_over && cost < best))) {
          best = cost;
          best_over = over;
          pick[0] = TR, pick[1] = g, pick[2] = o;
        }
  if (!pick[0] || !split(pick[0], pick[1], pick[2], &cost, &over)) return false;
  const int TR = pick[0];
  const int columns = a.ngc * ((at + a.ao - 1) / a.ao);
  const uint32_t cols = (uint32_t)(a.sets * a.ao * G * 3 * a.CB);
  for (a.ncols = 32; a.ncols < cols;) a.ncols *= 2;
  WgradMaps m{};
  if (!pixel_map(&m.dout, c.dout, c.N, c.H, c.W, c.Cout, 1, 1, a.KO, 8, TR + 2)) return false;
  if (!c.s1.up && !pixel_map(&m.src[0], c.s1.ptr, c.N, c.H, c.W, a.C1, 1, 1, a.CB, 10, TR)) return false;
  if (a.C2 && !pixel_map(&m.src[1], c.s2.ptr, c.N, c.H, c.W, a.C2, 1, 1, a.CB, 10, TR)) return false;
  // no more stages than units; past half the SM's shared memory where two CTAs'
  // TMEM columns do not fit side by side
  a.S = std::min(a.S, std::max(2, a.per));
  const size_t ring = (size_t)a.S * a.stage + kPad + kExpanders * kXch;
  const size_t smem = a.ncols > 256 ? std::max<size_t>(ring, 116 * 1024) : ring;
  auto k = held == 2 ? k_wgrad_tile<2> : (held == 1 ? k_wgrad_tile<1> : k_wgrad_tile<0>);
  if ((*e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))) return true;
  k<<<dim3(columns, (a.tiles + a.per - 1) / a.per), kThreadsW, smem, st>>>(a, m);
  *e = cudaGetLastError();
  return true;
}

}  // namespace nn
}  // namespace rtx
