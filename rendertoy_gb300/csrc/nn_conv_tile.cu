// nn_conv_tile.cu — forward and data-gradient 3 x 3 convolutions on the
// tcgen05 tensor cores from swizzled tensor copies (TMA).
//
// Work unit: a tile of 8 x 16 pixels (the 128 accumulator lanes of one MMA),
// lane m = pixel (m % 8, m / 8).  Per slab of KC input channels (32; 16 where
// a channel count asks for it) one tensor copy brings the tile's halo,
// 10 x 18 pixels of KC channels, into shared memory in the swizzled K-major
// layout whose rows are one pixel (KC * 2 bytes).  The swizzle is a function
// of the address alone, so a descriptor may start at any pixel: tap (dy, dx)
// reads the same halo (dy + 1) * 10 + dx + 1 pixels further on, its eight-lane
// groups one halo row (10 pixels) apart.  Every source byte is copied 1.4
// times per tile and never gathered per tap.
//
// What bounds it: an MMA of 128 pixels x N outputs x 16 channels reads its
// 4 KB A operand from shared memory (32 clocks at 128 B per clock) plus 32 N
// bytes of B, so below N = 128 a step costs about 32 + N / 4 clocks and the
// tensor pipe cannot fill; a tensor copy moves about one row (here 64 B) per
// 1.2 clocks (measured: 52 B per clock and SM for 64-byte rows, 13 B for the
// 16-byte rows of an unswizzled halo, which bounded the row kernels this
// replaces).
//
// k_conv_tile: the order of additions is slab of 16 channels, then tap (rows
// of 64 pixels or more).  Forms:
//   one or two full-resolution sources, MT = 1 or 2 vertically adjacent tiles
//   per unit (2 when weights are streamed: each slab's nine weight tiles then
//   serve 256 pixels);
//   kUp: the first source at half resolution (nearest upsampling).  A tile is
//   8 x 16 low-resolution pixels, i.e. 16 x 32 outputs in four parity classes
//   (py, px), each with its own accumulator.  Output (2 y + py, 2 x + px)
//   reads low pixel (y + floor((py + dy) / 2), x + floor((px + dx) / 2)): for
//   one parity class and tap a constant shift of the low-resolution halo.  A
//   skip source is read through four tensor maps, one per parity plane
//   (strides of two pixels and two rows), in which taps are shifts again.  So
//   neither source is expanded, and weights serve four MMAs per fetch.
// k_conv_narrow: the order of additions is tap, then 16 channels (rows
// shorter than 64 pixels): the tile's halo of all slabs stays resident while
// weights stream by (tap, slabs); an upsampled source is expanded into the
// halo by the copying warps.
//
// Roles (640 threads, one CTA per SM, persistent): warps 0 .. 3 are service
// warps, warps 4 .. 19 four epilogue groups of four.  R = 1, 2 or 4 rings, each
// a set of stages and every R-th tile, as many as stages and accumulators
// allow.  MMAs are issued by one elected lane of a converged warp, so that
// descriptors stay in uniform registers.  Such a warp spends ~800 clocks per
// tile on waits, commits and address work, and only another ring's MMAs fill
// the tensor pipe meanwhile (640 clocks of MMAs per tile of a 32 -> 32 channel
// layer: 88 us with one ring, 63 with four at 32 x 256^2; its data gradient 87
// -> 69).  Up to two rings: one warp issues a ring's MMAs, another its copies;
// four rings: each warp does both, copies one unit behind (with one ring that
// was 25 % slower).  The four-accumulator form has 72 MMAs per unit to hide
// the same work behind: one ring (150 us for d0, 155 with two).
#include <algorithm>
#include <cuda.h>
#include <cudaTypedefs.h>

#include "nn.h"
#include "nn_tile.cuh"
#include "nn_tile.h"

namespace rtx {
namespace nn {

namespace {

constexpr int kService = 4, kEpiWarps = 16, kThreadsT = 32 * (kService + kEpiWarps);
constexpr int kMaxS = 8, kMaxBuf = 8;
constexpr int kHW = 10, kPW = 9;  // halo width: full- and low-resolution tiles, parity planes

// bytes of a unit's A region
__host__ __device__ constexpr uint32_t halo_bytes(int KC, int MT) { return (uint32_t)kHW * (16 * MT + 2) * KC * 2; }
__host__ __device__ constexpr uint32_t plane_bytes(int KC) { return (uint32_t)kPW * 17 * KC * 2; }

struct TileArgs {
  int H, W;                 // output resolution
  int tx, ty, n_tiles;      // tiles per image row / column; images x ty x tx x n-tiles
  int ntn, NT, Nout;        // output-channel tiles of NT (multiples of 16)
  int nslab1, nslab;        // slabs of the first source, of both
  int R, S, nbuf;           // service warps, stages of each one's ring, accumulator buffers
  uint32_t stage, w_off;    // ring stage bytes, weights within a streamed stage
  uint32_t ncols;           // TMEM columns allocated
  // epilogue
  const float* bias;
  int relu;
  bf16* out;
  float* out_f32;
  bf16* pool;               // 2 x 2 averages of the output
  // data gradient: the sources (ReLU mask), and where the gradient goes
  Src s1, s2;
  int mask_relu;
  bf16 *din, *dlow, *dskip;
  KpHead head;              // the output layer with its filter (kHead != 0)
  int* err;
  // narrow form
  int G, nhalo;             // slabs per weight unit, halo buffers
  int up1, C1;              // expand the first source (x1, C1 channels) from half resolution
  const bf16* x1;
};

struct TileMaps {
  CUtensorMap w, s1, s2[4];
};

struct Bars {
  uint64_t full[kMaxS], empty[kMaxS], accf[kMaxBuf], acce[kMaxBuf], wbar;
};

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack2(uint32_t u) {
  return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
}

// 32 bytes to p: one store where p allows it, else two
__device__ __forceinline__ void st32(void* p, const uint32_t* u, bool wide) {
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(u[0]), "r"(u[1]), "r"(u[2]),
                 "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7])
                 : "memory");
  } else {
    uint4* q = reinterpret_cast<uint4*>(p);
    q[0] = make_uint4(u[0], u[1], u[2], u[3]);
    q[1] = make_uint4(u[4], u[5], u[6], u[7]);
  }
}

struct Tile {
  int n, x0, y0, nt;  // image, tile origin (in tiles' own resolution), output-channel tile
};
// Tiles first, first + step, ... in (image, y, x, output tile) order, without
// a division per tile.
struct TileIter {
  int nt, x, y, n, snt, sx, sy, sn;
  __device__ __forceinline__ TileIter(const TileArgs& a, int first, int step) {
    nt = first % a.ntn;
    first /= a.ntn;
    x = first % a.tx;
    first /= a.tx;
    y = first % a.ty;
    n = first / a.ty;
    snt = step % a.ntn;
    step /= a.ntn;
    sx = step % a.tx;
    step /= a.tx;
    sy = step % a.ty;
    sn = step / a.ty;
  }
  __device__ __forceinline__ void next(const TileArgs& a) {
    nt += snt;
    x += sx;
    y += sy;
    n += sn;
    if (nt >= a.ntn) nt -= a.ntn, ++x;
    if (x >= a.tx) x -= a.tx, ++y;
    if (y >= a.ty) y -= a.ty, ++n;
  }
  __device__ __forceinline__ Tile tile(int th) const { return Tile{n, x * 8, y * th, nt}; }
};

// The FP32 sums, in row order, of the 2 x 2 blocks of a warp's 8 x 4 pixels:
// each lane gives its pixel's 16 BF16 channels (u) and receives four channels
// (4 sub ..) of its block's sum.  Warp-wide.
__device__ __forceinline__ int block_sums(const uint32_t* u, int lane, uint4 (*xch)[2], float* s) {
  xch[lane][0] = make_uint4(u[0], u[1], u[2], u[3]);
  xch[lane][1] = make_uint4(u[4], u[5], u[6], u[7]);
  __syncwarp();
  const int lx = lane & 7, ly = lane >> 3, sub = (ly & 1) * 2 + (lx & 1);
  const int base = (ly & ~1) * 8 + (lx & ~1);
#pragma unroll
  for (int k = 0; k < 4; ++k) s[k] = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint2 g = reinterpret_cast<const uint2*>(xch[base + (k >> 1) * 8 + (k & 1)])[sub];
    const float2 g0 = unpack2(g.x), g1 = unpack2(g.y);
    s[0] += g0.x;
    s[1] += g0.y;
    s[2] += g1.x;
    s[3] += g1.y;
  }
  __syncwarp();
  return sub;
}

// 16 output columns (channels c .. c + 15 of this lane's pixel p) of a
// forward convolution.  Warp-wide.
__device__ __forceinline__ void store_fwd(const TileArgs& a, float* v, int c, size_t p, size_t plow, bool ok, int lane,
                                          uint4 (*xch)[2], const float* bias) {
  if (a.bias) {
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
      const float4 b4 = *reinterpret_cast<const float4*>(bias + c + k);
      v[k] += b4.x;
      v[k + 1] += b4.y;
      v[k + 2] += b4.z;
      v[k + 3] += b4.w;
    }
  }
  if (a.relu) {
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = fmaxf(v[k], 0.0f);
  }
  if (a.out) {
    uint32_t u[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) u[k] = pack2(v[2 * k], v[2 * k + 1]);
    if (ok) st32(a.out + p * a.Nout + c, u, (reinterpret_cast<uintptr_t>(a.out) & 31) == 0);
    if (a.pool) {
      float s[4];
      const int sub = block_sums(u, lane, xch, s);
      if (ok)
        *reinterpret_cast<uint2*>(a.pool + plow * a.Nout + c + 4 * sub) =
            make_uint2(pack2(s[0] * 0.25f, s[1] * 0.25f), pack2(s[2] * 0.25f, s[3] * 0.25f));
    }
  }
  if (ok && a.out_f32) {
    float* d = a.out_f32 + p * a.Nout + c;
    const uintptr_t al = reinterpret_cast<uintptr_t>(a.out_f32);
    if ((al & 15) == 0) {
      st32(d, reinterpret_cast<const uint32_t*>(v), (al & 31) == 0);
      st32(d + 8, reinterpret_cast<const uint32_t*>(v) + 8, (al & 31) == 0);
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k) d[k] = v[k];
    }
  }
}

// The same for a data gradient: the ReLU mask (`mk`: the source's 16 BF16
// values), then din, or the two sources' gradients.  Warp-wide.
__device__ __forceinline__ void store_dgrad(const TileArgs& a, float* v, const uint4* mk, int c, size_t p, size_t plow,
                                            bool ok, int lane, uint4 (*xch)[2]) {
  if (a.mask_relu) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(mk);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float2 s = unpack2(w[k]);
      if (!(s.x > 0.0f)) v[2 * k] = 0.0f;
      if (!(s.y > 0.0f)) v[2 * k + 1] = 0.0f;
    }
  }
  uint32_t u[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) u[k] = pack2(v[2 * k], v[2 * k + 1]);
  if (!a.dlow) {
    if (ok) st32(a.din + p * a.Nout + c, u, (reinterpret_cast<uintptr_t>(a.din) & 31) == 0);
  } else if (c >= a.s1.C) {
    if (ok) st32(a.dskip + p * a.s2.C + (c - a.s1.C), u, (reinterpret_cast<uintptr_t>(a.dskip) & 31) == 0);
  } else {
    // gradient of nearest upsampling: the 2 x 2 blocks' sums of the BF16 values
    float s[4];
    const int sub = block_sums(u, lane, xch, s);
    if (ok)
      *reinterpret_cast<uint2*>(a.dlow + plow * a.s1.C + c + 4 * sub) = make_uint2(pack2(s[0], s[1]), pack2(s[2], s[3]));
  }
}

// The output layer's epilogue: the tile's logits become filters in registers
// (a lane's 32 columns are its pixel's), so neither the FP32 logits nor a
// second pass over them exists.  kHead 1 filters the radiance, 2 computes the
// loss and its gradient.  `rad`: the group's 12 x 20 radiance halo (clamped to
// the frame, made safe).  Operations and order as the
// separate kernels (k_kp_apply, k_kp_loss).
// Halo pixels are float4s: a tap is one conflict-free 16-byte load (eight
// neighbouring pixels per quarter warp).
constexpr int kRadRow = 12, kRadTile = 20 * kRadRow;
constexpr int kHeadGroups = kEpiWarps / 4;

// Tap k of pixel (mx, my).  volatile: the second pass over the taps loads them
// again instead of holding 75 values through the softmax's registers.
__device__ __forceinline__ float4 rad_tap(uint32_t rad, int k) {
  float4 c;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(c.x), "=f"(c.y), "=f"(c.z), "=f"(c.w)
               : "r"(rad + ((k / kKpWidth) * kRadRow + k % kKpWidth) * 16));
  return c;
}

template <int kHead>
__device__ __forceinline__ void head_pixel(const TileArgs& a, float* l, uint32_t rad, const float* tgt, size_t p,
                                           size_t pc, bool ok, float& part) {
  float m = l[0];
#pragma unroll
  for (int k = 1; k < kKpTaps; ++k) m = fmaxf(m, l[k]);
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < kKpTaps; ++k) {
    l[k] = expf(l[k] - m);
    s += l[k];
  }
  const float inv_s = 1.0f / s;
  float o[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int k = 0; k < kKpTaps; ++k) {
    l[k] *= inv_s;
    const float4 c = rad_tap(rad, k);
    o[0] += l[k] * c.x;
    o[1] += l[k] * c.y;
    o[2] += l[k] * c.z;
  }
  if constexpr (kHead == 1) {
    if (ok) {
      float* d = a.head.out + 3 * pc;
      d[0] = o[0];
      d[1] = o[1];
      d[2] = o[2];
    }
  } else {
    float g[3], e = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const float d = o[i] - fminf(fmaxf(tgt[i], 0.0f), 65504.0f);
      const float den = o[i] * o[i] + kRelEps;
      e += d * d / den;
      g[i] = 2.0f * d / den * a.head.inv;
    }
    if (ok) part += e;
    // dw_k = sum_c g_c r_c(tap k), formed twice: held, it spills (192 us per
    // 32 x 256^2 minibatch; so 150)
    auto dw = [&](int k) {
      const float4 c = rad_tap(rad, k);
      return g[0] * c.x + g[1] * c.y + g[2] * c.z;
    };
    float t = 0.0f;
#pragma unroll
    for (int k = 0; k < kKpTaps; ++k) t += l[k] * dw(k);
    if (ok) {
      uint32_t u[16];
#pragma unroll
      for (int k = 0; k < 16; ++k)
        u[k] = pack2(2 * k < kKpTaps ? l[2 * k] * (dw(2 * k) - t) : 0.0f,
                     2 * k + 1 < kKpTaps ? l[2 * k + 1] * (dw(2 * k + 1) - t) : 0.0f);
      bf16* d = a.head.dpred + p * kPredCh;
      const bool wide = (reinterpret_cast<uintptr_t>(a.head.dpred) & 31) == 0;
      st32(d, u, wide);
      st32(d + 16, u + 8, wide);
    }
  }
}

// What a tile's head reads from memory: this thread's share of the radiance
// halo and its pixel's target.  Loaded one tile ahead.
struct HeadIn {
  float r[2][3], tgt[3];
};

template <int kHead>
__device__ __forceinline__ void head_load(const TileArgs& a, const Tile& t, int warp, int lane, HeadIn& in) {
  const int tid = ((warp - kService) & 3) * 32 + lane;
  const KpHead& h = a.head;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int i = tid + 128 * j, yy = i / 12, xx = i - 12 * yy;
    if (i < 240) {
      const int y = min(max(t.y0 + yy - 2, 0), h.Hc - 1), x = min(max(t.x0 + xx - 2, 0), h.Wc - 1);
      const float* s = h.rad + (size_t)h.rad_px * (((size_t)t.n * h.Hs + y) * h.Ws + x);
#pragma unroll
      for (int k = 0; k < 3; ++k) in.r[j][k] = __ldg(s + k);
    }
  }
  if (kHead == 2) {
    const int m = (warp & 3) * 32 + lane, x = t.x0 + (m & 7), y = t.y0 + (m >> 3);
    if (x < h.Wc && y < h.Hc) {
      const float* s = h.target + 3 * (((size_t)t.n * a.H + y) * a.W + x);
#pragma unroll
      for (int k = 0; k < 3; ++k) in.tgt[k] = __ldg(s + k);
    }
  }
}

// The group's previous tile must be behind it (its taps are read).  Returns
// false when this warp's wait ran out.
template <int kHead, class Next, class Wait, class Release>
__device__ __forceinline__ bool head_epilogue(const TileArgs& a, const Tile& t, uint32_t tmem, int warp, int lane,
                                              float4* rad, const float* bias, HeadIn& in, double& loss, Next&& next,
                                              Wait&& wait, Release&& release) {
  const int q = warp & 3, tid = ((warp - kService) & 3) * 32 + lane, g = (warp - kService) >> 2;
  const int m = q * 32 + lane, mx = m & 7, my = m >> 3;
  const KpHead& h = a.head;
  const int x = t.x0 + mx, y = t.y0 + my;
  const bool ok = x < h.Wc && y < h.Hc;
  const size_t p = ((size_t)t.n * a.H + y) * a.W + x, pc = ((size_t)t.n * h.Hc + y) * h.Wc + x;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int i = tid + 128 * j, yy = i / 12, xx = i - 12 * yy;
    auto sane = [](float v) { return fminf(fmaxf(v, 0.0f), 65504.0f); };
    if (i < 240) rad[yy * kRadRow + xx] = make_float4(sane(in.r[j][0]), sane(in.r[j][1]), sane(in.r[j][2]), 0.0f);
  }
  const float tgt[3] = {in.tgt[0], in.tgt[1], in.tgt[2]};
  asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
  next(in);
  if (!wait()) return false;
  float v[32];
  tmem_ld32(tmem + ((uint32_t)(q * 32) << 16), v);
  release();
#pragma unroll
  for (int k = 0; k < 28; k += 4) {
    const float4 b4 = *reinterpret_cast<const float4*>(bias + k);
    v[k] += b4.x;
    v[k + 1] += b4.y;
    v[k + 2] += b4.z;
    v[k + 3] += b4.w;
  }
  float part = 0.0f;
  head_pixel<kHead>(a, v, tc::smem_u32(rad + my * kRadRow + mx), tgt, p, pc, ok, part);
  if constexpr (kHead == 2) {
    for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
    loss += (double)part;
  }
  return true;
}

// The epilogue of accumulators [acc0, acc1) of a tile for one warp (its 32
// lanes, every column).  `wait` blocks until the accumulators are complete;
// a data gradient's first mask loads are issued before it.  `release` runs
// once the last column is in registers: the MMAs of a later tile need not
// wait for this one's stores.  Returns false when the wait ran out.
template <bool kUp, bool kDg, class Wait, class Release>
__device__ __forceinline__ bool tile_epilogue(const TileArgs& a, const Tile& t, uint32_t tmem, int acc0, int acc1,
                                              int warp, int lane, uint4 (*xch)[2], const float* bias, Wait&& wait,
                                              Release&& release) {
  const int q = warp & 3;
  const int m = q * 32 + lane, mx = m & 7, my = m >> 3;
  const int n0 = t.nt * a.NT, nt = min(a.NT, a.Nout - n0);
  const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
  bool ready = false;
  for (int acc = acc0; acc < acc1; ++acc) {
    const int x = kUp ? 2 * (t.x0 + mx) + (acc & 1) : t.x0 + mx;
    const int y = kUp ? 2 * (t.y0 + my) + (acc >> 1) : t.y0 + 16 * acc + my;
    const bool ok = x < a.W && y < a.H;
    const size_t p = ((size_t)t.n * a.H + y) * a.W + x;
    const size_t plow = ((size_t)t.n * (a.H >> 1) + (y >> 1)) * (a.W >> 1) + (x >> 1);
    const uint32_t taddr = lanes + acc * a.NT;
    if constexpr (kDg) {
      constexpr int kAhead = 4;  // 16-channel chunks whose mask loads are in flight together
      const size_t p1 = a.s1.up ? plow : p, p2 = a.s2.up ? plow : p;
      for (int c0 = 0; c0 < nt; c0 += 16 * kAhead) {
        uint4 mk[kAhead][2];
        if (a.mask_relu) {
#pragma unroll
          for (int b = 0; b < kAhead; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int c = n0 + c0 + 16 * b + 8 * h;
              mk[b][h] = make_uint4(0, 0, 0, 0);
              if (ok && c0 + 16 * b < nt)
                mk[b][h] = __ldg(reinterpret_cast<const uint4*>(c < a.s1.C ? a.s1.ptr + p1 * a.s1.C + c
                                                                           : a.s2.ptr + p2 * a.s2.C + (c - a.s1.C)));
            }
        }
        if (!ready) {
          if (!wait()) return false;
          ready = true;
        }
#pragma unroll
        for (int b = 0; b < kAhead; ++b) {
          if (c0 + 16 * b >= nt) break;
          float v[16];
          tmem_ld16(taddr + c0 + 16 * b, v);
          if (acc == acc1 - 1 && c0 + 16 * b + 16 >= nt) release();
          store_dgrad(a, v, mk[b], n0 + c0 + 16 * b, p, plow, ok, lane, xch);
        }
      }
    } else {
      if (!ready) {
        if (!wait()) return false;
        ready = true;
      }
      int c = 0;
      for (; c + 32 <= nt; c += 32) {
        float v[32];
        tmem_ld32(taddr + c, v);
        if (acc == acc1 - 1 && c + 32 == nt) release();
        store_fwd(a, v, n0 + c, p, plow, ok, lane, xch, bias);
        store_fwd(a, v + 16, n0 + c + 16, p, plow, ok, lane, xch, bias);
      }
      if (c < nt) {
        float v[16];
        tmem_ld16(taddr + c, v);
        if (acc == acc1 - 1) release();
        store_fwd(a, v, n0 + c, p, plow, ok, lane, xch, bias);
      }
    }
  }
  return true;
}

// swizzled K-major descriptor: 8-row groups `sbo` bytes apart
template <int KC>
__device__ __forceinline__ uint64_t kdesc(uint32_t addr, uint32_t sbo) {
  constexpr uint64_t layout = KC == 32 ? 4 : 6;  // 64- / 32-byte swizzle
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) |
         (layout << 61);
}

__device__ __forceinline__ void bars_init(Bars& b, int S, int readers) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < S; ++i) {
      tc::mbar_init(&b.full[i], 1);
      tc::mbar_init(&b.empty[i], 1);
    }
    for (int i = 0; i < kMaxBuf; ++i) {
      tc::mbar_init(&b.accf[i], 1);
      tc::mbar_init(&b.acce[i], readers);
    }
    tc::mbar_init(&b.wbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
}

template <int KC, int MT, bool kUp, bool kRes, bool kDg, int kHead = 0>
__global__ void __launch_bounds__(kThreadsT, 1) k_conv_tile(const TileArgs a, const __grid_constant__ TileMaps tm) {
  constexpr int NA = kUp ? 4 : MT;
  constexpr int RB = KC * 2;  // bytes of a pixel row
  constexpr int kTH = kUp ? 16 : 16 * MT;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) Bars bars;
  __shared__ uint32_t tmem_slot;
  constexpr bool kXch = !kUp && !kHead;  // exchanges between a 2 x 2 block's lanes
  __shared__ uint4 xch[kXch ? kEpiWarps : 1][32][2];
  __shared__ __align__(16) float bias[kDg ? 4 : 256];
  __shared__ float4 rad[kHead ? kHeadGroups : 1][kHead ? kRadTile : 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_tiles = (int)blockIdx.x < a.n_tiles ? (a.n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  if (warp == 0) tc::tmem_alloc(&tmem_slot, a.ncols);
  bars_init(bars, a.R * a.S, kUp ? kEpiWarps * 32 : 128);
  if (!kDg && a.bias)
    for (int k = tid; k < a.Nout; k += kThreadsT) bias[k] = a.bias[k];
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_slot, smem0 = tc::smem_u32(smem), sw = smem0 + a.R * a.S * a.stage;
  const uint32_t tap_bytes = (uint32_t)a.NT * RB, slab_w = 9 * tap_bytes;
  bool ok = true;
  if (warp < kService) {
    // up to two rings: warps 0, 1 issue MMAs and warps 2, 3 copy; four rings:
    // each warp does both
    const bool both = a.R == 4;
    const int ring = both ? warp : (warp & 1);
    if (ring < a.R) {
      uint64_t* const full = bars.full + ring * a.S;
      uint64_t* const empty = bars.empty + ring * a.S;
      const uint32_t s0 = smem0 + ring * a.S * a.stage, tap16 = tap_bytes >> 4;
      const int mine = n_tiles > ring ? (n_tiles - 1 - ring) / a.R + 1 : 0, units = mine * a.nslab;
      const int first = (int)blockIdx.x + ring * (int)gridDim.x, step = a.R * (int)gridDim.x;
      // the copying side: units in order, one stage behind the MMAs
      TileIter ci(a, first, step);
      int cs = 0, cst = 0, issued = 0;
      auto copy = [&] {
        const Tile t = ci.tile(kTH);
        const bool one = cs < a.nslab1;
        const uint32_t sa = s0 + cst * a.stage;
        uint64_t* const bar = &full[cst];
        if (elect_one()) {
          const uint32_t ab = kUp ? (one ? halo_bytes(KC, 1) : 4 * plane_bytes(KC)) : halo_bytes(KC, MT);
          tc::mbar_arrive_expect_tx(bar, ab + (kRes ? 0u : slab_w));
          if (!kUp || one) {
            tma4(sa, one ? &tm.s1 : &tm.s2[0], (one ? cs : cs - a.nslab1) * KC, t.x0 - 1, t.y0 - 1, t.n, bar);
          } else {
#pragma unroll
            for (int pl = 0; pl < 4; ++pl)  // plane (qy, qx) starts at shift -qy, -qx
              tma4(sa + pl * up1k(plane_bytes(KC)), &tm.s2[pl], (cs - a.nslab1) * KC, t.x0 - (pl & 1),
                   t.y0 - (pl >> 1), t.n, bar);
          }
          if (!kRes) tma3(sa + a.w_off, &tm.w, cs * KC, t.nt * a.NT, 0, bar);
        }
        __syncwarp();
        ++issued;
        if (++cst == a.S) cst = 0;
        if (++cs == a.nslab) {
          cs = 0;
          ci.next(a);
        }
      };
      if (kRes && warp == (both ? 0 : 2) && n_tiles > 0 && elect_one()) {
        tc::mbar_arrive_expect_tx(&bars.wbar, (uint32_t)(a.ntn * a.nslab) * slab_w);
        for (int k = 0; k < a.ntn * a.nslab; ++k)
          tma3(sw + k * slab_w, &tm.w, (k % a.nslab) * KC, (k / a.nslab) * a.NT, 0, &bars.wbar);
      }
      __syncwarp();
      if (both || warp >= 2) {
        while (issued < min(a.S, units)) copy();
        if (!both) {
          int st = 0;
          uint32_t ph = 0;
          while (issued < units) {
            ok = warp_wait(&empty[st], ph);
            if (!ok) break;
            copy();
            if (++st == a.S) {
              st = 0;
              ph ^= 1u;
            }
          }
        }
      }
      const int mmas = both || warp < 2 ? mine : 0;
      if (kRes && mmas > 0) ok = warp_wait(&bars.wbar, 0u);
      TileIter it(a, first, step);
      int st = 0, pst = 0;
      uint32_t ph = 0, eph = 0;  // phases of the stage in use, of the stage to refill
      for (int k = 0; k < mmas && ok; ++k, it.next(a)) {
        const int i = ring + k * a.R, buf = i % a.nbuf, lap = i / a.nbuf;
        ok = warp_wait(&bars.acce[buf], (uint32_t)(lap - 1) & 1u);  // lap 0: a fresh barrier reads complete
        const uint32_t idesc = tc::make_idesc_bf16(128, min(a.NT, a.Nout - it.nt * a.NT));
        const uint32_t d = tmem + buf * NA * a.NT;
        for (int s = 0; s < a.nslab && ok; ++s) {
          ok = warp_wait(&full[st], ph);
          if (!ok) break;
          tc::fence_after();
          const uint32_t sa = s0 + st * a.stage;
          const bool skip = kUp && s >= a.nslab1;
          const uint32_t sb = kRes ? sw + (uint32_t)(it.nt * a.nslab + s) * slab_w : sa + a.w_off;
          const uint64_t bd = kdesc<KC>(sb, 8 * RB);
          const uint64_t ad0 = kdesc<KC>(sa, (skip ? kPW : kHW) * RB);
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < KC / 16; ++ks) {
              const uint64_t ad = ad0 + 2 * ks;
              const bool acc0 = s > 0 || ks > 0;
              if (!skip) {
#pragma unroll
                for (int tap = 0; tap < 9; ++tap) {
                  const int dy = tap / 3 - 1, dx = tap % 3 - 1;
#pragma unroll
                  for (int c = 0; c < NA; ++c) {
                    int off;
                    if (kUp)
                      off = (((c >> 1) + dy + 2) / 2) * kHW + ((c & 1) + dx + 2) / 2;  // floor(./2) + 1
                    else
                      off = (16 * c + (kDg ? 1 - dy : 1 + dy)) * kHW + (kDg ? 1 - dx : 1 + dx);
                    tc::mma_bf16(d + c * a.NT, ad + (uint64_t)(off * RB >> 4), bd + 2 * ks + (uint64_t)tap * tap16,
                                 idesc, acc0 || tap > 0);
                  }
                }
              } else {
#pragma unroll
                for (int tap = 0; tap < 9; ++tap) {
                  const int dy = tap / 3 - 1, dx = tap % 3 - 1;
#pragma unroll
                  for (int c = 0; c < 4; ++c) {
                    // parity plane (qy, qx), shifts oy + qy, ox + qx of it
                    const int Y = (c >> 1) + dy, X = (c & 1) + dx, qy = Y & 1, qx = X & 1;
                    const int oy = (Y - qy) / 2, ox = (X - qx) / 2;
                    const uint32_t off = (2 * qy + qx) * up1k(plane_bytes(KC)) + ((oy + qy) * kPW + ox + qx) * RB;
                    tc::mma_bf16(d + c * a.NT, ad + (uint64_t)(off >> 4), bd + 2 * ks + (uint64_t)tap * tap16, idesc,
                                 acc0 || tap > 0);
                  }
                }
              }
            }
            tc::mma_commit(&empty[st]);
            if (s == a.nslab - 1) tc::mma_commit(&bars.accf[buf]);
          }
          __syncwarp();
          // refill the previous unit's stage (pst) once its MMAs are done:
          // this unit's are queued behind them
          if (both && (k > 0 || s > 0) && issued < units) {
            ok = warp_wait(&empty[pst], eph);
            if (ok) copy();
            if (++pst == a.S) {
              pst = 0;
              eph ^= 1u;
            }
          }
          if (++st == a.S) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
      if (!ok) {
        // a wait ran out: wait (bounded) for the copies issued last on each
        // stage, so that none lands after the CTA has left
        for (int u = max(0, issued - a.S); u < issued; ++u) tc::mbar_wait(&full[u % a.S], (uint32_t)(u / a.S) & 1u);
      }
    }
  } else {
    // Groups of four warps: each takes every groups-th tile, or (kUp) one of
    // each tile's four accumulators.  A group must not be given a buffer
    // whose previous phase it cannot know to be complete, so there are no
    // more groups on alternate tiles than buffers.
    const int g = (warp - kService) >> 2, groups = kUp ? 1 : min(kEpiWarps / 4, a.nbuf),
              g0 = kUp ? 0 : g;
    double loss = 0.0;
    if (g0 < groups) {
      TileIter it(a, (int)(blockIdx.x + g0 * gridDim.x), groups * (int)gridDim.x);
      HeadIn in{};
      if (kHead && g0 < n_tiles) head_load<kHead>(a, it.tile(kTH), warp, lane, in);
      for (int i = g0; i < n_tiles && (kHead || ok); i += groups) {
        // the head's warps share barriers within a tile: they leave together
        if (kHead && !(ok = tc::group_all(1 + g, ok))) break;
        const Tile t = it.tile(kTH);
        it.next(a);
        const int buf = i % a.nbuf, lap = i / a.nbuf;
        auto wait = [&] {
          const bool w = warp_wait(&bars.accf[buf], (uint32_t)lap & 1u);
          tc::fence_after();
          return w;
        };
        auto release = [&] {
          tc::fence_before();
          tc::mbar_arrive(&bars.acce[buf]);
        };
        const uint32_t acc = tmem + buf * NA * a.NT;
        if constexpr (kHead)
          ok = head_epilogue<kHead>(
              a, t, acc, warp, lane, rad[g], bias, in, loss,
              [&](HeadIn& n) {
                if (i + groups < n_tiles) head_load<kHead>(a, it.tile(kTH), warp, lane, n);
              },
              wait, release);
        else
          ok = tile_epilogue<kUp, kDg>(a, t, acc, kUp ? g : 0, kUp ? g + 1 : MT, warp, lane,
                                       xch[kXch ? warp - kService : 0], bias, wait, release);
      }
      if (kHead == 2 && lane == 0) atomicAdd(a.head.loss, loss);
    }
  }
  if (!__syncthreads_and(ok) && lane == 0) atomicOr(a.err, tc::kErrMbarTimeout);
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, a.ncols);
}

// Narrow rows: additions in tap-major order.  The tile's halo of every slab
// stays in shared memory while the weights stream past it in units of one tap
// x G slabs; with two halo buffers the next tile's halo loads meanwhile.  An
// upsampled first source is expanded into the halo by four warps (cp.async),
// the rest arrives by tensor copy.  Warps 2 .. 5 expand, 6 .. 13 are two
// epilogue groups on alternate tiles.
constexpr int kExpandWarps = 4, kNarrowEpi = 8, kThreadsN = 64 + 32 * (kExpandWarps + kNarrowEpi);

struct NarrowBars {
  uint64_t full[kMaxS], empty[kMaxS], accf[2], acce[2], hfull[2], hempty[2];
};

template <int KC, bool kDg>
__global__ void __launch_bounds__(kThreadsN, 1) k_conv_narrow(const TileArgs a, const __grid_constant__ TileMaps tm) {
  constexpr int RB = KC * 2;
  constexpr uint32_t kSlab = up1k(halo_bytes(KC, 1));
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) NarrowBars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ uint4 xch[kNarrowEpi][32][2];
  __shared__ __align__(16) float bias[kDg ? 4 : 256];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_tiles = (int)blockIdx.x < a.n_tiles ? (a.n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  if (warp == 0) tc::tmem_alloc(&tmem_slot, a.ncols);
  if (tid == 0) {
    for (int i = 0; i < a.S; ++i) {
      tc::mbar_init(&bars.full[i], 1);
      tc::mbar_init(&bars.empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bars.accf[i], 1);
      tc::mbar_init(&bars.acce[i], 128);
      tc::mbar_init(&bars.hfull[i], 1 + (a.up1 ? kExpandWarps : 0));
      tc::mbar_init(&bars.hempty[i], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (!kDg && a.bias)
    for (int k = tid; k < a.Nout; k += kThreadsN) bias[k] = a.bias[k];
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_slot, s0 = tc::smem_u32(smem), sw = s0 + a.nhalo * a.nslab * kSlab;
  const uint32_t slab_w = (uint32_t)a.NT * RB;
  const int ngrp = (a.nslab + a.G - 1) / a.G;  // weight units per tap
  bool ok = true;
  if (warp == 0) {
    int st = 0, hb = 0, buf = 0;
    uint32_t ph = 0, hph = 0, bph = 1;
    TileIter it(a, (int)blockIdx.x, (int)gridDim.x);
    for (int i = 0; i < n_tiles && ok; ++i, it.next(a)) {
      ok = warp_wait(&bars.acce[buf], bph) && warp_wait(&bars.hfull[hb], hph);
      const uint32_t idesc = tc::make_idesc_bf16(128, min(a.NT, a.Nout - it.nt * a.NT));
      const uint32_t d = tmem + buf * a.NT, sh = s0 + hb * a.nslab * kSlab;
      int tap = 0, g = 0;
      for (int u = 0; u < 9 * ngrp && ok; ++u) {
        ok = warp_wait(&bars.full[st], ph);
        if (!ok) break;
        tc::fence_after();
        const int dy = tap / 3 - 1, dx = tap - (dy + 1) * 3 - 1;
        const int off = (kDg ? 1 - dy : 1 + dy) * kHW + (kDg ? 1 - dx : 1 + dx);
        const int sl0 = g * a.G, sn = min(a.G, a.nslab - sl0);
        const uint64_t ad = kdesc<KC>(sh + sl0 * kSlab + off * RB, kHW * RB);
        const uint64_t bd = kdesc<KC>(sw + st * a.stage, 8 * RB);
        if (elect_one()) {
          for (int s = 0; s < sn; ++s)
#pragma unroll
            for (int ks = 0; ks < KC / 16; ++ks)
              tc::mma_bf16(d, ad + (uint64_t)(s * (kSlab >> 4) + 2 * ks), bd + (uint64_t)(s * (slab_w >> 4) + 2 * ks), idesc,
                           u > 0 || s > 0 || ks > 0);
          tc::mma_commit(&bars.empty[st]);
          if (u == 9 * ngrp - 1) {
            tc::mma_commit(&bars.hempty[hb]);
            tc::mma_commit(&bars.accf[buf]);
          }
        }
        __syncwarp();
        if (++g == ngrp) {
          g = 0;
          ++tap;
        }
        if (++st == a.S) {
          st = 0;
          ph ^= 1u;
        }
      }
      if (++hb == a.nhalo) {
        hb = 0;
        hph ^= 1u;
      }
      buf ^= 1;
      if (buf == 0) bph ^= 1u;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int st = 0, issued = 0, hb = 0, hissued = 0;
      uint32_t ph = 1, hph = 1;
      const int sk = a.up1 ? a.nslab1 : 0;  // expanded slabs are not copied
      TileIter it(a, (int)blockIdx.x, (int)gridDim.x);
      for (int i = 0; i < n_tiles && ok; ++i, it.next(a)) {
        const Tile t = it.tile(16);
        ok = tc::mbar_wait(&bars.hempty[hb], hph);
        if (!ok) break;
        tc::mbar_arrive_expect_tx(&bars.hfull[hb], (uint32_t)(a.nslab - sk) * halo_bytes(KC, 1));
        for (int s = sk; s < a.nslab; ++s) {
          const bool first = s < a.nslab1;
          tma4(s0 + (hb * a.nslab + s) * kSlab, first ? &tm.s1 : &tm.s2[0], (first ? s : s - a.nslab1) * KC, t.x0 - 1,
               t.y0 - 1, t.n, &bars.hfull[hb]);
        }
        ++hissued;
        if (++hb == a.nhalo) {
          hb = 0;
          hph ^= 1u;
        }
        for (int u = 0; u < 9 * ngrp; ++u) {
          ok = tc::mbar_wait(&bars.empty[st], ph);
          if (!ok) break;
          const int tap = u / ngrp, sl0 = (u - tap * ngrp) * a.G, sn = min(a.G, a.nslab - sl0);
          tc::mbar_arrive_expect_tx(&bars.full[st], (uint32_t)sn * slab_w);
          for (int s = 0; s < sn; ++s)
            tma3(sw + st * a.stage + s * slab_w, &tm.w, (sl0 + s) * KC, t.nt * a.NT, tap, &bars.full[st]);
          ++issued;
          if (++st == a.S) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
      if (!ok) {  // wait (bounded) for the copies in flight before leaving
        for (int u = max(0, issued - a.S); u < issued; ++u) tc::mbar_wait(&bars.full[u % a.S], (uint32_t)(u / a.S) & 1u);
        for (int u = max(0, hissued - a.nhalo); u < hissued; ++u)
          tc::mbar_wait(&bars.hfull[u % a.nhalo], (uint32_t)(u / a.nhalo) & 1u);
      }
    }
  } else if (warp < 2 + kExpandWarps) {
    if (a.up1) {
      constexpr int cpp = KC / 8, pxs = kExpandWarps * 32 / cpp;  // 16-byte chunks per pixel
      const int ch = (tid - 64) % cpp, p0 = (tid - 64) / cpp, Hl = a.H >> 1, Wl = a.W >> 1;
      int hb = 0;
      uint32_t hph = 1;
      TileIter it(a, (int)blockIdx.x, (int)gridDim.x);
      for (int i = 0; i < n_tiles && ok; ++i, it.next(a)) {
        const Tile t = it.tile(16);
        ok = warp_wait(&bars.hempty[hb], hph);
        if (!ok) break;
        for (int h = p0; h < kHW * 18; h += pxs) {
          const int r = h / kHW, X = t.x0 - 1 + (h - kHW * r), Y = t.y0 - 1 + r;
          const bool in = X >= 0 && X < a.W && Y >= 0 && Y < a.H;
          const bf16* px = a.x1 + (in ? (((size_t)t.n * Hl + (Y >> 1)) * Wl + (X >> 1)) * a.C1 : 0) + 8 * ch;
          const uint32_t dst = s0 + hb * a.nslab * kSlab + h * RB + ((KC == 32 ? ch ^ ((h >> 1) & 3) : ch ^ ((h >> 2) & 1)) << 4);
          for (int s = 0; s < a.nslab1; ++s) tc::cp_async16(dst + s * kSlab, px + s * KC, in ? 16u : 0u);
        }
        tc::cp_async_commit();
        tc::cp_async_wait<0>();
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bars.hfull[hb]);
        if (++hb == a.nhalo) {
          hb = 0;
          hph ^= 1u;
        }
      }
    }
  } else {
    const int g = (warp - 2 - kExpandWarps) >> 2;
    TileIter it(a, (int)(blockIdx.x + g * gridDim.x), 2 * (int)gridDim.x);
    for (int i = g; i < n_tiles && ok; i += 2, it.next(a)) {
      const Tile t = it.tile(16);
      ok = tile_epilogue<false, kDg>(
          a, t, tmem + (i & 1) * a.NT, 0, 1, warp, lane, xch[warp - 2 - kExpandWarps], bias,
          [&] {
            const bool w = warp_wait(&bars.accf[i & 1], (uint32_t)(i >> 1) & 1u);
            tc::fence_after();
            return w;
          },
          [&] {
            tc::fence_before();
            tc::mbar_arrive(&bars.acce[i & 1]);
          });
    }
  }
  if (!__syncthreads_and(ok) && lane == 0) atomicOr(a.err, tc::kErrMbarTimeout);
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, a.ncols);
}

}  // namespace

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

static CUtensorMapSwizzle swizzle_of(int KC) {
  return KC == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : (KC == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

bool pixel_map(CUtensorMap* m, const bf16* base, int imgs, int H, int W, int C, int step_x, int step_y, int KC, int bw,
               int bh) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = encoder();
  if (!enc || (reinterpret_cast<uintptr_t>(base) & 15) || C % 8 || H <= 0 || W <= 0) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)imgs};
  const cuuint64_t row = (cuuint64_t)W * step_x * C * 2;
  const cuuint64_t strides[3] = {(cuuint64_t)step_x * C * 2, (cuuint64_t)step_y * row, (cuuint64_t)H * step_y * row};
  const cuuint32_t box[4] = {(cuuint32_t)KC, (cuuint32_t)bw, (cuuint32_t)bh, 1};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_of(KC), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// [rows][9][K] weights as (K, row, tap); a box of (KC, NT, taps) lands tap-major
static bool tap_map(CUtensorMap* m, const bf16* base, int rows, int K, int KC, int NT, int taps) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = encoder();
  if (!enc || (reinterpret_cast<uintptr_t>(base) & 15) || K % 8) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, 9};
  const cuuint64_t strides[2] = {(cuuint64_t)9 * K * 2, (cuuint64_t)K * 2};
  const cuuint32_t box[3] = {(cuuint32_t)KC, (cuuint32_t)NT, (cuuint32_t)taps};
  const cuuint32_t es[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_of(KC), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int tile_sm_count() {
  static const int count = [] {  // once, also with several threads
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 152;
    return n;
  }();
  return count;
}

static uint32_t pow2_cols(uint32_t c) {
  uint32_t p = 32;
  while (p < c) p *= 2;
  return p;
}

constexpr uint32_t kSmem = 208 * 1024;  // dynamic shared memory a CTA may plan with

template <int KC, int MT, bool kUp, bool kRes, bool kDg, int kHead = 0>
static cudaError_t launch_tile(const TileArgs& a, const TileMaps& m, size_t smem, cudaStream_t st) {
  auto k = k_conv_tile<KC, MT, kUp, kRes, kDg, kHead>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e) return e;
  k<<<std::min(a.n_tiles, tile_sm_count()), kThreadsT, smem, st>>>(a, m);
  return cudaGetLastError();
}

// The wide (slab-major) form.  kDg: the data gradient (taps mirrored, single
// source dout).  False: not a shape (or alignment) it takes.
template <int KC, bool kDg, int kHead = 0>
static bool plan_wide(TileArgs a, const Src& x1, const Src& x2, const bf16* w, int imgs, cudaStream_t st,
                      cudaError_t* e) {
  const bool up = !kDg && x1.up;
  const int K = x1.C + x2.C, K1 = x1.C;
  a.nslab1 = K1 / KC;
  a.nslab = K / KC;
  TileMaps m{};
  auto weights = [&](int NT) { return (size_t)9 * NT * KC * 2; };
  // resident weights when they leave room for three halo stages
  const uint32_t stage_a = up ? std::max(up1k(halo_bytes(KC, 1)), x2.ptr ? 4 * up1k(plane_bytes(KC)) : 0u)
                              : up1k(halo_bytes(KC, 1));
  a.ntn = (a.Nout + 255) / 256;
  a.NT = ((a.Nout + a.ntn - 1) / a.ntn + 15) / 16 * 16;
  const int NA1 = up ? 4 : 1;
  const size_t res_bytes = (size_t)a.ntn * a.nslab * weights(a.NT);
  const bool fits = NA1 * a.NT <= 512;
  const bool res = fits && res_bytes + 3 * (size_t)stage_a <= kSmem && res_bytes < (1u << 20);
  int MT = 1;
  if (!res) {
    // streamed weights: two tiles per unit (four parity classes when
    // upsampling), output tiles of at most 128 channels, so that the
    // accumulators of two units fit TMEM and at least two stages fit
    MT = up ? 1 : 2;
    a.ntn = (a.Nout + 127) / 128;
    for (;; ++a.ntn) {
      a.NT = ((a.Nout + a.ntn - 1) / a.ntn + 15) / 16 * 16;
      const size_t s = (up ? stage_a : up1k(halo_bytes(KC, 2))) + up1k((uint32_t)weights(a.NT));
      if (2 * s <= kSmem || a.NT <= 16) break;
    }
  }
  const uint32_t sa = (up || MT == 1) ? stage_a : up1k(halo_bytes(KC, 2));
  a.w_off = sa;
  a.stage = res ? sa : sa + up1k((uint32_t)weights(a.NT));
  a.S = (int)std::min<size_t>(kMaxS, (kSmem - (res ? res_bytes : 0)) / a.stage);
  if (a.S < 2) return false;
  const int NA = up ? 4 : MT;
  a.nbuf = std::min(kMaxBuf, 512 / (NA * a.NT));
  // service warps: each needs two stages and its own accumulator buffers
  const int S = a.S;
  a.R = up ? 1 : (S >= 8 && a.nbuf >= 4 ? 4 : (S >= 4 && a.nbuf >= 2 ? 2 : 1));
  a.nbuf -= a.nbuf % a.R;
  a.S = S / a.R;
  if (!up && a.nbuf < 2) return false;
  a.ncols = pow2_cols(a.nbuf * NA * a.NT);
  const int th = up ? 32 : 16 * MT, tw = up ? 16 : 8;
  a.tx = (a.W + tw - 1) / tw;
  a.ty = (a.H + th - 1) / th;
  const long long T = (long long)imgs * a.tx * a.ty * a.ntn;
  if (T > (1LL << 30)) return false;
  a.n_tiles = (int)T;
  if (!tap_map(&m.w, w, a.Nout, K, KC, a.NT, 9)) return false;
  if (up) {
    if (!pixel_map(&m.s1, x1.ptr, imgs, a.H / 2, a.W / 2, x1.C, 1, 1, KC, kHW, 18)) return false;
    if (x2.ptr)
      for (int pl = 0; pl < 4; ++pl)
        if (!pixel_map(&m.s2[pl], x2.ptr + ((size_t)(pl >> 1) * a.W + (pl & 1)) * x2.C, imgs, a.H / 2, a.W / 2, x2.C, 2,
                       2, KC, kPW, 17))
          return false;
  } else {
    if (!pixel_map(&m.s1, x1.ptr, imgs, a.H, a.W, x1.C, 1, 1, KC, kHW, 16 * MT + 2)) return false;
    if (x2.ptr && !pixel_map(&m.s2[0], x2.ptr, imgs, a.H, a.W, x2.C, 1, 1, KC, kHW, 16 * MT + 2)) return false;
  }
  // past half the SM's shared memory: one CTA per SM (TMEM columns)
  const size_t smem = std::max<size_t>((size_t)a.R * a.S * a.stage + (res ? res_bytes : 0), 116 * 1024);
  if constexpr (kHead) {
    if (up || !res || a.ntn != 1 || a.NT != kPredCh) return false;
    *e = launch_tile<KC, 1, false, true, false, kHead>(a, m, smem, st);
    return true;
  }
  if constexpr (!kDg) {
    if (up) {
      *e = res ? launch_tile<KC, 1, true, true, false>(a, m, smem, st)
               : launch_tile<KC, 1, true, false, false>(a, m, smem, st);
      return true;
    }
  }
  *e = res ? launch_tile<KC, 1, false, true, kDg>(a, m, smem, st) : launch_tile<KC, 2, false, false, kDg>(a, m, smem, st);
  return true;
}

// The narrow (tap-major) form.  Its halo must fit beside two weight units.
static bool narrow_fits(int KC, int K) {
  return (size_t)(K / KC) * up1k(halo_bytes(KC, 1)) + 2 * up1k(128 * KC * 2) <= kSmem;
}

template <int KC, bool kDg>
static bool plan_narrow(TileArgs a, const Src& x1, const Src& x2, const bf16* w, int imgs, cudaStream_t st,
                        cudaError_t* e) {
  const int K = x1.C + x2.C;
  if (!narrow_fits(KC, K)) return false;
  const uint32_t slab = up1k(halo_bytes(KC, 1));
  a.nslab1 = x1.C / KC;
  a.nslab = K / KC;
  a.up1 = x1.up;
  a.C1 = x1.C;
  a.x1 = x1.ptr;
  a.tx = (a.W + 7) / 8;
  a.ty = (a.H + 15) / 16;
  const long long T = (long long)imgs * a.tx * a.ty;
  if (T > (1LL << 24)) return false;
  // Output-channel tiles of at most 128: the split with the shortest rounds
  // of tiles over the SMs (an MMA costs max(N / 2, 32 + N / 4) clocks; a
  // tensor copy one row of its weights per 1.2)
  double best = 0;
  for (int k = (a.Nout + 127) / 128; k <= (a.Nout + 31) / 32; ++k) {
    const int nt = ((a.Nout + k - 1) / k + 15) / 16 * 16, ntn = (a.Nout + nt - 1) / nt;
    const double step = std::max({nt * 0.5, 32 + nt * 0.25, nt * 1.2 * 16 / KC});
    const double cost = (double)((T * ntn + tile_sm_count() - 1) / tile_sm_count()) * (step * 9 * (K / 16) + 3000);
    if (best == 0 || cost < best) best = cost, a.NT = nt, a.ntn = ntn;
  }
  a.n_tiles = (int)(T * a.ntn);
  const size_t unit1 = (size_t)a.NT * KC * 2;
  a.nhalo = (size_t)2 * a.nslab * slab + 4 * up1k((uint32_t)unit1) <= kSmem ? 2 : 1;
  const size_t room = kSmem - (size_t)a.nhalo * a.nslab * slab;
  // weight units of up to 24 KB, of which four fit
  a.G = (int)std::max<size_t>(1, std::min<size_t>({(size_t)a.nslab, 24 * 1024 / unit1, room / 4 / unit1}));
  a.stage = up1k((uint32_t)(a.G * unit1));
  a.S = (int)std::min<size_t>(kMaxS, room / a.stage);
  if (a.S < 2) return false;
  a.nbuf = 2;
  a.ncols = pow2_cols(2 * a.NT);
  TileMaps m{};
  if (!tap_map(&m.w, w, a.Nout, K, KC, a.NT, 1)) return false;
  if (!x1.up && !pixel_map(&m.s1, x1.ptr, imgs, a.H, a.W, x1.C, 1, 1, KC, kHW, 18)) return false;
  if (x2.ptr && !pixel_map(&m.s2[0], x2.ptr, imgs, a.H, a.W, x2.C, 1, 1, KC, kHW, 18)) return false;
  if (x1.up && (reinterpret_cast<uintptr_t>(x1.ptr) & 15)) return false;
  const size_t smem = std::max<size_t>((size_t)a.nhalo * a.nslab * slab + (size_t)a.S * a.stage, 116 * 1024);
  auto k = k_conv_narrow<KC, kDg>;
  if ((*e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))) return true;
  k<<<std::min(a.n_tiles, tile_sm_count()), kThreadsN, smem, st>>>(a, m);
  *e = cudaGetLastError();
  return true;
}

static bool takes_fwd(const ConvFwd& c, bool wide) {
  const int g = c.s2.ptr ? (c.s1.C | c.s2.C) : c.s1.C;
  if (g % 16 || c.Cout % 16 || c.s2.up || (c.s1.up && (c.H % 2 || c.W % 2))) return false;
  if (c.out && (reinterpret_cast<uintptr_t>(c.out) & 15)) return false;
  return wide || narrow_fits(g % 32 == 0 ? 32 : 16, c.Cin);
}

bool conv_tile_fwd(const ConvFwd& c, bool wide, cudaStream_t st, cudaError_t* e) {
  if (!takes_fwd(c, wide)) return false;
  const int g = c.s2.ptr ? (c.s1.C | c.s2.C) : c.s1.C;
  TileArgs a{};
  a.H = c.H;
  a.W = c.W;
  a.Nout = c.Cout;
  a.bias = c.bias;
  a.relu = c.relu;
  a.out = c.out;
  a.out_f32 = c.out_f32;
  a.pool = c.pool;
  a.err = c.err;
  const Src s2 = c.s2.ptr ? c.s2 : Src{nullptr, 0, 0};
  if (!wide)
    return g % 32 == 0 ? plan_narrow<32, false>(a, c.s1, s2, c.w, c.N, st, e)
                       : plan_narrow<16, false>(a, c.s1, s2, c.w, c.N, st, e);
  return g % 32 == 0 ? plan_wide<32, false>(a, c.s1, s2, c.w, c.N, st, e)
                     : plan_wide<16, false>(a, c.s1, s2, c.w, c.N, st, e);
}

bool conv_tile_head(const ConvFwd& c, const KpHead& h, cudaStream_t st, cudaError_t* e) {
  if (c.s1.up || c.s2.ptr || c.s1.C % 32 || c.Cout != kPredCh || !c.bias || c.relu) return false;
  if (h.dpred && (reinterpret_cast<uintptr_t>(h.dpred) & 15)) return false;
  TileArgs a{};
  a.H = c.H;
  a.W = c.W;
  a.Nout = c.Cout;
  a.bias = c.bias;
  a.head = h;
  a.err = c.err;
  const Src none{nullptr, 0, 0};
  return h.out ? plan_wide<32, false, 1>(a, c.s1, none, c.w, c.N, st, e)
               : plan_wide<32, false, 2>(a, c.s1, none, c.w, c.N, st, e);
}

static bool takes_dgrad(const ConvDgrad& c, bool wide) {
  if (c.Cout % 16 || c.Cin % 16) return false;
  return wide || narrow_fits(c.Cout % 32 == 0 ? 32 : 16, c.Cout);
}

bool conv_tile_dgrad(const ConvDgrad& c, bool wide, cudaStream_t st, cudaError_t* e) {
  if (!takes_dgrad(c, wide)) return false;
  TileArgs a{};
  a.H = c.H;
  a.W = c.W;
  a.Nout = c.Cin;
  a.s1 = c.s1;
  a.s2 = c.s2;
  a.mask_relu = c.mask_relu;
  a.din = c.din;
  a.dlow = c.dlow;
  a.dskip = c.dskip;
  a.err = c.err;
  const Src d{c.dout, c.Cout, 0}, none{nullptr, 0, 0};
  if (!wide)
    return c.Cout % 32 == 0 ? plan_narrow<32, true>(a, d, none, c.wt, c.N, st, e)
                            : plan_narrow<16, true>(a, d, none, c.wt, c.N, st, e);
  return c.Cout % 32 == 0 ? plan_wide<32, true>(a, d, none, c.wt, c.N, st, e)
                          : plan_wide<16, true>(a, d, none, c.wt, c.N, st, e);
}

}  // namespace nn
}  // namespace rtx
