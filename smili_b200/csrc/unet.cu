// BF16 kernels of the warm-start U-Net (no reference counterpart).
//
// Activations are NHWC bf16 with an explicit channel stride (`ld`), so a
// layer can read or write a channel slice of a wider buffer: the decoder's
// concatenation of the upsampled path and the encoder skip is one buffer
// that two producers write into, with no copy.  Weights are [Cout][3][3][Cin]
// bf16 (FP32 master copies live with the optimiser).  Every contraction
// accumulates in FP32 on the tensor cores (mma.sync m16n8k16 bf16).
//
// conv3x3 (pad 1, stride 1) is an implicit GEMM: D[pixel][cout] =
// sum over (ky, kx, cin) of X[pixel + (ky-1, kx-1)][cin] W[cout][ky][kx][cin].
// A CTA owns an 8 x 16 pixel tile (one m16 row block per warp) and a chunk of
// 8*NT output channels; it stages a (8+2) x (16+2) input halo and the weight
// slab of one 16-channel input chunk in shared memory at a time.
// The data gradient is the same kernel on the ReLU-masked output gradient
// with flipped, transposed weights; the weight gradient is a second
// implicit GEMM over pixels with deterministic per-split partial sums.
// Convolutions whose input rows and weights TMA can address (Cin and the
// channel stride multiples of 8, 16-byte aligned bases) run instead on the
// tcgen05 tensor cores with the accumulator in tensor memory (conv_tc.cuh),
// and so do weight gradients whose channel counts and strides are multiples
// of 8; the mma.sync kernels below take the rest (the one-channel input and
// output layers).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "../../include/smili_unet.h"
#include "conv_tc.cuh"

namespace {

constexpr int TH = 8, TW = 16;          // pixel tile of one CTA
constexpr int KC = 16;                  // input channels per staged chunk
constexpr int KP = KC + 8;              // padded channel stride in shared memory (conflict-free)
constexpr int HALO_H = TH + 2, HALO_W = TW + 2;

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t ld32(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// ---------------------------------------------------------------------------
// Eight bf16 channels as one 16-byte access: the elementwise kernels below take
// it where every channel count and stride is a multiple of 8 and the bases
// are 16-byte aligned, and single elements elsewhere.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(u[i] << 16);
    f[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 v;
  v.x = pack2(__float2bfloat16(f[0]), __float2bfloat16(f[1]));
  v.y = pack2(__float2bfloat16(f[2]), __float2bfloat16(f[3]));
  v.z = pack2(__float2bfloat16(f[4]), __float2bfloat16(f[5]));
  v.w = pack2(__float2bfloat16(f[6]), __float2bfloat16(f[7]));
  return v;
}
__device__ __forceinline__ uint4 ld8(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void st8(__nv_bfloat16* p, const uint4& v) { *reinterpret_cast<uint4*>(p) = v; }

// dy where y > 0, else 0 (also where y is NaN)
__device__ __forceinline__ uint32_t mask2(uint32_t y, uint32_t dy) {
  const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
  return dy & __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&y), zero);
}
__device__ __forceinline__ uint4 mask8(const uint4& y, const uint4& d) {
  return make_uint4(mask2(y.x, d.x), mask2(y.y, d.y), mask2(y.z, d.z), mask2(y.w, d.w));
}

// ---------------------------------------------------------------------------
// conv3x3 forward / data-gradient
// ---------------------------------------------------------------------------
struct ConvArgs {
  const __nv_bfloat16* x;
  int N, H, W, Cin, ldx;
  const __nv_bfloat16* w;  // [Cout][3][3][Cin]
  const float* bias;       // [Cout] or null
  __nv_bfloat16* y;
  int ldy, Cout;
  int relu, accumulate;
  int tiles_x, tiles_y;
};

template <int NT>
__global__ void __launch_bounds__(256) conv3x3_kernel(ConvArgs a) {
  __shared__ __align__(16) __nv_bfloat16 halo[HALO_H * HALO_W * KP];
  __shared__ __align__(16) __nv_bfloat16 wsm[NT * 8 * 9 * KP];
  const int tile = blockIdx.x;
  const int tx = tile % a.tiles_x;
  const int ty = (tile / a.tiles_x) % a.tiles_y;
  const int n = tile / (a.tiles_x * a.tiles_y);
  const int x0 = tx * TW, y0 = ty * TH;
  const int co0 = blockIdx.y * NT * 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  const bool vec = (a.Cin % 8 == 0) && (a.ldx % 8 == 0) && ((reinterpret_cast<uintptr_t>(a.x) & 15) == 0);
  const bool wvec = (a.Cin % 8 == 0) && ((reinterpret_cast<uintptr_t>(a.w) & 15) == 0);
  for (int ci0 = 0; ci0 < a.Cin; ci0 += KC) {
    __syncthreads();
    // input halo: HALO_H x HALO_W pixels x KC channels (zero outside the image / channels)
    if (vec) {
      for (int q = threadIdx.x; q < HALO_H * HALO_W * 2; q += blockDim.x) {
        const int pix = q >> 1, half = q & 1;
        const int hy = pix / HALO_W, hx = pix - hy * HALO_W;
        const int iy = y0 + hy - 1, ix = x0 + hx - 1;
        const int c = ci0 + half * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (iy >= 0 && iy < a.H && ix >= 0 && ix < a.W && c < a.Cin)
          v = *reinterpret_cast<const uint4*>(a.x + (((size_t)n * a.H + iy) * a.W + ix) * a.ldx + c);
        *reinterpret_cast<uint4*>(halo + pix * KP + half * 8) = v;
      }
    } else {
      for (int q = threadIdx.x; q < HALO_H * HALO_W * KC; q += blockDim.x) {
        const int pix = q / KC, c = q - pix * KC;
        const int hy = pix / HALO_W, hx = pix - hy * HALO_W;
        const int iy = y0 + hy - 1, ix = x0 + hx - 1;
        __nv_bfloat16 v = zero;
        if (iy >= 0 && iy < a.H && ix >= 0 && ix < a.W && ci0 + c < a.Cin)
          v = a.x[(((size_t)n * a.H + iy) * a.W + ix) * a.ldx + ci0 + c];
        halo[pix * KP + c] = v;
      }
    }
    // weights: (NT*8) output channels x 9 taps x KC input channels
    if (wvec) {
      for (int q = threadIdx.x; q < NT * 8 * 9 * 2; q += blockDim.x) {
        const int row = q >> 1, half = q & 1;  // row = co_local * 9 + tap
        const int col = row / 9, tap = row - col * 9;
        const int co = co0 + col, c = ci0 + half * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (co < a.Cout && c < a.Cin)
          v = *reinterpret_cast<const uint4*>(a.w + ((size_t)co * 9 + tap) * a.Cin + c);
        *reinterpret_cast<uint4*>(wsm + row * KP + half * 8) = v;
      }
    } else {
      for (int q = threadIdx.x; q < NT * 8 * 9 * KC; q += blockDim.x) {
        const int row = q / KC, c = q - row * KC;
        const int col = row / 9, tap = row - col * 9;
        const int co = co0 + col;
        __nv_bfloat16 v = zero;
        if (co < a.Cout && ci0 + c < a.Cin) v = a.w[((size_t)co * 9 + tap) * a.Cin + ci0 + c];
        wsm[row * KP + c] = v;
      }
    }
    __syncthreads();
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      const int ky = tap / 3, kx = tap - ky * 3;
      const __nv_bfloat16* hrow = halo + ((warp + ky) * HALO_W + kx) * KP;
      uint32_t af[4];
      af[0] = ld32(hrow + g * KP + 2 * t);
      af[1] = ld32(hrow + (g + 8) * KP + 2 * t);
      af[2] = ld32(hrow + g * KP + 2 * t + 8);
      af[3] = ld32(hrow + (g + 8) * KP + 2 * t + 8);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const __nv_bfloat16* wrow = wsm + ((nt * 8 + g) * 9 + tap) * KP;
        mma_bf16(acc[nt], af, ld32(wrow + 2 * t), ld32(wrow + 2 * t + 8));
      }
    }
  }
  // epilogue: bias, ReLU, bf16 store (optionally accumulating)
  const int oy = y0 + warp;
  if (oy >= a.H) return;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
    for (int hlf = 0; hlf < 2; ++hlf) {
      const int ox = x0 + g + hlf * 8;
      if (ox >= a.W) continue;
      __nv_bfloat16* dst = a.y + (((size_t)n * a.H + oy) * a.W + ox) * a.ldy;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int co = co0 + nt * 8 + 2 * t + e;
        if (co >= a.Cout) continue;
        float v = acc[nt][hlf * 2 + e];
        if (a.bias) v += a.bias[co];
        if (a.relu) v = fmaxf(v, 0.f);
        if (a.accumulate) v += __bfloat162float(dst[co]);
        dst[co] = __float2bfloat16(v);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// conv3x3 of a one-channel input (the network's first layer), 8 NT output
// channels per CTA.  The same mma.sync products in the same order as
// conv3x3_kernel, of whose 16 input channels 15 are zero padding; here the
// weights stay in registers, the fragments of the padding are the constant
// zero, and only the input's own halo is staged.  32 x 128 x 128 pixels, 24
// channels: 97 -> 21 us (25 MB to write).
// ---------------------------------------------------------------------------
constexpr int C1_H = 64;  // rows per CTA; a warp takes every eighth
template <int NT>
__global__ void __launch_bounds__(256) conv3x3_c1_kernel(ConvArgs a) {
  __shared__ unsigned short halo[(C1_H + 2) * HALO_W];
  const int tile = blockIdx.x;
  const int tx = tile % a.tiles_x;
  const int ty = (tile / a.tiles_x) % a.tiles_y;
  const int n = tile / (a.tiles_x * a.tiles_y);
  const int x0 = tx * TW, y0 = ty * C1_H;
  const int co0 = blockIdx.y * NT * 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const unsigned short* x = reinterpret_cast<const unsigned short*>(a.x);
  const unsigned short* w = reinterpret_cast<const unsigned short*>(a.w);
  uint32_t bf[9][NT];  // k = 0 sits in the low half of lane t = 0
#pragma unroll
  for (int tap = 0; tap < 9; ++tap)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int co = co0 + nt * 8 + g;
      bf[tap][nt] = (t == 0 && co < a.Cout) ? w[(size_t)co * 9 + tap] : 0u;
    }
  for (int q = threadIdx.x; q < (C1_H + 2) * HALO_W; q += blockDim.x) {
    const int hy = q / HALO_W, hx = q - hy * HALO_W;
    const int iy = y0 + hy - 1, ix = x0 + hx - 1;
    halo[q] = (iy >= 0 && iy < a.H && ix >= 0 && ix < a.W) ? x[(((size_t)n * a.H + iy) * a.W + ix) * a.ldx] : 0;
  }
  float bias[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int co = co0 + nt * 8 + 2 * t + e;
      bias[nt][e] = a.bias && co < a.Cout ? a.bias[co] : 0.f;
    }
  const bool pair = a.ldy % 2 == 0 && (reinterpret_cast<uintptr_t>(a.y) & 3) == 0;
  __syncthreads();
  for (int r = warp; r < C1_H && y0 + r < a.H; r += 8) {
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      const int ky = tap / 3, kx = tap - ky * 3;
      const unsigned short* h = halo + (r + ky) * HALO_W + kx + g;
      const uint32_t af[4] = {t == 0 ? (uint32_t)h[0] : 0u, t == 0 ? (uint32_t)h[8] : 0u, 0u, 0u};
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[nt], af, bf[tap][nt], 0u);
    }
#pragma unroll
    for (int hlf = 0; hlf < 2; ++hlf) {
      const int ox = x0 + g + hlf * 8;
      if (ox >= a.W) continue;
      __nv_bfloat16* dst = a.y + (((size_t)n * a.H + y0 + r) * a.W + ox) * a.ldy;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int co = co0 + nt * 8 + 2 * t;
        __nv_bfloat16 o[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float v = acc[nt][hlf * 2 + e];
          if (a.bias) v += bias[nt][e];
          if (a.relu) v = fmaxf(v, 0.f);
          if (a.accumulate && co + e < a.Cout) v += __bfloat162float(dst[co + e]);
          o[e] = __float2bfloat16(v);
        }
        if (pair && co + 1 < a.Cout) {
          *reinterpret_cast<uint32_t*>(dst + co) = pack2(o[0], o[1]);
        } else {
          if (co < a.Cout) dst[co] = o[0];
          if (co + 1 < a.Cout) dst[co + 1] = o[1];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// conv3x3 weight gradient: dW[co][tap][ci] = sum_p dY[p][co] X[p + s(tap)][ci]
// A = dY^T (co x pixels), B = shifted X (pixels x ci); one k16 step is one
// tile row of 16 pixels.  A CTA owns 64 output x 16 input channels for all 9
// taps (warp w: co block w%4, ci block w/4) and loops over the pixel tiles
// of its split; each split writes its own partial (deterministic sum later).
// ---------------------------------------------------------------------------
struct WgradArgs {
  const __nv_bfloat16* x;
  int ldx;
  const __nv_bfloat16* dy;
  int lddy;
  int N, H, W, Cin, Cout;
  int tiles_x, tiles_y, ntiles, nsplit;
  float* partial;  // [nsplit][Cout][9][Cin]
};

__global__ void __launch_bounds__(256) conv3x3_wgrad_kernel(WgradArgs a) {
  __shared__ __align__(16) __nv_bfloat16 xt[KC * HALO_H * HALO_W];  // [ci][pixel]
  __shared__ __align__(16) __nv_bfloat16 dyt[64 * TH * TW];         // [co][pixel]
  const int split = blockIdx.x;
  const int co0 = blockIdx.y * 64, ci0 = blockIdx.z * KC;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int mb = warp & 3, nb = warp >> 2;  // 16 co x 8 ci block of this warp
  float acc[9][4];
#pragma unroll
  for (int i = 0; i < 9; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  for (int tile = split; tile < a.ntiles; tile += a.nsplit) {
    const int tx = tile % a.tiles_x;
    const int ty = (tile / a.tiles_x) % a.tiles_y;
    const int n = tile / (a.tiles_x * a.tiles_y);
    const int x0 = tx * TW, y0 = ty * TH;
    __syncthreads();
    for (int q = threadIdx.x; q < KC * HALO_H * HALO_W; q += blockDim.x) {
      const int pix = q / KC, c = q - pix * KC;
      const int hy = pix / HALO_W, hx = pix - hy * HALO_W;
      const int iy = y0 + hy - 1, ix = x0 + hx - 1;
      __nv_bfloat16 v = zero;
      if (iy >= 0 && iy < a.H && ix >= 0 && ix < a.W && ci0 + c < a.Cin)
        v = a.x[(((size_t)n * a.H + iy) * a.W + ix) * a.ldx + ci0 + c];
      xt[c * (HALO_H * HALO_W) + pix] = v;
    }
    for (int q = threadIdx.x; q < 64 * TH * TW; q += blockDim.x) {
      const int pix = q / 64, c = q - pix * 64;
      const int py = pix / TW, px = pix - py * TW;
      const int iy = y0 + py, ix = x0 + px;
      __nv_bfloat16 v = zero;
      if (iy < a.H && ix < a.W && co0 + c < a.Cout)
        v = a.dy[(((size_t)n * a.H + iy) * a.W + ix) * a.lddy + co0 + c];
      dyt[c * (TH * TW) + pix] = v;
    }
    __syncthreads();
    for (int r = 0; r < TH; ++r) {
      // A fragment: rows co (mb*16 + g, +8), k = pixel x of tile row r
      const __nv_bfloat16* arow = dyt + r * TW;
      uint32_t af[4];
      af[0] = ld32(arow + (mb * 16 + g) * (TH * TW) + 2 * t);
      af[1] = ld32(arow + (mb * 16 + g + 8) * (TH * TW) + 2 * t);
      af[2] = ld32(arow + (mb * 16 + g) * (TH * TW) + 2 * t + 8);
      af[3] = ld32(arow + (mb * 16 + g + 8) * (TH * TW) + 2 * t + 8);
      const __nv_bfloat16* bcol = xt + (nb * 8 + g) * (HALO_H * HALO_W);
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        const int ky = tap / 3, kx = tap - ky * 3;
        const __nv_bfloat16* b = bcol + (r + ky) * HALO_W + kx;
        const uint32_t b0 = pack2(b[2 * t], b[2 * t + 1]);
        const uint32_t b1 = pack2(b[2 * t + 8], b[2 * t + 9]);
        mma_bf16(acc[tap], af, b0, b1);
      }
    }
  }
  float* out = a.partial + (size_t)split * a.Cout * 9 * a.Cin;
#pragma unroll
  for (int tap = 0; tap < 9; ++tap) {
#pragma unroll
    for (int hlf = 0; hlf < 2; ++hlf) {
      const int co = co0 + mb * 16 + g + hlf * 8;
      if (co >= a.Cout) continue;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int ci = ci0 + nb * 8 + 2 * t + e;
        if (ci < a.Cin) out[((size_t)co * 9 + tap) * a.Cin + ci] = acc[tap][hlf * 2 + e];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Weight gradient where one side has one channel (the network's first layer
// and its head): the products of conv3x3_wgrad_kernel in its order (per split the
// tiles in turn, per tile its eight 16-pixel rows), without its staging of 64 x
// 16 channels of which one side is padding.  A CTA owns 32 channels of the wide
// side, one warp each tap; the wide side's tile lies in shared memory as it
// lies in global memory and its fragments come transposed by ldmatrix, the
// thin side's are a few of its pixels; the next tile's loads are in flight
// meanwhile.  THIN_X: x is the thin side (its halo is staged) and dY the A
// operand; otherwise dY is thin and x (its halo) the B operand.  32 x 128 x 128
// pixels, 24 channels: 246 and 462 us with the padding, 25 and 36 without.
// ---------------------------------------------------------------------------
constexpr int THIN_CH = 32, THIN_ROW = THIN_CH + 8, THIN_THREADS = 9 * 32;
template <bool THIN_X>
__global__ void __launch_bounds__(THIN_THREADS) wgrad_thin_kernel(WgradArgs a) {
  constexpr int WPX = THIN_X ? TH * TW : HALO_H * HALO_W;  // staged pixels of the wide side
  constexpr int TPX = THIN_X ? HALO_H * HALO_W : TH * TW;  // and of the thin side
  constexpr int NV = (WPX * (THIN_CH / 8) + THIN_THREADS - 1) / THIN_THREADS;
  __shared__ __align__(16) __nv_bfloat16 ws[2][WPX * THIN_ROW];
  __shared__ __align__(4) unsigned short ts[2][TPX + 1];
  const int split = blockIdx.x, c0 = blockIdx.y * THIN_CH, C = THIN_X ? a.Cout : a.Cin;
  const __nv_bfloat16* wide = THIN_X ? a.dy : a.x;
  const unsigned short* thin = reinterpret_cast<const unsigned short*>(THIN_X ? a.x : a.dy);
  const int ldw = THIN_X ? a.lddy : a.ldx, ldt = THIN_X ? a.ldx : a.lddy;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tap = warp, ky = tap / 3, kx = tap - ky * 3;
  uint4 v[NV];
  unsigned short tv = 0;
  auto fetch = [&](int tile) {  // a tile's pixels into registers (zeros outside the image)
    const int tx = tile % a.tiles_x, ty = (tile / a.tiles_x) % a.tiles_y, n = tile / (a.tiles_x * a.tiles_y);
    const int x0 = tx * TW, y0 = ty * TH;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const int i = threadIdx.x + q * THIN_THREADS, px = i / (THIN_CH / 8), ch = c0 + (i % (THIN_CH / 8)) * 8;
      const int iy = THIN_X ? y0 + px / TW : y0 + px / HALO_W - 1, ix = THIN_X ? x0 + px % TW : x0 + px % HALO_W - 1;
      v[q] = make_uint4(0, 0, 0, 0);
      if (px < WPX && ch < C && iy >= 0 && iy < a.H && ix >= 0 && ix < a.W)
        v[q] = ld8(wide + (((size_t)n * a.H + iy) * a.W + ix) * ldw + ch);
    }
    if (threadIdx.x < TPX) {
      const int px = threadIdx.x;
      const int iy = THIN_X ? y0 + px / HALO_W - 1 : y0 + px / TW, ix = THIN_X ? x0 + px % HALO_W - 1 : x0 + px % TW;
      tv = (iy >= 0 && iy < a.H && ix >= 0 && ix < a.W) ? thin[(((size_t)n * a.H + iy) * a.W + ix) * ldt] : 0;
    }
  };
  auto stage = [&](int b) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const int i = threadIdx.x + q * THIN_THREADS, px = i / (THIN_CH / 8);
      if (px < WPX) st8(ws[b] + px * THIN_ROW + (i % (THIN_CH / 8)) * 8, v[q]);
    }
    if (threadIdx.x < TPX) ts[b][threadIdx.x] = tv;
  };
  // fragments of 16 output channels (THIN_X) or 8 input channels
  constexpr int NF = THIN_X ? THIN_CH / 16 : THIN_CH / 8;
  float acc[NF][4];
#pragma unroll
  for (int f = 0; f < NF; ++f) acc[f][0] = acc[f][1] = acc[f][2] = acc[f][3] = 0.f;
  if (split < a.ntiles) fetch(split);
  int b = 0;
  for (int tile = split; tile < a.ntiles; tile += a.nsplit, b ^= 1) {
    stage(b);
    __syncthreads();
    if (tile + a.nsplit < a.ntiles) fetch(tile + a.nsplit);
#pragma unroll
    for (int r = 0; r < TH; ++r) {
      // the thin side's 16 pixels: lanes of its one channel hold two pairs
      const unsigned short* h = THIN_X ? &ts[b][(r + ky) * HALO_W + kx + 2 * t] : &ts[b][r * TW + 2 * t];
      const uint32_t t0 = g == 0 ? (uint32_t)h[0] | ((uint32_t)h[1] << 16) : 0u;
      const uint32_t t1 = g == 0 ? (uint32_t)h[8] | ((uint32_t)h[9] << 16) : 0u;
      const __nv_bfloat16* row = ws[b] + (THIN_X ? r * TW : (r + ky) * HALO_W + kx) * THIN_ROW;
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        if constexpr (THIN_X) {  // A = dY^T: (channels 0-7 | 8-15) x (pixels 0-7 | 8-15)
          uint32_t af[4];
          const __nv_bfloat16* src = row + ((lane & 7) + (lane & 16 ? 8 : 0)) * THIN_ROW + 16 * f + (lane & 8 ? 8 : 0);
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                       : "=r"(af[0]), "=r"(af[1]), "=r"(af[2]), "=r"(af[3])
                       : "r"((uint32_t)__cvta_generic_to_shared(src))
                       : "memory");
          mma_bf16(acc[f], af, t0, t1);
        } else {  // B = x: pixels (0-7 | 8-15) x 8 channels
          uint32_t b0, b1;
          const __nv_bfloat16* src = row + (lane & 15) * THIN_ROW + 8 * f;
          asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];"
                       : "=r"(b0), "=r"(b1)
                       : "r"((uint32_t)__cvta_generic_to_shared(src))
                       : "memory");
          const uint32_t af[4] = {t0, 0u, t1, 0u};
          mma_bf16(acc[f], af, b0, b1);
        }
      }
    }
  }
  // partial[split][co][tap][ci], one of co and ci zero
  float* out = a.partial + (size_t)split * 9 * C;
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    if constexpr (THIN_X) {  // column 0: rows g and g + 8
      const int c = c0 + 16 * f + g;
      if (t == 0 && c < C) out[(size_t)c * 9 + tap] = acc[f][0];
      if (t == 0 && c + 8 < C) out[(size_t)(c + 8) * 9 + tap] = acc[f][2];
    } else {  // row 0: columns 2 t and 2 t + 1
      const int c = c0 + 8 * f + 2 * t;
      if (g == 0 && c < C) out[(size_t)tap * C + c] = acc[f][0];
      if (g == 0 && c + 1 < C) out[(size_t)tap * C + c + 1] = acc[f][1];
    }
  }
}

// Sum the split partials in their order: dw (+)= sum_s partial[s], the loads of
// 32 splits in flight before their additions (148 splits of 5184 values: 18
// us with a load per addition, 7 with 32).
__global__ void __launch_bounds__(128) sum_partials_kernel(const float* partial, int nsplit, size_t count, float* dw,
                                                           int accumulate) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float* p = partial + i;
  float s = 0.f;
  int k = 0;
  for (; k + 32 <= nsplit; k += 32, p += 32 * count) {
    float v[32];
#pragma unroll
    for (int q = 0; q < 32; ++q) v[q] = p[(size_t)q * count];
#pragma unroll
    for (int q = 0; q < 32; ++q) s += v[q];
  }
#pragma unroll 8
  for (; k < nsplit; ++k, p += count) s += *p;
  dw[i] = accumulate ? dw[i] + s : s;
}

// Bias gradient db[c] (+)= sum over pixels of dy[p][c], with MASK after dy *=
// (y > 0) in place.  The order of the sum is fixed: 256 chains, chain t over the
// pixels t, t + 256, ... one after another, then a tree over the chains.  A
// cluster of 16 CTAs sums one group of 8 channels (one channel where 16-byte
// access does not apply): each CTA owns 16 chains, all its threads bring
// their pixels into shared memory (eight 16-byte loads in flight each, the
// next ones while this batch is added), one thread per chain and channel
// adds, and rank 0 gathers the chains over distributed shared memory.  Nothing
// may reach into rank 0's shared memory before its CTA has started: the cluster
// barrier that says so is arrived at on entry and waited for before the stores,
// behind the whole sum.
// 24 channels of 32 x 128 x 128 pixels took 400 to 930 us with one CTA per
// channel and 2-byte loads a row apart, 43 us with this and the mask.
constexpr int BG_CTAS = 16, BG_THREADS = 512, BG_U = 8, BG_CHAINS = 256 / BG_CTAS;
constexpr int BG_STEPS = BG_U * BG_THREADS / BG_CHAINS;  // additions per chain and batch: 256
template <int E>
constexpr int bg_smem() { return BG_STEPS * BG_CHAINS * E * 2; }
template <bool VEC, bool MASK>
__global__ void __launch_bounds__(BG_THREADS) bias_grad_kernel(const __nv_bfloat16* y, int ldy, __nv_bfloat16* dy,
                                                               int lddy, size_t npix, float* db, int accumulate) {
  constexpr int E = VEC ? 8 : 1;
  typedef typename std::conditional<VEC, uint4, unsigned short>::type V;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char bg_dyn[];  // [step][chain][E] bf16
  __shared__ float red[256 * E];
  V* buf = reinterpret_cast<V*>(bg_dyn);
  const unsigned short* buf1 = reinterpret_cast<const unsigned short*>(bg_dyn);
  const int c0 = (int)(blockIdx.x / BG_CTAS) * E, rank = blockIdx.x % BG_CTAS;
  // loader: pixel (step, chain); adder: chain tid / E, channel tid % E
  const int lt = threadIdx.x % BG_CHAINS, lk = threadIdx.x / BG_CHAINS;
  const size_t steps = (npix + 255) / 256;
  V v[BG_U], a[BG_U];
  memset(a, 0, sizeof(a));
  cluster.barrier_arrive();  // this CTA runs
  auto pixel = [&](size_t k0, int u) { return (k0 + u * (BG_THREADS / BG_CHAINS) + lk) * 256 + rank * BG_CHAINS + lt; };
  auto load = [&](size_t k0) {
#pragma unroll
    for (int u = 0; u < BG_U; ++u) {
      const size_t p = pixel(k0, u);
      memset(&v[u], 0, sizeof(V));
      if (p < npix) {
        v[u] = *reinterpret_cast<const V*>(dy + p * lddy + c0);
        if (MASK) a[u] = *reinterpret_cast<const V*>(y + p * ldy + c0);
      }
    }
  };
  auto store = [&](size_t k0) {
#pragma unroll
    for (int u = 0; u < BG_U; ++u) {
      if (MASK) {
        if constexpr (VEC) {
          v[u] = mask8(a[u], v[u]);
        } else {
          v[u] = __bfloat162float(__ushort_as_bfloat16(a[u])) > 0.f ? v[u] : (unsigned short)0;
        }
        const size_t p = pixel(k0, u);
        if (p < npix) *reinterpret_cast<V*>(dy + p * lddy + c0) = v[u];
      }
      buf[(u * (BG_THREADS / BG_CHAINS) + lk) * BG_CHAINS + lt] = v[u];
    }
  };
  float s = 0.f;
  load(0);
  for (size_t k0 = 0; k0 < steps; k0 += BG_STEPS) {
    store(k0);
    __syncthreads();
    if (k0 + BG_STEPS < steps) load(k0 + BG_STEPS);
    if (threadIdx.x < BG_CHAINS * E) {
#pragma unroll 32
      for (int k = 0; k < BG_STEPS; ++k)
        s += __uint_as_float((uint32_t)buf1[k * BG_CHAINS * E + threadIdx.x] << 16);
    }
    __syncthreads();
  }
  cluster.barrier_wait();  // and so do all others of the cluster
  if (threadIdx.x < BG_CHAINS * E)
    cluster.map_shared_rank(red, 0)[rank * BG_CHAINS * E + threadIdx.x] = s;
  cluster.sync();
  if (rank != 0) return;
  for (int w = 128; w > 0; w >>= 1) {
    for (int i = threadIdx.x; i < w * E; i += BG_THREADS) red[i] += red[i + w * E];
    __syncthreads();
  }
  if (threadIdx.x < E) db[c0 + threadIdx.x] = accumulate ? db[c0 + threadIdx.x] + red[threadIdx.x] : red[threadIdx.x];
}

// The same sum, in the same order, by one CTA per channel: where the device
// has no room for a cluster of 16 (a partition of a few SMs, say).
__global__ void __launch_bounds__(256) bias_grad_block_kernel(const __nv_bfloat16* dy, int ld, size_t npix, float* db,
                                                              int accumulate) {
  __shared__ float red[256];
  const int c = blockIdx.x;
  float s = 0.f;
  for (size_t p = threadIdx.x; p < npix; p += 256) s += __bfloat162float(dy[p * ld + c]);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) db[c] = accumulate ? db[c] + red[0] : red[0];
}

// wt[ci][ky][kx][co] = w[co][2-ky][2-kx][ci]
__global__ void flip_weights_kernel(const __nv_bfloat16* w, __nv_bfloat16* wt, int Cout, int Cin) {
  const size_t total = (size_t)Cout * 9 * Cin;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int ci = (int)(i % Cin);
    const int tap = (int)((i / Cin) % 9);
    const int co = (int)(i / ((size_t)Cin * 9));
    wt[((size_t)ci * 9 + (8 - tap)) * Cout + co] = w[i];
  }
}

// dy *= (y > 0) over an N*H*W x C slice
__global__ void relu_mask_kernel(const __nv_bfloat16* y, int ldy, __nv_bfloat16* dy, int lddy, size_t npix, int C) {
  const size_t total = npix * C;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t p = i / C;
    const int c = (int)(i - p * C);
    if (!(__bfloat162float(y[p * ldy + c]) > 0.f)) dy[p * lddy + c] = __float2bfloat16(0.f);
  }
}

// The 16-byte forms: chunk i of 8 channels of pixel p, with 32-bit indices
// (the launch takes them where N H W C fits).  One thread reads or writes a
// whole 2 x 2 block, in the scalar kernels' order of additions.
struct Pool8 {
  unsigned total, nch, Wh, Hh;  // chunks in all, chunks per pixel, coarse width and height
};
__device__ __forceinline__ void pool_index(const Pool8& q, unsigned i, unsigned& c, size_t& coarse, size_t& fine) {
  const unsigned p = i / q.nch;
  c = (i - p * q.nch) * 8;
  const unsigned r = p / q.Wh, x = p - r * q.Wh, n = r / q.Hh, y = r - n * q.Hh;
  coarse = p;
  fine = ((size_t)n * 2 * q.Hh + 2 * y) * 2 * q.Wh + 2 * x;
}
__global__ void relu_mask8_kernel(const __nv_bfloat16* y, int ldy, __nv_bfloat16* dy, int lddy, unsigned total,
                                  unsigned nch) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned p = i / nch, c = (i - p * nch) * 8;
    __nv_bfloat16* d = dy + (size_t)p * lddy + c;
    st8(d, mask8(ld8(y + (size_t)p * ldy + c), ld8(d)));
  }
}
__global__ void avgpool2x8_kernel(const __nv_bfloat16* x, int ldx, __nv_bfloat16* y, int ldy, Pool8 q) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < q.total; i += gridDim.x * blockDim.x) {
    unsigned c;
    size_t o, b;
    pool_index(q, i, c, o, b);
    const size_t W = 2 * q.Wh;
    const uint4 v[4] = {ld8(x + b * ldx + c), ld8(x + (b + 1) * ldx + c), ld8(x + (b + W) * ldx + c),
                        ld8(x + (b + W + 1) * ldx + c)};
    float f[4][8], r[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) unpack8(v[k], f[k]);
#pragma unroll
    for (int e = 0; e < 8; ++e) r[e] = 0.25f * (f[0][e] + f[1][e] + f[2][e] + f[3][e]);
    st8(y + o * ldy + c, pack8(r));
  }
}
__global__ void avgpool2x8_bwd_kernel(const __nv_bfloat16* dy, int lddy, __nv_bfloat16* dx, int lddx, Pool8 q,
                                      int accumulate) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < q.total; i += gridDim.x * blockDim.x) {
    unsigned c;
    size_t o, b;
    pool_index(q, i, c, o, b);
    const size_t W = 2 * q.Wh, px[4] = {b, b + 1, b + W, b + W + 1};
    const uint4 g = ld8(dy + o * lddy + c);
    uint4 old[4];
    if (accumulate) {
#pragma unroll
      for (int k = 0; k < 4; ++k) old[k] = ld8(dx + px[k] * lddx + c);
    }
    float f[8];
    unpack8(g, f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float r[8], a[8];
      if (accumulate) unpack8(old[k], a);
#pragma unroll
      for (int e = 0; e < 8; ++e) r[e] = accumulate ? 0.25f * f[e] + a[e] : 0.25f * f[e];
      st8(dx + px[k] * lddx + c, pack8(r));
    }
  }
}
__global__ void upsample2x8_kernel(const __nv_bfloat16* x, int ldx, __nv_bfloat16* y, int ldy, Pool8 q) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < q.total; i += gridDim.x * blockDim.x) {
    unsigned c;
    size_t o, b;
    pool_index(q, i, c, o, b);
    const size_t W = 2 * q.Wh;
    const uint4 v = ld8(x + o * ldx + c);
    st8(y + b * ldy + c, v);
    st8(y + (b + 1) * ldy + c, v);
    st8(y + (b + W) * ldy + c, v);
    st8(y + (b + W + 1) * ldy + c, v);
  }
}
__global__ void upsample2x8_bwd_kernel(const __nv_bfloat16* dy, int lddy, __nv_bfloat16* dx, int lddx, Pool8 q,
                                       int accumulate) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < q.total; i += gridDim.x * blockDim.x) {
    unsigned c;
    size_t o, b;
    pool_index(q, i, c, o, b);
    const size_t W = 2 * q.Wh;
    const uint4 v[4] = {ld8(dy + b * lddy + c), ld8(dy + (b + 1) * lddy + c), ld8(dy + (b + W) * lddy + c),
                        ld8(dy + (b + W + 1) * lddy + c)};
    float f[4][8], r[8], a[8];
    if (accumulate) unpack8(ld8(dx + o * lddx + c), a);
#pragma unroll
    for (int k = 0; k < 4; ++k) unpack8(v[k], f[k]);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      r[e] = f[0][e] + f[1][e] + f[2][e] + f[3][e];
      if (accumulate) r[e] += a[e];
    }
    st8(dx + o * lddx + c, pack8(r));
  }
}

__global__ void avgpool2_kernel(const __nv_bfloat16* x, int ldx, __nv_bfloat16* y, int ldy, int N, int H, int W,
                                int C) {
  const int Ho = H / 2, Wo = W / 2;
  const size_t total = (size_t)N * Ho * Wo * C;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    size_t p = i / C;
    const int ox = (int)(p % Wo);
    p /= Wo;
    const int oy = (int)(p % Ho);
    const int n = (int)(p / Ho);
    const size_t b = ((size_t)n * H + 2 * oy) * W + 2 * ox;
    const float s = __bfloat162float(x[b * ldx + c]) + __bfloat162float(x[(b + 1) * ldx + c]) +
                    __bfloat162float(x[(b + W) * ldx + c]) + __bfloat162float(x[(b + W + 1) * ldx + c]);
    y[(((size_t)n * Ho + oy) * Wo + ox) * ldy + c] = __float2bfloat16(0.25f * s);
  }
}

__global__ void avgpool2_bwd_kernel(const __nv_bfloat16* dy, int lddy, __nv_bfloat16* dx, int lddx, int N, int H,
                                    int W, int C, int accumulate) {
  const size_t total = (size_t)N * H * W * C;
  const int Wo = W / 2, Ho = H / 2;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    size_t p = i / C;
    const int ix = (int)(p % W);
    p /= W;
    const int iy = (int)(p % H);
    const int n = (int)(p / H);
    float v = 0.25f * __bfloat162float(dy[(((size_t)n * Ho + iy / 2) * Wo + ix / 2) * lddy + c]);
    __nv_bfloat16* d = dx + (((size_t)n * H + iy) * W + ix) * lddx + c;
    if (accumulate) v += __bfloat162float(*d);
    *d = __float2bfloat16(v);
  }
}

// nearest-neighbour 2x upsampling and its gradient (sum of the 4 children)
__global__ void upsample2_kernel(const __nv_bfloat16* x, int ldx, __nv_bfloat16* y, int ldy, int N, int H, int W,
                                 int C) {
  const int Ho = 2 * H, Wo = 2 * W;
  const size_t total = (size_t)N * Ho * Wo * C;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    size_t p = i / C;
    const int ox = (int)(p % Wo);
    p /= Wo;
    const int oy = (int)(p % Ho);
    const int n = (int)(p / Ho);
    y[(((size_t)n * Ho + oy) * Wo + ox) * ldy + c] = x[(((size_t)n * H + oy / 2) * W + ox / 2) * ldx + c];
  }
}

__global__ void upsample2_bwd_kernel(const __nv_bfloat16* dy, int lddy, __nv_bfloat16* dx, int lddx, int N, int H,
                                     int W, int C, int accumulate) {
  const size_t total = (size_t)N * H * W * C;
  const int Wo = 2 * W;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    size_t p = i / C;
    const int ix = (int)(p % W);
    p /= W;
    const int iy = (int)(p % H);
    const int n = (int)(p / H);
    const size_t b = ((size_t)n * 2 * H + 2 * iy) * Wo + 2 * ix;
    float v = __bfloat162float(dy[b * lddy + c]) + __bfloat162float(dy[(b + 1) * lddy + c]) +
              __bfloat162float(dy[(b + Wo) * lddy + c]) + __bfloat162float(dy[(b + Wo + 1) * lddy + c]);
    __nv_bfloat16* d = dx + (((size_t)n * H + iy) * W + ix) * lddx + c;
    if (accumulate) v += __bfloat162float(*d);
    *d = __float2bfloat16(v);
  }
}

// mean squared error of a 1-channel output against an FP32 target:
// loss_part[block] = sum (y - t)^2 over the block's pixels; dy = 2 (y - t) / n
__global__ void mse_kernel(const __nv_bfloat16* y, int ldy, const float* target, size_t n, __nv_bfloat16* dy,
                           int lddy, float* loss_part) {
  __shared__ float red[256];
  float s = 0.f;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float r = __bfloat162float(y[i * ldy]) - target[i];
    s += r * r;
    dy[i * lddy] = __float2bfloat16(2.f * r / (float)n);
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) loss_part[blockIdx.x] = red[0];
}

// Adam with decoupled weight decay on FP32 master weights; writes the bf16 copy
__global__ void adam_kernel(float* w, __nv_bfloat16* w16, const float* g, float* m, float* v, size_t n, float lr,
                            float b1, float b2, float eps, float wd, float bc1, float bc2) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float upd = (mi / bc1) / (sqrtf(vi / bc2) + eps);
    const float wi = w[i] * (1.f - lr * wd) - lr * upd;
    w[i] = wi;
    if (w16) w16[i] = __float2bfloat16(wi);
  }
}

__global__ void f32_to_bf16_kernel(const float* x, __nv_bfloat16* y, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16(x[i]);
}

// 0: tensor-core (tcgen05) path where it applies, else mma.sync; 1: always
// mma.sync, and bias gradients without clusters; 2: tcgen05 with one 128-pixel tile per group (for comparisons)
int g_conv_path = 0;

int grid_for(size_t n, int block = 256) {
  size_t g = (n + block - 1) / block;
  if (g > 148 * 32) g = 148 * 32;
  return (int)(g < 1 ? 1 : g);
}

// whether two tensors' channels can be taken eight at a time
bool vec8(const void* a, int lda, const void* b, int ldb, int C) {
  return C % 8 == 0 && lda % 8 == 0 && ldb % 8 == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(b) & 15) == 0;
}

// the 2 x 2 blocks of an N x 2 Hh x 2 Wh image with C channels; false when
// the 32-bit indices of the 16-byte kernels do not reach
bool pool8(Pool8& q, int N, int Hh, int Wh, int C) {
  const size_t total = (size_t)N * Hh * Wh * (C / 8);
  q.total = (unsigned)total;
  q.nch = C / 8;
  q.Wh = Wh;
  q.Hh = Hh;
  return total <= 0x7fffffffull;
}

int check_launch() {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : SMILI_UNET_ERR_CUDA;
}

// Whether the current device can hold a cluster of this launch: 16 CTAs are
// beyond the portable 8.  Asked once per device.
bool cluster_fits(const void* fn, const cudaLaunchConfig_t& cfg) {
  constexpr int kDevs = 64;
  static std::atomic<int> known[kDevs];  // 0: not asked, 1: no, 2: yes
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevs) return false;
  int k = known[dev].load();
  if (k == 0) {
    k = cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0 ? 2 : 1;
    if (k == 1) cudaGetLastError();
    known[dev].store(k);
  }
  return k == 2;
}

// bias gradient, after masking dy by y > 0 where y is given
int launch_bias_grad(const void* y, int ldy, void* dy, int lddy, long long npix, int C, float* db, int accumulate,
                     void* stream) {
  const bool vec = vec8(dy, lddy, y ? y : dy, y ? ldy : lddy, C);
  const void* fn = vec ? (y ? (const void*)bias_grad_kernel<true, true> : (const void*)bias_grad_kernel<true, false>)
                       : (y ? (const void*)bias_grad_kernel<false, true> : (const void*)bias_grad_kernel<false, false>);
  // 16 CTAs of a cluster, beyond the portable 8, and 64 KB of shared memory:
  // both opted into, per device
  const int smem = vec ? bg_smem<8>() : bg_smem<1>();
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = BG_CTAS;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)BG_CTAS * (vec ? C / 8 : C));
  cfg.blockDim = dim3(BG_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const __nv_bfloat16* yp = static_cast<const __nv_bfloat16*>(y);
  __nv_bfloat16* dp = static_cast<__nv_bfloat16*>(dy);
  size_t n = (size_t)npix;
  if (g_conv_path != 1) {
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return SMILI_UNET_ERR_CUDA;
    if (cluster_fits(fn, cfg)) {
      void* args[] = {&yp, &ldy, &dp, &lddy, &n, &db, &accumulate};
      if (cudaLaunchKernelExC(&cfg, fn, args) != cudaSuccess) return SMILI_UNET_ERR_CUDA;
      return check_launch();
    }
  }
  if (y) {
    const int rc = smili_unet_relu_mask(y, ldy, dy, lddy, npix, C, stream);
    if (rc != 0) return rc;
  }
  bias_grad_block_kernel<<<C, 256, 0, cfg.stream>>>(dp, lddy, n, db, accumulate);
  return check_launch();
}

}  // namespace

extern "C" {

int smili_unet_conv3x3(const void* x, int N, int H, int W, int Cin, int ldx, const void* w, const float* bias,
                       void* y, int ldy, int Cout, int relu, int accumulate, void* stream) {
  if (!x || !w || !y || N < 1 || H < 1 || W < 1 || Cin < 1 || Cout < 1 || ldx < Cin || ldy < Cout)
    return SMILI_UNET_ERR_ARG;
  ConvArgs a;
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.N = N;
  a.H = H;
  a.W = W;
  a.Cin = Cin;
  a.ldx = ldx;
  a.w = static_cast<const __nv_bfloat16*>(w);
  a.bias = bias;
  a.y = static_cast<__nv_bfloat16*>(y);
  a.ldy = ldy;
  a.Cout = Cout;
  a.relu = relu;
  a.accumulate = accumulate;
  a.tiles_x = (W + TW - 1) / TW;
  a.tiles_y = (H + TH - 1) / TH;
  const long long tiles = (long long)a.tiles_x * a.tiles_y * N;
  if (tiles > 0x7fffffffLL) return SMILI_UNET_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (g_conv_path != 1 && tc::eligible(x, Cin, ldx, w, Cout))
    return tc::launch(a.x, N, H, W, Cin, ldx, a.w, bias, a.y, ldy, Cout, relu, accumulate, s,
                      g_conv_path == 2 ? 1 : tc::MAX_SUB) == 0
               ? 0
               : SMILI_UNET_ERR_CUDA;
  if (g_conv_path != 1 && Cin == 1) {
    a.tiles_y = (H + C1_H - 1) / C1_H;
    const unsigned t1 = (unsigned)((long long)a.tiles_x * a.tiles_y * N);
    if (Cout <= 8) conv3x3_c1_kernel<1><<<t1, 256, 0, s>>>(a);
    else if (Cout <= 16) conv3x3_c1_kernel<2><<<t1, 256, 0, s>>>(a);
    else if (Cout <= 24) conv3x3_c1_kernel<3><<<t1, 256, 0, s>>>(a);
    else conv3x3_c1_kernel<4><<<dim3(t1, (Cout + 31) / 32), 256, 0, s>>>(a);
    return check_launch();
  }
  if (Cout <= 8) {
    conv3x3_kernel<1><<<dim3((unsigned)tiles, 1), 256, 0, s>>>(a);
  } else if (Cout <= 16) {
    conv3x3_kernel<2><<<dim3((unsigned)tiles, 1), 256, 0, s>>>(a);
  } else if (Cout <= 32) {
    conv3x3_kernel<4><<<dim3((unsigned)tiles, 1), 256, 0, s>>>(a);
  } else {
    conv3x3_kernel<8><<<dim3((unsigned)tiles, (Cout + 63) / 64), 256, 0, s>>>(a);
  }
  return check_launch();
}

int smili_unet_conv3x3_wgrad(const void* x, int ldx, const void* dy, int lddy, int N, int H, int W, int Cin,
                             int Cout, float* partial, int nsplit, float* dw, int accumulate, void* stream) {
  if (!x || !dy || !partial || !dw || N < 1 || H < 1 || W < 1 || Cin < 1 || Cout < 1 || nsplit < 1 || ldx < Cin ||
      lddy < Cout)
    return SMILI_UNET_ERR_ARG;
  WgradArgs a;
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.ldx = ldx;
  a.dy = static_cast<const __nv_bfloat16*>(dy);
  a.lddy = lddy;
  a.N = N;
  a.H = H;
  a.W = W;
  a.Cin = Cin;
  a.Cout = Cout;
  a.tiles_x = (W + TW - 1) / TW;
  a.tiles_y = (H + TH - 1) / TH;
  a.ntiles = a.tiles_x * a.tiles_y * N;
  a.nsplit = nsplit;
  a.partial = partial;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (g_conv_path != 1 && tc::wgrad_eligible(x, ldx, dy, lddy, Cin, Cout)) {
    if (tc::launch_wgrad(a.x, ldx, a.dy, lddy, N, H, W, Cin, Cout, partial, nsplit, s) != 0)
      return SMILI_UNET_ERR_CUDA;
  } else if (g_conv_path != 1 && Cin == 1 && vec8(dy, lddy, dy, lddy, Cout) && Cout <= 65535 * THIN_CH) {
    wgrad_thin_kernel<true><<<dim3(nsplit, (Cout + THIN_CH - 1) / THIN_CH), THIN_THREADS, 0, s>>>(a);
  } else if (g_conv_path != 1 && Cout == 1 && vec8(x, ldx, x, ldx, Cin) && Cin <= 65535 * THIN_CH) {
    wgrad_thin_kernel<false><<<dim3(nsplit, (Cin + THIN_CH - 1) / THIN_CH), THIN_THREADS, 0, s>>>(a);
  } else {
    conv3x3_wgrad_kernel<<<dim3(nsplit, (Cout + 63) / 64, (Cin + KC - 1) / KC), 256, 0, s>>>(a);
  }
  const size_t count = (size_t)Cout * 9 * Cin;
  sum_partials_kernel<<<(unsigned)((count + 127) / 128), 128, 0, s>>>(partial, nsplit, count, dw, accumulate);
  return check_launch();
}

int smili_unet_bias_grad(const void* dy, int ld, long long npix, int C, float* db, int accumulate, void* stream) {
  if (!dy || !db || npix < 1 || C < 1 || ld < C) return SMILI_UNET_ERR_ARG;
  return launch_bias_grad(nullptr, C, const_cast<void*>(dy), ld, npix, C, db, accumulate, stream);
}

int smili_unet_relu_bias_grad(const void* y, int ldy, void* dy, int lddy, long long npix, int C, float* db,
                              int accumulate, void* stream) {
  if (!y || !dy || !db || npix < 1 || C < 1 || ldy < C || lddy < C) return SMILI_UNET_ERR_ARG;
  return launch_bias_grad(y, ldy, dy, lddy, npix, C, db, accumulate, stream);
}

int smili_unet_flip_weights(const void* w, void* wt, int Cout, int Cin, void* stream) {
  if (!w || !wt || Cout < 1 || Cin < 1) return SMILI_UNET_ERR_ARG;
  flip_weights_kernel<<<grid_for((size_t)Cout * 9 * Cin), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(wt), Cout, Cin);
  return check_launch();
}

int smili_unet_relu_mask(const void* y, int ldy, void* dy, int lddy, long long npix, int C, void* stream) {
  if (!y || !dy || npix < 1 || C < 1 || ldy < C || lddy < C) return SMILI_UNET_ERR_ARG;
  const size_t chunks = (size_t)npix * (C / 8);
  if (vec8(y, ldy, dy, lddy, C) && chunks <= 0x7fffffffull) {
    relu_mask8_kernel<<<grid_for(chunks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(y), ldy, static_cast<__nv_bfloat16*>(dy), lddy, (unsigned)chunks, C / 8);
    return check_launch();
  }
  relu_mask_kernel<<<grid_for((size_t)npix * C), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(y), ldy, static_cast<__nv_bfloat16*>(dy), lddy, (size_t)npix, C);
  return check_launch();
}

int smili_unet_avgpool2(const void* x, int ldx, void* y, int ldy, int N, int H, int W, int C, void* stream) {
  if (!x || !y || N < 1 || H < 2 || W < 2 || (H & 1) || (W & 1) || C < 1 || ldx < C || ldy < C)
    return SMILI_UNET_ERR_ARG;
  Pool8 q;
  if (vec8(x, ldx, y, ldy, C) && pool8(q, N, H / 2, W / 2, C)) {
    avgpool2x8_kernel<<<grid_for(q.total), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(x), ldx, static_cast<__nv_bfloat16*>(y), ldy, q);
    return check_launch();
  }
  avgpool2_kernel<<<grid_for((size_t)N * H * W * C / 4), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), ldx, static_cast<__nv_bfloat16*>(y), ldy, N, H, W, C);
  return check_launch();
}

int smili_unet_avgpool2_bwd(const void* dy, int lddy, void* dx, int lddx, int N, int H, int W, int C,
                            int accumulate, void* stream) {
  if (!dy || !dx || N < 1 || H < 2 || W < 2 || (H & 1) || (W & 1) || C < 1 || lddx < C || lddy < C)
    return SMILI_UNET_ERR_ARG;
  Pool8 q;
  if (vec8(dy, lddy, dx, lddx, C) && pool8(q, N, H / 2, W / 2, C)) {
    avgpool2x8_bwd_kernel<<<grid_for(q.total), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(dy), lddy, static_cast<__nv_bfloat16*>(dx), lddx, q, accumulate);
    return check_launch();
  }
  avgpool2_bwd_kernel<<<grid_for((size_t)N * H * W * C), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(dy), lddy, static_cast<__nv_bfloat16*>(dx), lddx, N, H, W, C, accumulate);
  return check_launch();
}

int smili_unet_upsample2(const void* x, int ldx, void* y, int ldy, int N, int H, int W, int C, void* stream) {
  if (!x || !y || N < 1 || H < 1 || W < 1 || C < 1 || ldx < C || ldy < C) return SMILI_UNET_ERR_ARG;
  Pool8 q;
  if (vec8(x, ldx, y, ldy, C) && pool8(q, N, H, W, C)) {
    upsample2x8_kernel<<<grid_for(q.total), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(x), ldx, static_cast<__nv_bfloat16*>(y), ldy, q);
    return check_launch();
  }
  upsample2_kernel<<<grid_for((size_t)N * H * W * C * 4), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), ldx, static_cast<__nv_bfloat16*>(y), ldy, N, H, W, C);
  return check_launch();
}

int smili_unet_upsample2_bwd(const void* dy, int lddy, void* dx, int lddx, int N, int H, int W, int C,
                             int accumulate, void* stream) {
  if (!dy || !dx || N < 1 || H < 1 || W < 1 || C < 1 || lddx < C || lddy < C) return SMILI_UNET_ERR_ARG;
  Pool8 q;
  if (vec8(dy, lddy, dx, lddx, C) && pool8(q, N, H, W, C)) {
    upsample2x8_bwd_kernel<<<grid_for(q.total), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(dy), lddy, static_cast<__nv_bfloat16*>(dx), lddx, q, accumulate);
    return check_launch();
  }
  upsample2_bwd_kernel<<<grid_for((size_t)N * H * W * C), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(dy), lddy, static_cast<__nv_bfloat16*>(dx), lddx, N, H, W, C, accumulate);
  return check_launch();
}

int smili_unet_mse(const void* y, int ldy, const float* target, long long n, void* dy, int lddy, float* loss_part,
                   int nblocks, void* stream) {
  if (!y || !target || !dy || !loss_part || n < 1 || nblocks < 1 || ldy < 1 || lddy < 1) return SMILI_UNET_ERR_ARG;
  mse_kernel<<<nblocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(y), ldy,
                                                                      target, (size_t)n,
                                                                      static_cast<__nv_bfloat16*>(dy), lddy,
                                                                      loss_part);
  return check_launch();
}

int smili_unet_adam(float* w, void* w16, const float* g, float* m, float* v, long long n, float lr, float b1,
                    float b2, float eps, float wd, int step, void* stream) {
  if (!w || !g || !m || !v || n < 1 || step < 1) return SMILI_UNET_ERR_ARG;
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  adam_kernel<<<grid_for((size_t)n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      w, static_cast<__nv_bfloat16*>(w16), g, m, v, (size_t)n, lr, b1, b2, eps, wd, bc1, bc2);
  return check_launch();
}

int smili_unet_set_conv_path(int path) {
  if (path < 0 || path > 2) return SMILI_UNET_ERR_ARG;
  g_conv_path = path;
  return 0;
}

const char* smili_unet_last_error(void) { return tc::last_error().c_str(); }

int smili_unet_tc_status(void) {
  int e = 0;
  if (cudaMemcpyFromSymbol(&e, tc::g_tc_err, sizeof(int)) != cudaSuccess) return SMILI_UNET_ERR_CUDA;
  if (e) {
    const int zero = 0;
    if (cudaMemcpyToSymbol(tc::g_tc_err, &zero, sizeof(int)) != cudaSuccess) return SMILI_UNET_ERR_CUDA;
  }
  return e;
}

int smili_unet_f32_to_bf16(const float* x, void* y, long long n, void* stream) {
  if (!x || !y || n < 1) return SMILI_UNET_ERR_ARG;
  f32_to_bf16_kernel<<<grid_for((size_t)n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      x, static_cast<__nv_bfloat16*>(y), (size_t)n);
  return check_launch();
}

}  // extern "C"
