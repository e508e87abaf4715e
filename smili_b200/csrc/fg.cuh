// One function/gradient evaluation of the static-imaging objective, split into
// stages that the CTAs of a group share (a group barrier separates stages).
//
// Replaces calc_cost (src/fortlib/fftim2d.f90:387-607) =
//   calc_chisq (src/fortlib/fftlib.f90:250-382):
//     I1d_I2d_fwd + FINUFFT type 2 (wrapfinufft.f90:94-128)   -> stages F1-F3
//     calc_chisq_fcv/amp/ca/cp (fftlib.f90:384-655)           -> stage F4
//     NUFFT_adj_resid: 2 x FINUFFT type 1 (fftlib.f90:152-174) -> stages F5-F7
//       (one type-1 of c = Vresre - i Vresim: Re T1(c) = Re T1(Vresre) + Im T1(Vresim))
//   + calc_cost_reg (src/fortlib/image.f90:12-200)             -> stage F8
//
// NUFFT (exponential-of-semicircle kernel, upsampling 2) restricted to the
// "band" of fine-grid cells that the uv points touch: the type-2 row pass
// keeps only band columns and the column pass only runs on band columns; the
// type-1 passes run only on band rows.  Fine-grid coordinates xi = u n / 2pi
// are precomputed at set-up.
#pragma once
#include "common.cuh"
#include "fft.cuh"

template <typename R>
__device__ __forceinline__ R es_kernel(R z, R beta) {
  const R s = (R)1 - z * z;
  return s > (R)0 ? exp(beta * (sqrt(s) - (R)1)) : (R)0;
}

// FP32: the hardware exponential; its error (a few ulps over the kernel's
// argument range [-beta, 0]) is far below the 1e-6 tolerance of the transform
template <>
__device__ __forceinline__ float es_kernel<float>(float z, float beta) {
  const float s = 1.f - z * z;
  return s > 0.f ? __expf(beta * (sqrtf(s) - 1.f)) : 0.f;
}

__device__ __forceinline__ int imod(int a, int n) {
  if ((unsigned)a < (unsigned)n) return a;  // the common case
  int r = a % n;
  return r < 0 ? r + n : r;
}
// a in (-n, 2n): one conditional add or subtract
__device__ __forceinline__ int wrapn(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

__device__ __forceinline__ double smabs(double x) { return sqrt(x * x + 1e-10); }
__device__ __forceinline__ float smabs(float x) { return sqrtf(x * x + 1e-10f); }

// rows (sequences) per CTA pass for an FFT of length n
__device__ __forceinline__ int fft_batch(int n) {
  int s = (int)(blockDim.x * 8) / n;
  return s < 1 ? 1 : s;
}

// global atomic addition of a complex value: one vector reduction in FP32, two in FP64
__device__ __forceinline__ void acc_add(cpx<float>* p, cpx<float> v) {
  atomicAdd(reinterpret_cast<float2*>(p), make_float2(v.x, v.y));
}
__device__ __forceinline__ void acc_add(cpx<double>* p, cpx<double> v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}

// Working context of one problem inside a kernel
template <typename R>
struct FgCtx {
  const ProbDesc* P;
  char* base;
  cpx<R>* sbuf;   // shared: 2 * SMEM_CPX complex values
  cpx<R>* swork;
  int smem_cpx;   // capacity of each of the two FFT buffers (complex elements)
  int dyn_cpx;    // capacity of the whole dynamic shared region (complex elements)
};

// Running compensated sum (TwoSum) used for the chi-square terms
struct KSum {
  double s, c;
  __device__ void add(double v) {
    const double t = s + v;
    const double bp = t - s;
    c += (s - (t - bp)) + (v - bp);
    s = t;
  }
  __device__ double value() const { return s + c; }
};
struct KSumF {
  float s, c;
  __device__ void add(float v) {
    const float t = s + v;
    const float bp = t - s;
    c += (s - (t - bp)) + (v - bp);
    s = t;
  }
  __device__ double value() const { return (double)s + (double)c; }
};

// ---------------------------------------------------------------------------
// Band passes as dense products (P.dft): with the twiddle matrices
//   Ex[b][ix] = exp(+2 pi i (ix - nx/2)(b1s + b) / nf1)   [b1n][nx]
//   Ey[r][iy] = exp(+2 pi i (iy - ny/2)(b2s + r) / nf2)   [b2n][ny]
// the four FFT passes of the band-pruned NUFFT are
//   F1  tmpA[iy][b]  = sum_ix U[iy][ix] Ex[b][ix],  U = x dc1[ix] dc2[iy]
//   F2  bandA[r][b]  = sum_iy Ey[r][iy] tmpA[iy][b]
//   F6  tmpC[r][ix]  = sum_b  bandC[r][b] Ex[b][ix]
//   F7  gchi[iy][ix] = Re sum_r Ey[r][iy] tmpC[r][ix]  * dc1[ix] dc2[iy]
// (the same twiddles the radix passes apply, exp periodic in nf).  Used
// for bands of at most 64 x 64 cells, 2048 in all, where each pass is a few
// million multiply-adds.  F1 splits the image rows over the CTAs, F2 the band
// cells; F6 and F7 are one stage, a CTA taking its share of the image columns
// through both.  In FP64 the lanes of a warp share the sums of F1 and F2; in
// FP32 every sum runs along its row or column in one thread, in the order of
// the radix-free definition: a solve amplifies the last bit of an FP32
// visibility by up to 1e4, and sums in another order move its image by more
// than the spreading's atomics do.  (F1 and F2 as one stage that adds each
// CTA's part of the band with atomics is no faster, and an FP64 solve with
// near-null baselines then changes from run to run by 4e-9 instead of 1e-11.)
// As register tiles of 64 rows, 512 cells, 8 band rows and 4 image rows the
// stages had work for 4 to 16 CTAs only: 256 x 256, 44 x 21 cells, FP64 on 64
// CTAs, 70 + 40 + 24 + 14 us per evaluation, 18 + 7 + 21 on 96 now; FP32 on
// groups of 2 CTAs (148 problems) 100 + 40 + 44 + 141, now 112 + 42 + 96.  (On
// groups of 4 the FP32 rows take 106 us; with the earlier tiles back, 2 rows by 4
// cells on all 512 threads, 94, but the launch of 74 problems 73.6 ms against 73.4.)
// ---------------------------------------------------------------------------
constexpr int DFT_NB = 64;  // largest band side on this path (and 2048 cells in all)
constexpr int DFT_KC = 32;  // image columns per staged chunk of the FP32 F1

// One pixel of the dense image grid: its value into xg, its moments, and the
// deconvolved value that the transform takes.
template <typename R>
__device__ __forceinline__ R dense_pixel(const ProbDesc& P, const double* x, const int* inv, double* xg, double d1,
                                         double d2, int iy, int ix, bool need_mom, double (&mom)[10]) {
  const int cell = iy * P.nx + ix, pv = P.ident ? cell : inv[cell];
  const double val = pv >= 0 ? x[pv] : 0.0;
  if (!P.ident) xg[cell] = val;
  if (need_mom && pv >= 0) {
    const double fx = ix + 1, fy = iy + 1;  // 1-based pixel numbers as the reference
    mom[0] += val;
    mom[1] += fabs(val);
    mom[2] += val * fx;
    mom[3] += val * fy;
    mom[4] += val * fx * fx;
    mom[5] += val * fy * fy;
    mom[6] += val * fx * fy;
    if (P.has_cen) {
      const double Ip = fabs(P.cen_alpha - 1) < 1e-10 ? smabs(val) : pow(smabs(val), P.cen_alpha);
      mom[7] += Ip * (fx - P.nxref);
      mom[8] += Ip * (fy - P.nyref);
      mom[9] += Ip;
    }
  }
  return (R)(val * d1 * d2);
}

// Sum of each of v[0..N) over the warp (N a power of two up to 32): lane l
// returns the sum of value l / (32 / N).
template <int N, typename R>
__device__ __forceinline__ R warp_fold_r(R (&v)[N], int lane) {
  int b = 16;
#pragma unroll
  for (int h = N / 2; h >= 1; h >>= 1, b >>= 1) {
    const bool up = (lane & b) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const R send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, b);
    }
  }
#pragma unroll
  for (int q = 16 / N; q >= 1; q >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], q);
  return v[0];
}

// F1 in FP64.  Up to 32 image rows at a time in shared memory; a warp takes RB of
// them and two band columns, its lanes the image columns (coalesced in Ex,
// conflict free in the rows).  Also writes the dense image grid and
// accumulates the moments.
template <int RB>
__device__ __noinline__ void dft_rows(FgCtx<double>& c, const GroupCtx& g, double (&mom)[10]) {
  using R = double;
  const ProbDesc& P = *c.P;
  const double* x = at<double>(c.base, P.o_x);
  const int* inv = at<int>(c.base, P.o_inv);
  double* xg = at<double>(c.base, P.o_xg);
  const double* dc1 = at<double>(c.base, P.o_dc1);
  const double* dc2 = at<double>(c.base, P.o_dc2);
  const cpx<R>* Ex = at<cpx<R>>(c.base, P.o_ex);
  cpx<R>* tmpA = at<cpx<R>>(c.base, P.o_tmpA);  // [nb][ny]
  cpx<R>* bandC = at<cpx<R>>(c.base, P.o_bandC);
  const int nx = P.nx, ny = P.ny, nb = P.b1n, ncell = P.b1n * P.b2n;
  const int T = blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = T >> 5;
  const int share = (ny + g.G - 1) / g.G, y1 = min(ny, (g.rank + 1) * share);
  int RS = (min(share, 32) + RB - 1) / RB * RB;  // staged rows (nx <= 1024: at least 8 fit)
  while (RS > RB && (size_t)RS * nx > (size_t)c.dyn_cpx * 2) RS -= RB;
  R* Us = reinterpret_cast<R*>(c.sbuf);  // [RS][nx]
  for (int i = g.rank * T + threadIdx.x; i < ncell; i += g.G * T) bandC[i] = cmk<R>(0, 0);
  const bool need_mom = P.has_tfd || P.has_cen || P.has_sm;
  const int npair = (nb + 1) >> 1;
  for (int y0 = g.rank * share; y0 < y1; y0 += RS) {
    const int rows = min(RS, y1 - y0), nsub = (rows + RB - 1) / RB;
    for (int i = threadIdx.x; i < nsub * RB * nx; i += T) {
      const int rr = i / nx, ix = i - rr * nx, iy = y0 + rr;
      R u = 0;
      if (iy < y1) u = dense_pixel<R>(P, x, inv, xg, dc1[ix], dc2[iy], iy, ix, need_mom, mom);
      Us[i] = u;
    }
    __syncthreads();
    for (int task = warp; task < nsub * npair; task += nw) {
      const int sb = task / npair, b0 = 2 * (task - sb * npair);
      const R* us = Us + sb * RB * nx;
      const cpx<R>* e0 = Ex + (size_t)b0 * nx;
      const cpx<R>* e1 = Ex + (size_t)min(b0 + 1, nb - 1) * nx;
      R v[4 * RB];  // [row][column][re, im]
#pragma unroll
      for (int q = 0; q < 4 * RB; ++q) v[q] = 0;
#pragma unroll 2
      for (int ix = lane; ix < nx; ix += 32) {
        const cpx<R> ea = e0[ix], eb = e1[ix];
#pragma unroll
        for (int r = 0; r < RB; ++r) {
          const R u = us[r * nx + ix];
          v[4 * r] += u * ea.x;
          v[4 * r + 1] += u * ea.y;
          v[4 * r + 2] += u * eb.x;
          v[4 * r + 3] += u * eb.y;
        }
      }
      const R sum = warp_fold_r<4 * RB>(v, lane);
      const int q = lane / (32 / (4 * RB)), iy = y0 + sb * RB + (q >> 2), b = b0 + ((q >> 1) & 1);
      if (lane % (32 / (4 * RB)) == 0 && b < nb && iy < y1)
        (q & 1 ? tmpA[(size_t)b * ny + iy].y : tmpA[(size_t)b * ny + iy].x) = sum;
    }
    __syncthreads();
  }
}

// F2 in FP64.  A warp takes NR band rows of one or two band columns, its lanes iy
// (coalesced in Ey and tmpA).  Tiles of 4 x 2 cells where every warp has
// several (5 loads of L2 serve 8 products), single cells where the group has
// warps to spare and the latency of one product counts.
template <int NR, int NC>
__device__ __noinline__ void dft_cols(FgCtx<double>& c, const GroupCtx& g) {
  using R = double;
  const ProbDesc& P = *c.P;
  const cpx<R>* Ey = at<cpx<R>>(c.base, P.o_ey);
  const cpx<R>* tmpA = at<cpx<R>>(c.base, P.o_tmpA);  // [nb][ny]
  cpx<R>* bandA = at<cpx<R>>(c.base, P.o_bandA);
  const int ny = P.ny, nb = P.b1n, nr = P.b2n;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, tc = (nb + NC - 1) / NC, tr = (nr + NR - 1) / NR;
  for (int task = g.rank * nw + (threadIdx.x >> 5); task < tc * tr; task += g.G * nw) {
    const int r0 = task / tc * NR, b0 = task % tc * NC;
    R v[2 * NR * NC];
#pragma unroll
    for (int q = 0; q < 2 * NR * NC; ++q) v[q] = 0;
#pragma unroll 2
    for (int iy = lane; iy < ny; iy += 32) {
      cpx<R> t[NC];
#pragma unroll
      for (int k = 0; k < NC; ++k) t[k] = tmpA[(size_t)min(b0 + k, nb - 1) * ny + iy];
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const cpx<R> e = Ey[(size_t)min(r0 + r, nr - 1) * ny + iy];
#pragma unroll
        for (int k = 0; k < NC; ++k) {
          v[2 * (r * NC + k)] += e.x * t[k].x - e.y * t[k].y;
          v[2 * (r * NC + k) + 1] += e.x * t[k].y + e.y * t[k].x;
        }
      }
    }
    const R sum = warp_fold_r<2 * NR * NC>(v, lane);
    constexpr int L = 32 / (2 * NR * NC);
    const int q = lane / L, r = r0 + (q >> 1) / NC, b = b0 + (q >> 1) % NC;
    if (lane % L == 0 && r < nr && b < nb) (q & 1 ? bandA[r * nb + b].y : bandA[r * nb + b].x) = sum;
  }
}

// F1 in FP32.  Up to 128 rows at a time, the image and Ex staged in chunks of
// DFT_KC columns; a thread takes TR rows and TC band columns (4 x 4: three
// 16-byte shared loads per 32 multiply-adds; single sums for narrow shares).
template <int TR, int TC>
__device__ __noinline__ void dft_rows_seq(FgCtx<float>& c, const GroupCtx& g, double (&mom)[10]) {
  const ProbDesc& P = *c.P;
  const double* x = at<double>(c.base, P.o_x);
  const int* inv = at<int>(c.base, P.o_inv);
  double* xg = at<double>(c.base, P.o_xg);
  const double* dc1 = at<double>(c.base, P.o_dc1);
  const double* dc2 = at<double>(c.base, P.o_dc2);
  const float2* Ex = at<float2>(c.base, P.o_ex);
  float2* tmpA = at<float2>(c.base, P.o_tmpA);  // [ny][nb]
  float2* bandC = at<float2>(c.base, P.o_bandC);
  const int nx = P.nx, ny = P.ny, nb = P.b1n, ncell = P.b1n * P.b2n, T = blockDim.x;
  constexpr int RM = 128, US = RM + 4;
  const int share = (ny + g.G - 1) / g.G, y1 = min(ny, (g.rank + 1) * share);
  float* Us = reinterpret_cast<float*>(c.sbuf);              // [DFT_KC][US]
  float2* Es = reinterpret_cast<float2*>(Us + DFT_KC * US);  // [DFT_KC][DFT_NB + 2]
  constexpr int ES = DFT_NB + 2;
  for (int i = g.rank * T + threadIdx.x; i < ncell; i += g.G * T) bandC[i] = make_float2(0.f, 0.f);
  const bool need_mom = P.has_tfd || P.has_cen || P.has_sm;
  const int tcn = (nb + TC - 1) / TC;
  for (int y0 = g.rank * share; y0 < y1; y0 += RM) {
    const int rows = min(RM, y1 - y0), rpad = (rows + TR - 1) / TR * TR, ntask = rpad / TR * tcn;
    for (int t0 = 0; t0 < ntask; t0 += T) {  // one pass of the threads over the tiles
      const int task = t0 + (int)threadIdx.x, r0 = task / tcn * TR, b0 = task % tcn * TC;
      float2 acc[TR][TC];
#pragma unroll
      for (int a = 0; a < TR; ++a)
#pragma unroll
        for (int q = 0; q < TC; ++q) acc[a][q] = make_float2(0.f, 0.f);
      for (int k0 = 0; k0 < nx; k0 += DFT_KC) {
        for (int i = threadIdx.x; i < rpad * DFT_KC; i += T) {
          const int rr = i / DFT_KC, kk = i % DFT_KC, iy = y0 + rr, ix = k0 + kk;
          float u = 0.f;
          if (iy < y1 && ix < nx)
            u = dense_pixel<float>(P, x, inv, xg, dc1[ix], dc2[iy], iy, ix, need_mom && t0 == 0, mom);
          Us[kk * US + rr] = u;
        }
        for (int i = threadIdx.x; i < tcn * TC * DFT_KC; i += T) {
          const int b = i / DFT_KC, kk = i % DFT_KC, ix = k0 + kk;
          Es[kk * ES + b] = (b < nb && ix < nx) ? Ex[(size_t)b * nx + ix] : make_float2(0.f, 0.f);
        }
        __syncthreads();
        if (task < ntask) {
#pragma unroll 4
          for (int kk = 0; kk < DFT_KC; ++kk) {
            float u[TR];
            float2 e[TC];
            if constexpr (TR == 4 && TC == 4) {
              *reinterpret_cast<float4*>(u) = *reinterpret_cast<const float4*>(Us + kk * US + r0);
              *reinterpret_cast<float4*>(e) = *reinterpret_cast<const float4*>(Es + kk * ES + b0);
              *reinterpret_cast<float4*>(e + 2) = *reinterpret_cast<const float4*>(Es + kk * ES + b0 + 2);
            } else {
#pragma unroll
              for (int a = 0; a < TR; ++a) u[a] = Us[kk * US + r0 + a];
#pragma unroll
              for (int q = 0; q < TC; ++q) e[q] = Es[kk * ES + b0 + q];
            }
#pragma unroll
            for (int a = 0; a < TR; ++a)
#pragma unroll
              for (int q = 0; q < TC; ++q) {
                acc[a][q].x += u[a] * e[q].x;
                acc[a][q].y += u[a] * e[q].y;
              }
          }
        }
        __syncthreads();
      }
      if (task < ntask) {
#pragma unroll
        for (int a = 0; a < TR; ++a)
#pragma unroll
          for (int q = 0; q < TC; ++q)
            if (y0 + r0 + a < y1 && b0 + q < nb) tmpA[(size_t)(y0 + r0 + a) * nb + b0 + q] = acc[a][q];
      }
    }
  }
}

// F2 in FP32.  A thread takes a band cell; consecutive threads read
// consecutive tmpA and the same Ey.
__device__ __noinline__ void dft_cols_seq(FgCtx<float>& c, const GroupCtx& g) {
  const ProbDesc& P = *c.P;
  const float2* Ey = at<float2>(c.base, P.o_ey);
  const float2* tmpA = at<float2>(c.base, P.o_tmpA);  // [ny][nb]
  float2* bandA = at<float2>(c.base, P.o_bandA);
  const int ny = P.ny, nb = P.b1n, ncell = nb * P.b2n, share = (ncell + g.G - 1) / g.G;
  const int o1 = min(ncell, (g.rank + 1) * share);
  for (int o = g.rank * share + threadIdx.x; o < o1; o += blockDim.x) {
    const int r = o / nb;
    const float2* ey = Ey + (size_t)r * ny;
    const float2* t = tmpA + (o - r * nb);
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll 8
    for (int iy = 0; iy < ny; ++iy) {
      const float2 e = ey[iy], v = t[(size_t)iy * nb];
      acc.x += e.x * v.x - e.y * v.y;
      acc.y += e.x * v.y + e.y * v.x;
    }
    bandA[o] = acc;
  }
}

// F6 + F7.  CB image columns at a time: their tmpC in shared memory beside
// bandC, then a thread takes one image row and JC of the columns (wide shares
// take 16, so that a twiddle from L2 serves 32 multiply-adds).
template <int CB, int JC, typename R>
__device__ __noinline__ void dft_adjoint(FgCtx<R>& c, const GroupCtx& g) {
  const ProbDesc& P = *c.P;
  const cpx<R>* Ex = at<cpx<R>>(c.base, P.o_ex);
  const cpx<R>* Ey = at<cpx<R>>(c.base, P.o_ey);
  const cpx<R>* bandC = at<cpx<R>>(c.base, P.o_bandC);
  const double* dc1 = at<double>(c.base, P.o_dc1);
  const double* dc2 = at<double>(c.base, P.o_dc2);
  double* gchi = at<double>(c.base, P.o_gchi);
  const int nx = P.nx, ny = P.ny, nb = P.b1n, nr = P.b2n;
  const int T = blockDim.x;
  cpx<R>* Cs = c.sbuf;                    // [nr][CB]
  cpx<R>* Bs = c.sbuf + DFT_NB * CB;      // [nr][nb]
  const int share = (nx + g.G - 1) / g.G, x1 = min(nx, (g.rank + 1) * share);
  if (g.rank * share >= x1) return;
  for (int i = threadIdx.x; i < nr * nb; i += T) Bs[i] = bandC[i];
  for (int x0 = g.rank * share; x0 < x1; x0 += CB) {
    const int cols = min(CB, x1 - x0), cj = (cols + JC - 1) / JC;
    __syncthreads();
    for (int i = threadIdx.x; i < nr * JC * cj; i += T) {
      const int r = i / (JC * cj), cc = i - r * JC * cj;
      cpx<R> t = cmk<R>(0, 0);
      if (cc < cols) {
        const cpx<R>* ex = Ex + x0 + cc;
        const cpx<R>* v = Bs + r * nb;
#pragma unroll 8
        for (int b = 0; b < nb; ++b) {
          const cpx<R> e = ex[(size_t)b * nx], w = v[b];
          t.x += w.x * e.x - w.y * e.y;
          t.y += w.x * e.y + w.y * e.x;
        }
      }
      Cs[r * CB + cc] = t;
    }
    __syncthreads();
    for (int it = threadIdx.x; it < ny * cj; it += T) {
      const int cq = it / ny, iy = it - cq * ny;
      const cpx<R>* ey = Ey + iy;
      const cpx<R>* t = Cs + JC * cq;
      R acc[JC];
#pragma unroll
      for (int j = 0; j < JC; ++j) acc[j] = 0;
#pragma unroll 4
      for (int r = 0; r < nr; ++r) {
        const cpx<R> e = ey[(size_t)r * ny];
#pragma unroll
        for (int j = 0; j < JC; ++j) acc[j] += e.x * t[r * CB + j].x - e.y * t[r * CB + j].y;
      }
      const double d2 = dc2[iy];
#pragma unroll
      for (int j = 0; j < JC; ++j) {
        const int ix = x0 + JC * cq + j;
        if (ix < x1) gchi[(size_t)iy * nx + ix] = (double)acc[j] * dc1[ix] * d2;
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// F1: type-2 row pass.  Deconvolved image rows -> band columns of the
// row-transformed fine grid (tmpA[iy][b], b < b1n).  Also zeroes bandC.
// Optionally accumulates image moments for the global regularizers.
// ---------------------------------------------------------------------------
template <typename R>
__device__ __noinline__ void fg_t2_rows(FgCtx<R>& c, const GroupCtx& g, double (&mom)[10]) {
  if (c.P->dft) {
    const int share = (c.P->ny + g.G - 1) / g.G;
    if constexpr (sizeof(R) == 8) {
      if (share <= 4) dft_rows<4>(c, g, mom);
      else dft_rows<8>(c, g, mom);
    } else {
      if (share <= 16) dft_rows_seq<1, 1>(c, g, mom);
      else dft_rows_seq<4, 4>(c, g, mom);
    }
    return;
  }
  const ProbDesc& P = *c.P;
  const double* x = at<double>(c.base, P.o_x);
  const int* inv = at<int>(c.base, P.o_inv);
  double* xg = at<double>(c.base, P.o_xg);
  const double* dc1 = at<double>(c.base, P.o_dc1);
  const double* dc2 = at<double>(c.base, P.o_dc2);
  const cpx<R>* tw1 = at<cpx<R>>(c.base, P.o_tw1);
  cpx<R>* tmpA = at<cpx<R>>(c.base, P.o_tmpA);
  cpx<R>* bandC = at<cpx<R>>(c.base, P.o_bandC);
  const int n1 = P.nf1, nx = P.nx, ny = P.ny;
  const FftPlan pl = make_plan(n1);
  const int S = min(fft_batch(n1), c.smem_cpx / n1);
  for (int i = g.rank * blockDim.x + threadIdx.x; i < P.b2n * P.b1n; i += g.G * blockDim.x)
    bandC[i] = cmk<R>(0, 0);
  const bool need_mom = P.has_tfd || P.has_cen || P.has_sm;
  for (int row0 = g.rank * S; row0 < ny; row0 += g.G * S) {
    const int rows = min(S, ny - row0);
    for (int i = threadIdx.x; i < rows * n1; i += blockDim.x) c.sbuf[i] = cmk<R>(0, 0);
    __syncthreads();
    for (int i = threadIdx.x; i < rows * nx; i += blockDim.x) {
      const int s = i / nx, ix = i - s * nx, iy = row0 + s;
      const int pv = P.ident ? iy * nx + ix : inv[iy * nx + ix];
      const double val = pv >= 0 ? x[pv] : 0.0;
      if (!P.ident) xg[(size_t)iy * nx + ix] = val;
      c.sbuf[s * n1 + wrapn(ix - nx / 2, n1)] = cmk<R>((R)(val * dc1[ix] * dc2[iy]), (R)0);
      if (need_mom && pv >= 0) {
        const double fx = ix + 1, fy = iy + 1;  // 1-based pixel numbers as the reference
        mom[0] += val;
        mom[1] += fabs(val);
        mom[2] += val * fx;
        mom[3] += val * fy;
        mom[4] += val * fx * fx;
        mom[5] += val * fy * fy;
        mom[6] += val * fx * fy;
        if (P.has_cen) {
          const double Ip = fabs(P.cen_alpha - 1) < 1e-10 ? smabs(val) : pow(smabs(val), P.cen_alpha);
          mom[7] += Ip * (fx - P.nxref);
          mom[8] += Ip * (fy - P.nyref);
          mom[9] += Ip;
        }
      }
    }
    __syncthreads();
    const cpx<R>* out = smem_fft(c.sbuf, c.swork, pl, rows, tw1);
    for (int i = threadIdx.x; i < rows * P.b1n; i += blockDim.x) {
      const int s = i / P.b1n, b = i - s * P.b1n;
      tmpA[(size_t)(row0 + s) * P.b1n + b] = out[s * n1 + wrapn(P.b1s + b, n1)];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// F2: type-2 column pass over band columns -> bandA[b2][b1]
// ---------------------------------------------------------------------------
template <typename R>
__device__ __noinline__ void fg_t2_cols(FgCtx<R>& c, const GroupCtx& g) {
  if (c.P->dft) {
    if constexpr (sizeof(R) == 8) {
      if (c.P->b1n * c.P->b2n > g.G * (int)(blockDim.x >> 5) * 8) dft_cols<4, 2>(c, g);
      else dft_cols<1, 1>(c, g);
    } else {
      dft_cols_seq(c, g);
    }
    return;
  }
  const ProbDesc& P = *c.P;
  const cpx<R>* tw2 = at<cpx<R>>(c.base, P.o_tw2);
  const cpx<R>* tmpA = at<cpx<R>>(c.base, P.o_tmpA);
  cpx<R>* bandA = at<cpx<R>>(c.base, P.o_bandA);
  const int n2 = P.nf2, ny = P.ny, b1n = P.b1n;
  const FftPlan pl = make_plan(n2);
  const int S = min(fft_batch(n2), c.smem_cpx / n2);
  for (int b0 = g.rank * S; b0 < b1n; b0 += g.G * S) {
    const int cols = min(S, b1n - b0);
    for (int i = threadIdx.x; i < cols * n2; i += blockDim.x) c.sbuf[i] = cmk<R>(0, 0);
    __syncthreads();
    for (int i = threadIdx.x; i < cols * ny; i += blockDim.x) {
      const int iy = i / cols, s = i - iy * cols;
      c.sbuf[s * n2 + wrapn(iy - ny / 2, n2)] = tmpA[(size_t)iy * b1n + b0 + s];
    }
    __syncthreads();
    const cpx<R>* out = smem_fft(c.sbuf, c.swork, pl, cols, tw2);
    for (int i = threadIdx.x; i < cols * P.b2n; i += blockDim.x) {
      const int b2 = i / cols, s = i - b2 * cols;
      bandA[(size_t)b2 * b1n + b0 + s] = out[s * n2 + wrapn(P.b2s + b2, n2)];
    }
    __syncthreads();
  }
}

// The kernel weights of every uv point, taps[q][j] = psi at tap q < w of axis 1
// and [w + q][j] of axis 2, once per launch (P.o_taps).  The points do not
// move, and 2 w exponentials and roots per point and use cost more than
// everything else interpolation and spreading do (in FP32 some 280 of 500
// instructions of an interpolated point); read back, they are 2 w coalesced
// loads.
template <typename R>
__device__ __noinline__ void fg_taps(const ProbDesc& P, char* base, const GroupCtx& g) {
  const R* xu = at<R>(base, P.o_u);
  const R* xv = at<R>(base, P.o_v);
  R* taps = at<R>(base, P.o_taps);
  const int w = P.w, n = P.nuv;
  const R beta = (R)P.beta, half = (R)0.5 * (R)w, inv = (R)1 / half;
  for (int i = g.rank * blockDim.x + threadIdx.x; i < 2 * n; i += g.G * blockDim.x) {
    const int j = i < n ? i : i - n;
    const R x = i < n ? xu[j] : xv[j];
    const int l = (int)ceil(x - half);
    R* t = taps + (i < n ? (size_t)0 : (size_t)w * n) + j;
#pragma unroll 4
    for (int q = 0; q < w; ++q) t[(size_t)q * n] = es_kernel(((R)(l + q) - x) * inv, beta);
  }
}

// Interpolation of the points j = j0, j0 + dj, ... < nuv from the band:
// V_j = sum_b psi(v_j - l2 - b) sum_a psi(u_j - l1 - a) band[l2 + b][l1 + a].
// The kernel width W is a template constant so both tap vectors stay in
// registers and the W row loads of a tap row issue back to back.
template <int W, typename R>
__device__ __noinline__ void interp_points(const ProbDesc& P, const R* __restrict__ xu, const R* __restrict__ xv,
                                              const cpx<R>* bandA, cpx<R>* V, cpx<R>* cacc, R beta, int j0,
                                              int dj, const R* taps) {
  const R half = (R)0.5 * (R)W;
  const R inv = (R)1 / half;
  for (int j = j0; j < P.nuv; j += dj) {
    const R x1 = xu[j], x2 = xv[j];
    const int l1 = (int)ceil(x1 - half), l2 = (int)ceil(x2 - half);
    R k1[W], k2[W];
    if (taps) {
#pragma unroll
      for (int a = 0; a < W; ++a) {
        k1[a] = taps[(size_t)a * P.nuv + j];
        k2[a] = taps[(size_t)(W + a) * P.nuv + j];
      }
    } else {
#pragma unroll
      for (int a = 0; a < W; ++a) {
        k1[a] = es_kernel(((R)(l1 + a) - x1) * inv, beta);
        k2[a] = es_kernel(((R)(l2 + a) - x2) * inv, beta);
      }
    }
    const int c1 = imod(l1 - P.b1s, P.nf1), c2 = imod(l2 - P.b2s, P.nf2);
    R ar = 0, ai = 0;
#pragma unroll
    for (int b = 0; b < W; ++b) {
      int rw = c2 + b;  // wraps only when the band spans the whole fine grid
      if (rw >= P.nf2) rw -= P.nf2;
      const cpx<R>* row = bandA + (size_t)rw * P.b1n;
      R rr = 0, ri = 0;
#pragma unroll
      for (int a = 0; a < W; ++a) {
        int cl = c1 + a;
        if (cl >= P.nf1) cl -= P.nf1;
        const cpx<R> q = row[cl];
        rr += k1[a] * q.x;
        ri += k1[a] * q.y;
      }
      ar += k2[b] * rr;
      ai += k2[b] * ri;
    }
    V[j] = cmk(ar, ai);
    if (cacc) cacc[j] = cmk<R>(0, 0);
  }
}

// ---------------------------------------------------------------------------
// F3: type-2 interpolation, V_j = sum psi psi bandA.  With zero_acc it also
// clears the points' derivative accumulators that F4 adds into.
// ---------------------------------------------------------------------------
template <typename R>
__device__ void fg_interp(FgCtx<R>& c, const GroupCtx& g, bool zero_acc) {
  const ProbDesc& P = *c.P;
  const R* xu = at<R>(c.base, P.o_u);
  const R* xv = at<R>(c.base, P.o_v);
  const cpx<R>* gband = at<cpx<R>>(c.base, P.o_bandA);
  cpx<R>* V = at<cpx<R>>(c.base, P.o_V);
  cpx<R>* cacc = zero_acc ? at<cpx<R>>(c.base, P.o_contrib) : nullptr;
  const R* taps = P.o_taps ? at<R>(c.base, P.o_taps) : nullptr;
  const int w = P.w;
  const R beta = (R)P.beta;
  const int ncell = P.b1n * P.b2n;
  // the band is re-read w*w times per point: stage it in shared memory
  const bool staged = ncell <= c.dyn_cpx;
  const cpx<R>* bandA = gband;
  if (staged) {
    // only CTAs that own points load the band
    if (g.rank * (int)blockDim.x < P.nuv) {
      for (int i = threadIdx.x; i < ncell; i += blockDim.x) c.sbuf[i] = gband[i];
      __syncthreads();
      bandA = c.sbuf;
    }
  }
  const int j0 = g.rank * blockDim.x + threadIdx.x, dj = g.G * blockDim.x;
  switch (w) {
#define SMILI_INTERP_W(W) \
  case W: interp_points<W>(P, xu, xv, bandA, V, cacc, beta, j0, dj, taps); break;
    SMILI_INTERP_W(2) SMILI_INTERP_W(3) SMILI_INTERP_W(4) SMILI_INTERP_W(5) SMILI_INTERP_W(6)
    SMILI_INTERP_W(7) SMILI_INTERP_W(8) SMILI_INTERP_W(9) SMILI_INTERP_W(10) SMILI_INTERP_W(11)
    SMILI_INTERP_W(12) SMILI_INTERP_W(13) SMILI_INTERP_W(14) SMILI_INTERP_W(15)
    default: interp_points<16>(P, xu, xv, bandA, V, cacc, beta, j0, dj, taps); break;  // w <= SMILI_MAXW = 16
#undef SMILI_INTERP_W
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// F4: chi-square terms, and their derivatives with respect to each model
// visibility added into that uv point's accumulator (o_contrib, zeroed by F3)
// with global atomics: one vector reduction per contribution in FP32, two in
// FP64.  The accumulators (one complex value per uv point) are small enough
// to stay in L2 while the data stream past, and spreading then reads them in
// its own point order.
// chi[0..3] = fcv, amp, cp, ca (weighted by the normalised data weights).
// ---------------------------------------------------------------------------
template <typename R>
__device__ __noinline__ void fg_chisq(FgCtx<R>& c, const GroupCtx& g, double (&chi)[4]) {
  const ProbDesc& P = *c.P;
  const cpx<R>* V = at<cpx<R>>(c.base, P.o_V);
  const R* dre = at<R>(c.base, P.o_dre);
  const R* dim = at<R>(c.base, P.o_dim);
  const R* dvar = at<R>(c.base, P.o_dvar);
  const int* didx = at<int>(c.base, P.o_didx);
  const signed char* dsgn = at<signed char>(c.base, P.o_dsgn);
  cpx<R>* cacc = at<cpx<R>>(c.base, P.o_contrib);
  typedef typename std::conditional<sizeof(R) == 8, KSum, KSumF>::type Acc;
  Acc acc[4];
  for (int q = 0; q < 4; ++q) acc[q].s = acc[q].c = 0;
  const int e_amp = P.nfcv, e_cp = e_amp + P.namp, e_ca = e_cp + P.ncp, e_end = e_ca + P.nca;
  const int s_amp = P.nfcv, s_cp = s_amp + P.namp, s_ca = s_cp + 3 * P.ncp;
  const R wf = (R)P.wfcv, wa = (R)P.wamp, wc = (R)P.wcp, wq = (R)P.wca;
  // model_fcv/amp/cp/ca (fftlib.f90:744-1254) also return each datum's model and residual
  double* mres = P.o_model ? at<double>(c.base, P.o_model) : nullptr;
  // One loop per data type over the same items (i = j0 + k dj) in the same
  // order as a single loop, two items per step: both items' gathers are
  // issued before either is evaluated, so their latencies overlap.
  const int j0 = g.rank * blockDim.x + threadIdx.x, dj = g.G * blockDim.x;
  auto first = [&](int a) { return a <= j0 ? j0 : j0 + (a - j0 + dj - 1) / dj * dj; };
  auto put = [&](int i, R model, R model2, R resid, R resid2) {
    if (mres) {
      mres[4 * i] = model;
      mres[4 * i + 1] = model2;
      mres[4 * i + 2] = resid;
      mres[4 * i + 3] = resid2;
    }
  };
  // complex visibilities (fftlib.f90:384-439)
  auto fcv = [&](int i, int k, const cpx<R>& Vk, R sg, R var, R yr, R yi) {
    const R rr = yr - Vk.x, ri = yi - sg * Vk.y;
    acc[0].add(((rr * rr + ri * ri) / var) * wf);
    const R factor = (R)-2 / var * wf;
    acc_add(cacc + k, cmk(factor * rr, factor * ri * sg));
    put(i, Vk.x, sg * Vk.y, rr, ri);
  };
  for (int i = first(0); i < e_amp; i += 2 * dj) {
    const int ib = i + dj;
    const bool two = ib < e_amp;
    const int ka = didx[i], kb = two ? didx[ib] : ka;
    const cpx<R> Va = V[ka], Vb = V[kb];
    const R sa = (R)dsgn[i], sb = two ? (R)dsgn[ib] : sa;
    const R va = dvar[i], vb = two ? dvar[ib] : va;
    const R ra = dre[i], rb = two ? dre[ib] : ra, ia = dim[i], ibm = two ? dim[ib] : ia;
    fcv(i, ka, Va, sa, va, ra, ia);
    if (two) fcv(ib, kb, Vb, sb, vb, rb, ibm);
  }
  // amplitudes (fftlib.f90:442-493)
  auto amp = [&](int i, int k, const cpx<R>& Vk, R var, R y) {
    const R model = sqrt(Vk.x * Vk.x + Vk.y * Vk.y);
    const R resid = y - model;
    acc[1].add((resid * resid / var) * wa);
    const R factor = (R)-2 * resid / var / model * wa;
    acc_add(cacc + k, cmk(factor * Vk.x, factor * Vk.y));
    put(i, model, 0, resid, 0);
  };
  for (int i = first(e_amp); i < e_cp; i += 2 * dj) {
    const int ib = i + dj;
    const bool two = ib < e_cp;
    const int ka = didx[s_amp + (i - e_amp)], kb = two ? didx[s_amp + (ib - e_amp)] : ka;
    const cpx<R> Va = V[ka], Vb = V[kb];
    const R va = dvar[i], vb = two ? dvar[ib] : va;
    const R ya = dre[i], yb = two ? dre[ib] : ya;
    amp(i, ka, Va, va, ya);
    if (two) amp(ib, kb, Vb, vb, yb);
  }
  // closure phases (fftlib.f90:576-655)
  auto cp = [&](int i, const int (&kq)[3], const cpx<R> (&Vq)[3], const R (&sg)[3], R var, R y) {
    R a2[3];
    R model = 0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      a2[q] = Vq[q].x * Vq[q].x + Vq[q].y * Vq[q].y;
      model = atan2(Vq[q].y, Vq[q].x) * sg[q] + model;
    }
    const R resid = y - model;
    R sr, cr;
    if (sizeof(R) == 8) {
      double s_, c_;
      sincos((double)resid, &s_, &c_);
      sr = (R)s_;
      cr = (R)c_;
    } else {
      float s_, c_;
      sincosf((float)resid, &s_, &c_);
      sr = (R)s_;
      cr = (R)c_;
    }
    acc[2].add(((R)2 * ((R)1 - cr) / var) * wc);
    const R factor = (R)-2 * sr / var * wc;
#pragma unroll
    for (int q = 0; q < 3; ++q)
      acc_add(cacc + kq[q], cmk(-factor / a2[q] * Vq[q].y * sg[q], factor / a2[q] * Vq[q].x * sg[q]));
    put(i, model, 0, resid, 0);  // unwrapped; the host wraps both into (-pi, pi] as model_cp does
  };
  for (int i = first(e_cp); i < e_ca; i += 2 * dj) {
    const int ib = i + dj;
    const bool two = ib < e_ca;
    const int sa = s_cp + 3 * (i - e_cp), sb = two ? s_cp + 3 * (ib - e_cp) : sa;
    int ka[3], kb[3];
    cpx<R> Va[3], Vb[3];
    R ga[3], gb[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      ka[q] = didx[sa + q];
      kb[q] = didx[sb + q];
      ga[q] = (R)dsgn[sa + q];
      gb[q] = (R)dsgn[sb + q];
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      Va[q] = V[ka[q]];
      Vb[q] = V[kb[q]];
    }
    const R va = dvar[i], vb = two ? dvar[ib] : va;
    const R ya = dre[i], yb = two ? dre[ib] : ya;
    cp(i, ka, Va, ga, va, ya);
    if (two) cp(ib, kb, Vb, gb, vb, yb);
  }
  // log closure amplitudes (fftlib.f90:496-573)
  auto ca = [&](int i, const int (&kq)[4], const cpx<R> (&Vq)[4], R var, R y) {
    R a[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = sqrt(Vq[q].x * Vq[q].x + Vq[q].y * Vq[q].y);
    const R model = log(a[0]) + log(a[1]) - log(a[2]) - log(a[3]);
    const R resid = y - model;
    acc[3].add((resid * resid / var) * wq);
    const R factor = (R)-2 * resid / var * wq;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const R f = (q < 2 ? factor : -factor) / (a[q] * a[q]);
      acc_add(cacc + kq[q], cmk(f * Vq[q].x, f * Vq[q].y));
    }
    put(i, model, 0, resid, 0);
  };
  for (int i = first(e_ca); i < e_end; i += 2 * dj) {
    const int ib = i + dj;
    const bool two = ib < e_end;
    const int sa = s_ca + 4 * (i - e_ca), sb = two ? s_ca + 4 * (ib - e_ca) : sa;
    int ka[4], kb[4];
    cpx<R> Va[4], Vb[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      ka[q] = didx[sa + q];
      kb[q] = didx[sb + q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      Va[q] = V[ka[q]];
      Vb[q] = V[kb[q]];
    }
    const R va = dvar[i], vb = two ? dvar[ib] : va;
    const R ya = dre[i], yb = two ? dre[ib] : ya;
    ca(i, ka, Va, va, ya);
    if (two) ca(ib, kb, Vb, vb, yb);
  }
  for (int q = 0; q < 4; ++q) chi[q] += acc[q].value();
}

// ---------------------------------------------------------------------------
// F5: spread c_j = Vresre_j - i Vresim_j, read from the uv points'
// derivative accumulators in the bin-sorted point order, onto bandC.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void atomic_add_r(double* p, double v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_r(float* p, float v) { atomicAdd(p, v); }

// The work item that holds point p0 (items cover the points in order)
__device__ __forceinline__ int item_of(const int4* items, int nitems, int p0) {
  int it = 0;
  for (int hi = nitems; hi - it > 1;) {
    const int mid = (it + hi) >> 1;
    if (items[mid].x <= p0) it = mid;
    else hi = mid;
  }
  return it;
}

// ---------------------------------------------------------------------------
// F5 in FP64 with the subgrid in registers (w <= 9, 8 x 8 tiles).  The warps
// take equal contiguous ranges of the sorted points (at least 32), so that no
// warp walks a 128-point item while others have none.  A warp holds its
// tile's 16 x 16 subgrid as 8 rows of one column per lane; a point's weights
// sit in a zero-padded 16-entry row per axis in shared memory at its offset
// inside the tile, so a lane reads its column's weight, the 8 row weights
// (the same address in half a warp) and does 16 independent FMAs: no tap
// waits on the point before, as it does with a subgrid in shared memory.  The
// tile is added to the band when the next point lies in another one.
// 256 x 256 / 97 200 points, 64 CTAs, a solve's stage with its barrier: 126 us
// with shared subgrids and the weights evaluated each time, 33 us with this
// and fg_taps.
// ---------------------------------------------------------------------------
constexpr int SPREAD_ROW = 34;  // 16 axis-1 weights, 16 axis-2 weights, Re c, Im c
template <int W>
__device__ __noinline__ void fg_spread_reg(FgCtx<double>& c, const GroupCtx& g) {
  const ProbDesc& P = *c.P;
  const double* xu = at<double>(c.base, P.o_u);
  const double* xv = at<double>(c.base, P.o_v);
  const double* taps = P.o_taps ? at<double>(c.base, P.o_taps) : nullptr;
  const int4* items = at<int4>(c.base, P.o_items);
  const cpx<double>* cacc = at<cpx<double>>(c.base, P.o_contrib);
  double* gband = at<double>(c.base, P.o_bandC);
  const double beta = P.beta, half = 0.5 * W, inv = 1.0 / half;
  const int nuv = P.nuv, nf1 = P.nf1, nf2 = P.nf2, b1s = P.b1s, b2s = P.b2s, b1n = P.b1n, b2n = P.b2n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int col = lane & 15, r0 = (lane >> 4) * 8;
  double* tab = reinterpret_cast<double*>(c.sbuf) + (size_t)warp * 32 * SPREAD_ROW;
  const int nwt = g.G * nw, gw = g.rank * nw + warp;
  const int share = max(32, (nuv + nwt - 1) / nwt);
  const long first = (long)gw * share;
  if (first >= nuv) return;
  const int p0 = (int)first, p1 = min(nuv, p0 + share);
  int it = item_of(items, P.nitems, p0);
  double ar[8], ai[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) ar[i] = ai[i] = 0.0;
  int trow = -1, tcol = -1;
  auto flush = [&]() {
    int cl = tcol + col;
    if (cl >= nf1) cl -= nf1;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      int rw = trow + r0 + i;
      if (rw >= nf2) rw -= nf2;
      // outside the tile's 8 + W - 1 cells, or beyond the band, only zero taps land
      if (r0 + i < 8 + W - 1 && col < 8 + W - 1 && rw < b2n && cl < b1n && (ar[i] != 0.0 || ai[i] != 0.0)) {
        double* dst = gband + 2 * ((size_t)rw * b1n + cl);
        atomicAdd(dst, ar[i]);
        atomicAdd(dst + 1, ai[i]);
      }
      ar[i] = ai[i] = 0.0;
    }
  };
  for (int jb = p0; jb < p1; ++it) {
    const int4 item = items[it];
    if (item.z != trow || item.w != tcol) {
      if (trow >= 0) flush();
      trow = item.z;
      tcol = item.w;
    }
    const int je = min(p1, item.y);
    for (; jb < je; jb += 32) {
      const int np = min(32, je - jb);
      if (lane < np) {
        const int j = jb + lane;
        double* row = tab + lane * SPREAD_ROW;
        const cpx<double> cj = cacc[j];
        const double x1 = xu[j], x2 = xv[j];
        const int l1 = (int)ceil(x1 - half), l2 = (int)ceil(x2 - half);
        double k1[W], k2[W];
        if (taps) {
#pragma unroll
          for (int q = 0; q < W; ++q) {
            k1[q] = taps[(size_t)q * nuv + j];
            k2[q] = taps[(size_t)(W + q) * nuv + j];
          }
        } else {
#pragma unroll
          for (int q = 0; q < W; ++q) {
            k1[q] = es_kernel(((double)(l1 + q) - x1) * inv, beta);
            k2[q] = es_kernel(((double)(l2 + q) - x2) * inv, beta);
          }
        }
        const int lc = imod(l1 - b1s, nf1) - tcol, lr = imod(l2 - b2s, nf2) - trow;  // in [0, 8)
#pragma unroll
        for (int q = 0; q < 16; ++q) reinterpret_cast<double2*>(row)[q] = make_double2(0.0, 0.0);
        reinterpret_cast<double2*>(row)[16] = make_double2(cj.x, -cj.y);  // c = Vresre - i Vresim
#pragma unroll
        for (int q = 0; q < W; ++q) {
          row[lc + q] = k1[q];
          row[16 + lr + q] = k2[q];
        }
      }
      __syncwarp();
#pragma unroll 2
      for (int p = 0; p < np; ++p) {
        const double* row = tab + p * SPREAD_ROW;
        const double2 cv = *reinterpret_cast<const double2*>(row + 32);
        const double wx = row[col];
        const double2* wy = reinterpret_cast<const double2*>(row + 16 + r0);
        const double a = wx * cv.x, b = wx * cv.y;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double2 y = wy[i];
          ar[2 * i] += y.x * a;
          ai[2 * i] += y.x * b;
          ar[2 * i + 1] += y.y * a;
          ai[2 * i + 1] += y.y * b;
        }
      }
      __syncwarp();
    }
    jb = je;
  }
  flush();
}

// ---------------------------------------------------------------------------
// F5 in FP32 on the tensor cores (w <= 9, 8 x 8 tiles).  A tile's subgrid is
// a product of two thin matrices:
//   D[r][c] = sum_p wy_p[r] (c_p wx_p[c]),   r, c < 8 + w - 1 <= 16,
// with wy_p / wx_p the point's kernel weights placed at its offset inside
// the subgrid (zero elsewhere) and c_p = Vres_re - i Vres_im of the point.
// A warp accumulates the real and imaginary parts of one tile's 16 x 16
// subgrid in mma.sync.m16n8k8 TF32 fragments (8 points per k step) with the
// three-term split a b ~ ah bh + ah bl + al bh (a = ah + al in TF32), which
// keeps the products within a few FP32 ulps.  The operands of 16 points at a
// time lie in shared memory already padded and multiplied, wx Re c | wx Im c |
// wy, 56 floats apart (the 8 rows x 4 points a fragment reads are 32 banks),
// so a fragment element is one load and its split, and the loads of the next
// 16 points' taps are in flight meanwhile.  As in FP64 the warps take equal
// contiguous ranges; a tile is added to the band at the end of its work item
// (at most 128 points).
// 74 problems of 97 200 points on groups of 4 CTAs, a solve's stage with its
// barrier: 400 us with operands looked up and multiplied per fragment (520
// instructions per 8 points) and the weights evaluated each time; with a
// CUDA-core subgrid as in FP64 547 us (its row loads fill the shared-memory
// pipe); 372 us with this and fg_taps.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = to_tf32(x);
  lo = to_tf32(x - __uint_as_float(hi));
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int SPREAD_TC_ROW = 56;     // floats per point: 16 wx Re c, 16 wx Im c, 16 wy, 8 unused
constexpr int SPREAD_TC_POINTS = 16;  // points staged per warp
template <int W>
__device__ __noinline__ void fg_spread_tc(FgCtx<float>& c, const GroupCtx& g) {
  const ProbDesc& P = *c.P;
  const float* xu = at<float>(c.base, P.o_u);
  const float* xv = at<float>(c.base, P.o_v);
  const float* taps = P.o_taps ? at<float>(c.base, P.o_taps) : nullptr;
  const int4* items = at<int4>(c.base, P.o_items);
  const cpx<float>* cacc = at<cpx<float>>(c.base, P.o_contrib);
  cpx<float>* gband = at<cpx<float>>(c.base, P.o_bandC);
  const float beta = (float)P.beta, half = 0.5f * W, inv = 1.f / half;
  const int nuv = P.nuv, nf1 = P.nf1, nf2 = P.nf2, b1n = P.b1n, b2n = P.b2n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int gq = lane >> 2, t = lane & 3;
  float* tab = reinterpret_cast<float*>(c.sbuf) + (size_t)warp * SPREAD_TC_POINTS * SPREAD_TC_ROW;
  const int nwt = g.G * nw, gw = g.rank * nw + warp;
  const int share = max(32, (nuv + nwt - 1) / nwt);
  const long first = (long)gw * share;
  if (first >= nuv) return;
  const int p0 = (int)first, p1 = min(nuv, p0 + share);
  int it = item_of(items, P.nitems, p0);
  // lanes 0..15 prepare axis 1 (times c) of a point, lanes 16..31 axis 2
  const int pt = lane & 15;
  const bool ax1 = lane < 16;
  const float* xs = ax1 ? xu : xv;
  const float* tp = taps ? taps + (ax1 ? (size_t)0 : (size_t)W * nuv) : nullptr;
  const int bs = ax1 ? P.b1s : P.b2s, nf = ax1 ? nf1 : nf2;
  float k[W], x = 0.f;
  cpx<float> cj = cmk<float>(0.f, 0.f);
  auto fetch = [&](int j) {  // point j's coordinate, weights and value into registers
    if (j < p1) {
      x = xs[j];
      if (tp) {
#pragma unroll
        for (int q = 0; q < W; ++q) k[q] = tp[(size_t)q * nuv + j];
      }
      if (ax1) cj = cacc[j];
    }
  };
  fetch(p0 + pt);
  for (int jb = p0; jb < p1; ++it) {
    const int4 item = items[it];
    const int origin = ax1 ? item.w : item.z;
    const int je = min(p1, item.y);
    float dre[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}}, dim[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
    while (jb < je) {
      const int np = min(SPREAD_TC_POINTS, je - jb);
      {
        float* row = tab + pt * SPREAD_TC_ROW + (ax1 ? 0 : 32);
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4* r4 = reinterpret_cast<float4*>(row);
#pragma unroll
        for (int q = 0; q < 4; ++q) r4[q] = zero;
        if (ax1) {
#pragma unroll
          for (int q = 4; q < 8; ++q) r4[q] = zero;
        }
        if (pt < np) {
          const int l = (int)ceilf(x - half);
          if (!tp) {
#pragma unroll
            for (int q = 0; q < W; ++q) k[q] = es_kernel(((float)(l + q) - x) * inv, beta);
          }
          const int o = imod(l - bs, nf) - origin;  // in [0, 8)
          if (ax1) {
#pragma unroll
            for (int q = 0; q < W; ++q) {
              row[o + q] = k[q] * cj.x;
              row[16 + o + q] = k[q] * -cj.y;  // c = Vresre - i Vresim
            }
          } else {
#pragma unroll
            for (int q = 0; q < W; ++q) row[o + q] = k[q];
          }
        }
      }
      jb += np;
      fetch(jb + pt);
      __syncwarp();
      // 8 points per k step; lane (gq, t) feeds points t and t + 4
#pragma unroll
      for (int kb = 0; kb < SPREAD_TC_POINTS; kb += 8) {
        if (kb >= np) break;
        const float* w0 = tab + (kb + t) * SPREAD_TC_ROW + gq;
        const float* w1 = w0 + 4 * SPREAD_TC_ROW;
        uint32_t ah[4], al[4];
        split_tf32(w0[32], ah[0], al[0]);
        split_tf32(w0[40], ah[1], al[1]);
        split_tf32(w1[32], ah[2], al[2]);
        split_tf32(w1[40], ah[3], al[3]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint32_t h0, l0, h1, l1;
          split_tf32(w0[8 * j], h0, l0);
          split_tf32(w1[8 * j], h1, l1);
          mma_tf32(dre[j], ah, h0, h1);
          mma_tf32(dre[j], ah, l0, l1);
          mma_tf32(dre[j], al, h0, h1);
          split_tf32(w0[16 + 8 * j], h0, l0);
          split_tf32(w1[16 + 8 * j], h1, l1);
          mma_tf32(dim[j], ah, h0, h1);
          mma_tf32(dim[j], ah, l0, l1);
          mma_tf32(dim[j], al, h0, h1);
        }
      }
      __syncwarp();
    }
    // add the subgrid to the band: fragment element e of n-tile j is
    // (row gq + 8 (e >= 2), col 8 j + 2 t + (e & 1))
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = gq + (e >= 2 ? 8 : 0), cc = 8 * j + 2 * t + (e & 1);
        const float vr = dre[j][e], vi = dim[j][e];
        if (r >= 8 + W - 1 || cc >= 8 + W - 1 || (vr == 0.f && vi == 0.f)) continue;
        int rw = item.z + r, cl = item.w + cc;
        if (rw >= nf2) rw -= nf2;
        if (cl >= nf1) cl -= nf1;
        if (rw < b2n && cl < b1n) acc_add(gband + ((size_t)rw * b1n + cl), cmk(vr, vi));  // else only zero taps land here
      }
    }
  }
}

// F5 for any bin and width (the two above where they apply): subproblem
// spreading.  The bin-sorted points are cut into work items of at most 128
// points that share one bin of the band.  A warp owns an item and a private
// (bin+w-1)^2 subgrid in shared memory: for every point the lanes cover the w*w
// taps (all lanes hit different cells, and consecutive points are ordered by
// __syncwarp), so the inner loop needs no atomics.  The finished subgrid is
// added to the CTA's band copy (shared atomics, only the overlapping halos
// collide) and the CTA's band to the global band at the end.
template <typename R>
__device__ __noinline__ void fg_spread(FgCtx<R>& c, const GroupCtx& g) {
  if (c.P->bin == 8) {
    switch (c.P->w) {
#define SMILI_SPREAD_W(W)                                                      \
  case W:                                                                      \
    if constexpr (std::is_same<R, double>::value) fg_spread_reg<W>(c, g);      \
    else fg_spread_tc<W>(c, g);                                                \
    return;
      SMILI_SPREAD_W(2) SMILI_SPREAD_W(3) SMILI_SPREAD_W(4) SMILI_SPREAD_W(5) SMILI_SPREAD_W(6)
      SMILI_SPREAD_W(7) SMILI_SPREAD_W(8) SMILI_SPREAD_W(9)
#undef SMILI_SPREAD_W
      default: break;  // a subgrid wider than 16 cells
    }
  }
  const ProbDesc& P = *c.P;
  const R* xu = at<R>(c.base, P.o_u);
  const R* xv = at<R>(c.base, P.o_v);
  const int4* items = at<int4>(c.base, P.o_items);
  const cpx<R>* cacc = at<cpx<R>>(c.base, P.o_contrib);
  R* gband = at<R>(c.base, P.o_bandC);
  const int w = P.w, ww = P.w * P.w;
  const int SG = P.bin + w - 1;  // subgrid side
  const R beta = (R)P.beta;
  const R half = (R)0.5 * (R)w, inv = (R)1 / half;
  const int ncell = P.b1n * P.b2n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // shared memory: [nw][SG*SG] complex subgrids, [nw][PB][2w] kernel weights,
  // then (if it fits) a private copy of the band.  nw = the warps that own a
  // subgrid (all of the CTA's when they fit), PB = points prepared per phase,
  // the largest of 32/16/8 that fits.
  const size_t dyn_b = (size_t)c.dyn_cpx * sizeof(cpx<R>);
  int nw = blockDim.x >> 5;
  while (nw > 1 && (size_t)nw * (SG * SG * sizeof(cpx<R>) + 8 * 2 * w * sizeof(R)) + 16 > dyn_b) --nw;
  const size_t sub_b = (size_t)nw * SG * SG * sizeof(cpx<R>);
  int PB = 32;
  while (PB > 8 && sub_b + (size_t)nw * PB * 2 * w * sizeof(R) > dyn_b) PB >>= 1;
  const size_t wt_b = ((size_t)nw * PB * 2 * w * sizeof(R) + 15) / 16 * 16;
  cpx<R>* sub = c.sbuf + (size_t)warp * SG * SG;
  R* wtab = reinterpret_cast<R*>(reinterpret_cast<char*>(c.sbuf) + sub_b) + (size_t)warp * PB * 2 * w;
  cpx<R>* sband = reinterpret_cast<cpx<R>*>(reinterpret_cast<char*>(c.sbuf) + sub_b + wt_b);
  const bool staged = sub_b + wt_b + (size_t)ncell * sizeof(cpx<R>) <= dyn_b;
  R* band = staged ? reinterpret_cast<R*>(sband) : gband;
  if (staged) {
    for (int i = threadIdx.x; i < ncell; i += blockDim.x) sband[i] = cmk<R>(0, 0);
    __syncthreads();
  }
  const int ra = lane % w, rb = lane / w;
  const int gw = g.rank * nw + warp, nwt = g.G * nw;
  for (int it = warp < nw ? gw : P.nitems; it < P.nitems; it += nwt) {
    const int4 item = items[it];
    for (int i = lane; i < SG * SG; i += 32) sub[i] = cmk<R>(0, 0);
    for (int jb = item.x; jb < item.y; jb += PB) {
      // phase 1: lanes < PB prepare one point each (value, cell, kernel weights)
      const int jl = jb + lane;
      R cre_l = 0, cim_l = 0;
      int cell_l = 0;
      if (lane < PB && jl < item.y) {
        const cpx<R> cj = cacc[jl];
        cre_l = cj.x;
        cim_l = cj.y;
        const R xi1 = xu[jl], xi2 = xv[jl];
        const int l1 = (int)ceil(xi1 - half), l2 = (int)ceil(xi2 - half);
        R* wr = wtab + lane * 2 * w;
        for (int q = 0; q < w; ++q) {
          wr[q] = es_kernel(((R)(l1 + q) - xi1) * inv, beta);
          wr[w + q] = es_kernel(((R)(l2 + q) - xi2) * inv, beta);
        }
        // position inside the subgrid (item.z, item.w = subgrid origin row, col)
        const int lr = imod(l2 - P.b2s, P.nf2) - item.z, lc = imod(l1 - P.b1s, P.nf1) - item.w;
        cell_l = lr * SG + lc;
      }
      __syncwarp();
      // phase 2: the lanes cover the taps of one point at a time
      const int np = min(PB, item.y - jb);
      for (int p = 0; p < np; ++p) {
        const R cre = __shfl_sync(0xffffffffu, cre_l, p);
        const R cim = -__shfl_sync(0xffffffffu, cim_l, p);  // c = Vresre - i Vresim
        const int cell0 = __shfl_sync(0xffffffffu, cell_l, p);
        const R* wr = wtab + p * 2 * w;
        int a = ra, b = rb;
        for (int t0 = 0; t0 < ww; t0 += 32) {
          if (t0 + lane < ww) {
            cpx<R>& cell = sub[cell0 + b * SG + a];
            const R wt = wr[a] * wr[w + b];
            cell.x += wt * cre;
            cell.y += wt * cim;
          }
          a += 32 % w;
          b += 32 / w;
          if (a >= w) {
            a -= w;
            b += 1;
          }
        }
        __syncwarp();
      }
    }
    // add the subgrid to the band (rows/cols wrap only for a full-grid band)
    for (int i = lane; i < SG * SG; i += 32) {
      const cpx<R> v = sub[i];
      if (v.x == (R)0 && v.y == (R)0) continue;
      int rw = item.z + i / SG, cl = item.w + i % SG;
      if (rw >= P.nf2) rw -= P.nf2;
      if (cl >= P.nf1) cl -= P.nf1;
      if (rw >= P.b2n || cl >= P.b1n) continue;  // beyond the band: only zero taps land here
      R* dst = band + 2 * ((size_t)rw * P.b1n + cl);
      atomic_add_r(dst, v.x);
      atomic_add_r(dst + 1, v.y);
    }
    __syncwarp();
  }
  if (staged) {
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * ncell; i += blockDim.x) {
      const R vv = band[i];
      if (vv != (R)0) atomic_add_r(gband + i, vv);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// F6: type-1 row pass over band rows -> tmpC[b2][ix] (modes along axis 1)
// ---------------------------------------------------------------------------
template <typename R>
__device__ __noinline__ void fg_t1_rows(FgCtx<R>& c, const GroupCtx& g) {
  const ProbDesc& P = *c.P;
  const cpx<R>* tw1 = at<cpx<R>>(c.base, P.o_tw1);
  const cpx<R>* bandC = at<cpx<R>>(c.base, P.o_bandC);
  cpx<R>* tmpC = at<cpx<R>>(c.base, P.o_tmpC);
  const int n1 = P.nf1, nx = P.nx, b1n = P.b1n;
  const FftPlan pl = make_plan(n1);
  const int S = min(fft_batch(n1), c.smem_cpx / n1);
  for (int r0 = g.rank * S; r0 < P.b2n; r0 += g.G * S) {
    const int rows = min(S, P.b2n - r0);
    for (int i = threadIdx.x; i < rows * n1; i += blockDim.x) c.sbuf[i] = cmk<R>(0, 0);
    __syncthreads();
    for (int i = threadIdx.x; i < rows * b1n; i += blockDim.x) {
      const int s = i / b1n, b = i - s * b1n;
      c.sbuf[s * n1 + wrapn(P.b1s + b, n1)] = bandC[(size_t)(r0 + s) * b1n + b];
    }
    __syncthreads();
    const cpx<R>* out = smem_fft(c.sbuf, c.swork, pl, rows, tw1);
    for (int i = threadIdx.x; i < rows * nx; i += blockDim.x) {
      const int s = i / nx, ix = i - s * nx;
      tmpC[(size_t)(r0 + s) * nx + ix] = out[s * n1 + wrapn(ix - nx / 2, n1)];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// F7: type-1 column pass -> gchi[iy][ix] = Re(F) * dc1 * dc2
// ---------------------------------------------------------------------------
template <typename R>
__device__ __noinline__ void fg_t1_cols(FgCtx<R>& c, const GroupCtx& g) {
  if (c.P->dft) {
    if ((c.P->nx + g.G - 1) / g.G <= 16) dft_adjoint<16, 4>(c, g);
    else dft_adjoint<64, 16>(c, g);
    return;
  }
  const ProbDesc& P = *c.P;
  const cpx<R>* tw2 = at<cpx<R>>(c.base, P.o_tw2);
  const cpx<R>* tmpC = at<cpx<R>>(c.base, P.o_tmpC);
  const double* dc1 = at<double>(c.base, P.o_dc1);
  const double* dc2 = at<double>(c.base, P.o_dc2);
  double* gchi = at<double>(c.base, P.o_gchi);
  const int n2 = P.nf2, nx = P.nx, ny = P.ny;
  const FftPlan pl = make_plan(n2);
  const int S = min(fft_batch(n2), c.smem_cpx / n2);
  for (int x0 = g.rank * S; x0 < nx; x0 += g.G * S) {
    const int cols = min(S, nx - x0);
    for (int i = threadIdx.x; i < cols * n2; i += blockDim.x) c.sbuf[i] = cmk<R>(0, 0);
    __syncthreads();
    for (int i = threadIdx.x; i < cols * P.b2n; i += blockDim.x) {
      const int b2 = i / cols, s = i - b2 * cols;
      c.sbuf[s * n2 + wrapn(P.b2s + b2, n2)] = tmpC[(size_t)b2 * nx + x0 + s];
    }
    __syncthreads();
    const cpx<R>* out = smem_fft(c.sbuf, c.swork, pl, cols, tw2);
    for (int i = threadIdx.x; i < cols * ny; i += blockDim.x) {
      const int iy = i / cols, s = i - iy * cols, ix = x0 + s;
      gchi[(size_t)iy * nx + ix] = (double)out[s * n2 + wrapn(iy - ny / 2, n2)].x * dc1[ix] * dc2[iy];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// F8: regularizers + gradient assembly g = gradchisq + gradreg.
// reg[0..7] = l1, tv, tsv, kl, gs, tfd, cen, sm.  Also returns g.d and the
// projected-gradient infinity norm used by the optimiser.
// mom: reduced image moments from F1 (only when tfd/cen/sm are active).
// ---------------------------------------------------------------------------
// Image value at grid cell (ix, iy), 0 outside the image or at a pixel the
// solve does not include: through the pixel map (PxMap) or from the dense
// image grid that the type-2 row pass writes (PxGrid).
struct PxMap {
  const double* x;
  const int* inv;
  int nx, ny;
  __device__ __forceinline__ double operator()(int ix, int iy) const {
    if (ix < 0 || iy < 0 || ix >= nx || iy >= ny) return 0.0;
    const int p = inv[iy * nx + ix];
    return p >= 0 ? x[p] : 0.0;
  }
};
struct PxGrid {
  const double* xg;
  int nx, ny;
  __device__ __forceinline__ double operator()(int ix, int iy) const {
    if (ix < 0 || iy < 0 || ix >= nx || iy >= ny) return 0.0;
    return xg[(size_t)iy * nx + ix];
  }
};
// TV gradient (image.f90:512-612) at pixel (i1, j1) from preloaded values,
// reproducing the gradient reset: I11 = I(i1, j1), xp = I(i1+1, j1),
// yp = I(i1, j1+1), xm = I(i1-1, j1), ym = I(i1, j1-1), xmyp = I(i1-1, j1+1),
// xpym = I(i1+1, j1-1); the has_* flags say which neighbours lie inside the
// image (a value outside is never read).
template <typename T>
__device__ __forceinline__ T tv_grade_vals(T I11, T xp, T yp, T xm, T ym, T xmyp, T xpym, bool has_xp,
                                           bool has_yp, bool has_xm, bool has_ym) {
  T gr = 0;
  T dIx = has_xp ? xp - I11 : (T)0;
  T dIy = has_yp ? yp - I11 : (T)0;
  T e = sqrt(dIx * dIx + dIy * dIy);
  if (e > (T)1e-10) gr -= (dIx + dIy) / e;
  if (has_xm) {
    dIx = I11 - xm;
    dIy = has_yp ? xmyp - xm : (T)0;
    e = sqrt(dIx * dIx + dIy * dIy);
    if (e > (T)1e-10) gr += dIx / e;
    else gr = 0;
  }
  if (has_ym) {
    dIy = I11 - ym;
    dIx = has_xp ? xpym - ym : (T)0;
    e = sqrt(dIx * dIx + dIy * dIy);
    if (e > (T)1e-10) gr += dIy / e;
    else gr = 0;
  }
  return gr;
}
struct RegMoments {
  double Isum_abs, xcen, ycen, Sg[3], mom[2], Sp[3];
  double tfd_resid;
  double cen_sx, cen_sy, cen_sI, cen_cost;
};

__device__ void reg_moments(const ProbDesc& P, const double (&m)[10], RegMoments& r) {
  r.tfd_resid = m[0] - P.tfd_tgtfd;
  r.Isum_abs = m[1];
  r.xcen = m[2] / m[1];
  r.ycen = m[3] / m[1];
  const double S = m[0];
  // second moments about the |I|-normalised centroid from raw moments
  r.Sg[0] = (m[4] - 2 * r.xcen * m[2] + r.xcen * r.xcen * S) / r.Isum_abs;
  r.Sg[1] = (m[5] - 2 * r.ycen * m[3] + r.ycen * r.ycen * S) / r.Isum_abs;
  r.Sg[2] = (m[6] - r.xcen * m[3] - r.ycen * m[2] + r.xcen * r.ycen * S) / r.Isum_abs;
  r.mom[0] = m[2] - r.xcen * S;
  r.mom[1] = m[3] - r.ycen * S;
  const double cp = cos(P.sm_phi), sp = sin(P.sm_phi);
  r.Sp[0] = P.sm_min * cp * cp + P.sm_maj * sp * sp;
  r.Sp[1] = P.sm_min * sp * sp + P.sm_maj * cp * cp;
  r.Sp[2] = (P.sm_maj - P.sm_min) * sp * cp;
  r.cen_sI = m[9] + 1e-10;
  r.cen_sx = m[7] / r.cen_sI;
  r.cen_sy = m[8] / r.cen_sI;
  r.cen_cost = sqrt(r.cen_sx * r.cen_sx + r.cen_sy * r.cen_sy + 1e-10);
}

// image moments of a movie frame that has no data (the row pass of F1
// accumulates the same sums for frames with data): per-thread partials over
// this CTA's pixels lo..hi
__device__ void frame_moments(const ProbDesc& P, char* base, int lo, int hi, double (&mom)[10]) {
  const double* x = at<double>(base, P.o_x);
  const int* xi = at<int>(base, P.o_xidx);
  const int* yi = at<int>(base, P.o_yidx);
  for (int p = lo + threadIdx.x; p < hi; p += blockDim.x) {
    const double val = x[p], fx = xi[p] + 1, fy = yi[p] + 1;
    mom[0] += val;
    mom[1] += fabs(val);
    mom[2] += val * fx;
    mom[3] += val * fy;
    mom[4] += val * fx * fx;
    mom[5] += val * fy * fy;
    mom[6] += val * fx * fy;
  }
}

// log in the compute type of the regularizer stage
__device__ __forceinline__ double reg_log(double x) { return log(x); }
__device__ __forceinline__ float reg_log(float x) { return logf(x); }

// Per-pixel regularizer terms in the compute type T (float in the FP32 mode):
// L1, TV, TSV, MEM (kl) and the Gaussian-prior entropy (gs).  The moment
// terms (total flux, centroid, second moment) use differences of image-wide
// sums and stay in FP64; so do the regularizer sums, the gradient that the
// optimiser reads and g.d.
template <typename T, class PX>
__device__ void reg_grad_loop(const ProbDesc& P, char* base, const PX& px, const RegMoments& rm, int lo, int hi,
                              double (&reg)[8], double& gd, double& sbg, bool opt_terms) {
  const double* x = at<double>(base, P.o_x);
  const int* xi = at<int>(base, P.o_xidx);
  const int* yi = at<int>(base, P.o_yidx);
  const double* gchi = at<double>(base, P.o_gchi);
  const double* d = at<double>(base, P.o_d);
  double* gout = at<double>(base, P.o_g);
  // a weight array is read only when its weights differ between pixels;
  // otherwise its one value (wu) is used
  const double* l1w = (P.has_l1 && !(P.wuni & 1)) ? at<double>(base, P.o_l1w) : nullptr;
  const double* tvw = (P.has_tv && !(P.wuni & 2)) ? at<double>(base, P.o_tvw) : nullptr;
  const double* tsvw = (P.has_tsv && !(P.wuni & 4)) ? at<double>(base, P.o_tsvw) : nullptr;
  const double* klw = (P.has_kl && !(P.wuni & 8)) ? at<double>(base, P.o_klw) : nullptr;
  const double* gsw = (P.has_gs && !(P.wuni & 16)) ? at<double>(base, P.o_gsw) : nullptr;
  const int nx = P.nx, ny = P.ny;
  const T l1_l = (T)P.l1_l, tv_l = (T)P.tv_l, tsv_l = (T)P.tsv_l, kl_l = (T)P.kl_l, gs_l = (T)P.gs_l;
  const double g_tfd = P.has_tfd ? P.tfd_l * 2 * rm.tfd_resid : 0.0;
  // running sums in registers (the caller's accumulators are written once
  // at the end, so the stores of the loop cannot alias them)
  double r0 = reg[0], r1 = reg[1], r2 = reg[2], r3 = reg[3], r4 = reg[4], gdl = gd, sbgl = sbg;
  const bool nb = P.has_tv || P.has_tsv;
  const bool ident = P.ident;
  for (int p = lo + threadIdx.x; p < hi; p += blockDim.x) {
    // every load of the iteration first (two dependent rounds: the pixel's
    // indices, then its grid cell and neighbours), so that the arithmetic
    // below waits once per round and not once per term
    int ix, iy;
    if (ident) {  // row-major full grid: no index loads, so one round of loads below
      iy = p / nx;
      ix = p - iy * nx;
    } else {
      ix = xi[p];
      iy = yi[p];
    }
    const double I = x[p];
    const double w_l1 = l1w ? l1w[p] : P.wu[0], w_kl = klw ? klw[p] : P.wu[3], w_gs = gsw ? gsw[p] : P.wu[4];
    const double w_tv = tvw ? tvw[p] : P.wu[1], w_tsv = tsvw ? tsvw[p] : P.wu[2];
    const double dp = opt_terms ? d[p] : 0.0;
    const bool hxp = ix + 1 < nx, hyp = iy + 1 < ny, hxm = ix - 1 >= 0, hym = iy - 1 >= 0;
    const double gc = gchi[(size_t)iy * nx + ix];
    double vxp = 0, vyp = 0, vxm = 0, vym = 0, vxmyp = 0, vxpym = 0;
    if (nb) {
      vxp = hxp ? px(ix + 1, iy) : 0.0;
      vyp = hyp ? px(ix, iy + 1) : 0.0;
      vxm = hxm ? px(ix - 1, iy) : 0.0;
      vym = hym ? px(ix, iy - 1) : 0.0;
      if (P.has_tv) {
        vxmyp = (hxm && hyp) ? px(ix - 1, iy + 1) : 0.0;
        vxpym = (hxp && hym) ? px(ix + 1, iy - 1) : 0.0;
      }
    }
    const T It = (T)I;
    // each term is added to one FP64 sum, in the order of image.f90's
    // gradient: total flux, centroid, l1, MEM, gs, TV, TSV, second moment
    double gr = g_tfd;
    if (P.has_cen) {
      const double dix = (ix + 1) - P.nxref, diy = (iy + 1) - P.nyref;
      const double gIp = fabs(P.cen_alpha - 1) < 1e-10
                             ? I / smabs(I)
                             : I / smabs(I) * P.cen_alpha * pow(smabs(I), P.cen_alpha - 1);
      gr += P.cen_l * ((rm.cen_sx * (dix - rm.cen_sx) + rm.cen_sy * (diy - rm.cen_sy)) / rm.cen_sI /
                       rm.cen_cost * gIp);
    }
    if (P.has_l1) {
      const T a = smabs(It), w = l1_l * (T)w_l1;
      r0 += (double)(w * a);
      gr += (double)(w * (It / a));
    }
    if (P.has_kl) {
      const T a = smabs(It), pr = (T)w_kl, lr = reg_log(a / pr);
      r3 += (double)(kl_l * (a * lr + pr / (T)2.718281828459045235));
      gr += (double)(kl_l * (It / a) * (lr + 1));
    }
    if (P.has_gs) {
      const T a = smabs(It), pr = (T)w_gs, lr = reg_log(a / pr);
      r4 += (double)(gs_l * (a * (lr - 1) + pr));
      gr += (double)(gs_l * (It / a) * lr);
    }
    if (nb) {
      const T txp = (T)vxp, typ = (T)vyp, txm = (T)vxm, tym = (T)vym;
      const T dIx = hxp ? txp - It : (T)0;
      const T dIy = hyp ? typ - It : (T)0;
      if (P.has_tv) {
        const T w = tv_l * (T)w_tv;
        r1 += (double)(w * sqrt(dIx * dIx + dIy * dIy));
        gr += (double)(w * tv_grade_vals<T>(It, txp, typ, txm, tym, (T)vxmyp, (T)vxpym, hxp, hyp, hxm, hym));
      }
      if (P.has_tsv) {
        const T w = tsv_l * (T)w_tsv;
        r2 += (double)(w * (dIx * dIx + dIy * dIy));
        T gt = 0;
        if (hxp) gt -= 2 * (txp - It);
        if (hyp) gt -= 2 * (typ - It);
        if (hxm) gt += 2 * (It - txm);
        if (hym) gt += 2 * (It - tym);
        gr += (double)(w * gt);
      }
    }
    if (P.has_sm) {
      const double fx = ix + 1, fy = iy + 1;
      const double xg = (fx - rm.xcen) / rm.Isum_abs, yg = (fy - rm.ycen) / rm.Isum_abs;
      const double dx = fx - rm.xcen, dy = fy - rm.ycen;
      const double s0 = ((dx * dx - 2. * xg * rm.mom[0]) - rm.Sg[0]) / rm.Isum_abs;
      const double s1 = ((dy * dy - 2. * yg * rm.mom[1]) - rm.Sg[1]) / rm.Isum_abs;
      const double s2 = (dx * dy - xg * rm.mom[1] - yg * rm.mom[0] - rm.Sg[2]) / rm.Isum_abs;
      gr += P.sm_l * (2. * (rm.Sg[0] - rm.Sp[0]) * s0 + 2. * (rm.Sg[1] - rm.Sp[1]) * s1 +
                      4. * (rm.Sg[2] - rm.Sp[2]) * s2);
    }
    const double gv = gc + gr;
    gout[p] = gv;
    if (!opt_terms) continue;  // a movie frame: the movie pass forms g.d and the projected gradient
    gdl += gv * dp;
    // projected gradient (projgr, lbfgsb.f:2942-2990) with lower bound 0
    double gi = gv;
    if (P.nonneg && gi >= 0.0) gi = fmin(I, gi);
    sbgl = fmax(sbgl, fabs(gi));
  }
  reg[0] = r0;
  reg[1] = r1;
  reg[2] = r2;
  reg[3] = r3;
  reg[4] = r4;
  gd = gdl;
  sbg = sbgl;
}

// F8: regularizer values and the full gradient g = grad chi2 + grad reg over
// pixels [lo, hi); neighbours come from the dense image grid when F1 wrote
// it in this evaluation (frames without data use the pixel map).
template <typename T>
__device__ __noinline__ void fg_reg_grad(const ProbDesc& P, char* base, const GroupCtx& g, const RegMoments& rm,
                            int lo, int hi, double (&reg)[8], double& gd, double& sbg,
                            bool opt_terms = true) {
  if (P.ident || (P.nuv > 0 && P.o_xg)) {
    // the dense grid: x itself on a row-major full grid, else the copy F1 wrote
    const PxGrid px{at<double>(base, P.ident ? P.o_x : P.o_xg), P.nx, P.ny};
    reg_grad_loop<T>(P, base, px, rm, lo, hi, reg, gd, sbg, opt_terms);
  } else {
    const PxMap px{at<double>(base, P.o_x), at<int>(base, P.o_inv), P.nx, P.ny};
    reg_grad_loop<T>(P, base, px, rm, lo, hi, reg, gd, sbg, opt_terms);
  }
}
