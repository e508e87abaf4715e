// Device-resident L-BFGS-B (version 3.0), restating src/lbfgsb/lbfgsb.f.
//
// The CTAs of a group run the algorithm SPMD: vector work (length n) is split
// into one contiguous chunk per CTA; every reduction goes through
// group_reduce, whose result is bit-identical in every CTA, so each CTA keeps
// its own copy of the scalar state (LbState in shared memory, updated by
// thread 0) and all CTAs take the same branches without a broadcast.
//
// Differences from the sequential Fortran that only change rounding:
//  * dot products and norms are parallel reductions;
//  * formk builds the 2m x 2m matrix from Gram sums over the current free /
//    active sets instead of updating it with entering / leaving variables
//    (same matrix in exact arithmetic, lbfgsb.f:1848-2172);
//  * the generalized Cauchy point (cauchy, lbfgsb.f:1222-1719) visits the
//    breakpoints in increasing (t, index) order, bucketed and then sorted by
//    the CTAs of the group, and evaluates the piecewise quadratic in closed
//    form from prefix sums (D_k = sum d^2 over moving variables, P_k = W'd_k,
//    Q_k = sum t_i d_i w_i), instead of popping a heap and updating f1, f2
//    incrementally.  The f2 safeguard max(eps*f2_org, f2) is applied per
//    segment.  Ties between equal breakpoints are visited in index order.
// Only the bounds SMILI uses are supported: all variables unbounded
// (nbd = 0) or all bounded below by zero (nbd = 1, l = 0).
#pragma once
#include <cfloat>

#include "common.cuh"
#include "quotient.cuh"

#define SMILI_MAXM_DEV 6  // largest L-BFGS-B memory the device solver accepts
#define SMILI_KC 1024     // breakpoints of one sorted batch of the Cauchy search

typedef unsigned __int128 u128;

// SY: the storage type of the limited-memory matrices S and Y (double in the
// FP64 mode, float in the FP32 mode); every dot product over them
// accumulates in FP64.
template <typename SY>
struct LbCtxT {
  const ProbDesc* P;
  char* base;
  GroupCtx* g;
  LbState* S;  // shared
  int n, m, lo, hi;
  double *x, *gv, *z, *r, *d, *t, *xp;
  SY *ws, *wy;
  signed char* iwh;
  unsigned char* freef;
  unsigned long long* bkey;
  double* trace;
  double* red;    // shared [SMILI_REDK]
  double* scratch;  // shared, SMILI_SCRATCH(blockDim.x) doubles (group_reduce)
  char* dyn;      // shared scratch (the FFT buffers)
  Prof* prof;
};

// S and Y element i (column-major, n per column), widened to FP64
template <typename SY>
__device__ __forceinline__ double ld_ws(const LbCtxT<SY>& c, size_t i) { return (double)c.ws[i]; }
template <typename SY>
__device__ __forceinline__ double ld_wy(const LbCtxT<SY>& c, size_t i) { return (double)c.wy[i]; }
template <typename SY>
__device__ __forceinline__ void st_sy(const LbCtxT<SY>& c, size_t i, double s, double y) {
  c.ws[i] = (SY)s;
  c.wy[i] = (SY)y;
}

// ---------------------------------------------------------------------------
// small dense algebra, by one warp: an element or a row per lane, loops kept
// rolled.  Bound by latency: of dependent FP64 operations, of the divisions
// (avoided where the divisor is a known diagonal) and of fetching instructions,
// as this code runs once per iteration and the stages between push it out of
// the instruction cache.  Per call at m = 5, one thread in the reference's
// loops / a column per lane, unrolled / as here: formk 22 / 13 / 8 us, the
// two solves of subsm 9 / 7 / 2.8, an update 9 / 6 / 5 (B200).
// ---------------------------------------------------------------------------
// Cholesky factor of the symmetric matrix in the upper triangle of a (shared,
// column major, leading dimension ld).  The first n1 columns eliminate with
// the opposite sign beyond row n1: [A B; B' C] becomes the factors of A and of
// C + B' A^-1 B (formk's LEL' with E = diag(-I, I)); n1 = nn is the plain
// factor.  The square roots are taken at the end, off the chain of pivots.
// rdiag receives the reciprocals of the factor's diagonal.  One warp; returns
// 0, -1 or -2 (a pivot of the first or second block is not positive), in every
// lane.
__device__ __noinline__ int warp_factor(double* a, int ld, int nn, int n1, double* rdiag) {
  const int lane = threadIdx.x & 31;
  // lanes 0..15 and 16..31: two halves of the rows of column lane & 15
  const int j = lane & 15, half = lane >> 4;
#pragma unroll 1
  for (int k = 0; k < nn; ++k) {
    const double d = a[k + ld * k];
    if (d <= 0.0) return k < n1 ? -1 : -2;
    const double u = j > k && j < nn ? a[k + ld * j] / d : 0.0;
    if (j < nn) {
#pragma unroll 1
      for (int i = k + 1 + half; i <= j; i += 2) {
        const double p = a[k + ld * i] * u;
        a[i + ld * j] += k < n1 && i >= n1 ? p : -p;
      }
    }
    __syncwarp();
  }
  const double sq = lane < nn ? sqrt(a[lane + ld * lane]) : 1.0, r = rcp_of(sq);
  __syncwarp();
#pragma unroll 1
  for (int k = 0; k < nn; ++k) {
    const double sk = __shfl_sync(0xffffffffu, sq, k), rk = __shfl_sync(0xffffffffu, r, k);
    if (lane >= k && lane < nn) a[k + ld * lane] = lane == k ? sq : div_by(a[k + ld * lane], sk, rk);
  }
  if (lane < nn) rdiag[lane] = r;
  __syncwarp();
  return 0;
}

// x of R' x = b (trans) or R x = b, R the upper triangle of a as warp_factor
// leaves it: lane i holds b_i and returns x_i.  ok: false in every lane when a
// diagonal element is zero.
__device__ __forceinline__ double warp_tri_solve(const double* a, int ld, int nn, const double* rdiag, double b,
                                                 bool trans, bool& ok) {
  const int lane = threadIdx.x & 31;
  const bool in = lane < nn;
  const double dg = in ? a[lane + ld * lane] : 1.0, rd = in ? rdiag[lane] : 1.0;
  ok = !__any_sync(0xffffffffu, dg == 0.0);
#pragma unroll 1
  for (int s = 0; s < nn; ++s) {
    const int j = trans ? s : nn - 1 - s;
    if (lane == j) b = div_by(b, dg, rd);
    const double xj = __shfl_sync(0xffffffffu, b, j);
    if (in && (trans ? lane > j : lane < j)) b -= a[trans ? j + ld * lane : lane + ld * j] * xj;
  }
  return b;
}

// Product with the 2col x 2col middle matrix (bmv, lbfgsb.f:1106-1220): lane i
// < col holds (vy_i, vs_i) and gets (M v)_i and (M v)_{col + i} there.  One
// warp; false for a singular factor.
__device__ __noinline__ bool warp_bmv(const LbState& S, int m, int col, double& vy, double& vs) {
  const int lane = threadIdx.x & 31;
  const bool in = lane < col;
  double p = vs;
#pragma unroll 1
  for (int k = 0; k < col - 1; ++k) {
    const double vk = __shfl_sync(0xffffffffu, vy, k);
    if (in && lane > k) p += S.lt[lane + m * k] * vk;
  }
  bool ok, ok2;
  p = warp_tri_solve(S.wt, m, col, S.rwt, p, true, ok);
  p = warp_tri_solve(S.wt, m, col, S.rwt, p, false, ok2);
  const double sq = in ? S.sq[lane] : 1.0, rsq = in ? S.rsq[lane] : 1.0;
  double q = -div_by(div_by(vy, sq, rsq), sq, rsq);
#pragma unroll 1
  for (int k = 1; k < col; ++k) {
    const double pk = __shfl_sync(0xffffffffu, p, k);
    if (lane < k) q += S.lt[k + m * lane] * pk;
  }
  vy = q;
  vs = p;
  return ok;
}

// T = theta S'S + L D^-1 L' and its factor (formt, lbfgsb.f:2173-2240), with
// the quotients and roots that warp_bmv reads.  One warp; returns nonzero in
// every lane when T is not positive definite.
__device__ __noinline__ int warp_formt(LbState& S, int m) {
  const int col = S.col, lane = threadIdx.x & 31;
#define SY(i, j) S.sy[(i) + m * (j)]
#pragma unroll 1
  for (int e = lane; e < col * col; e += 32) {
    const int i = e % col, k = e / col;
    if (i > k) S.lt[i + m * k] = SY(i, k) / SY(k, k);
  }
  if (lane < col) {
    const double sq = sqrt(SY(lane, lane));
    S.sq[lane] = sq;
    S.rsq[lane] = rcp_of(sq);
  }
  __syncwarp();
#pragma unroll 1
  for (int e = lane; e < col * col; e += 32) {
    const int i = e % col, j = e / col;
    if (i > j) continue;
    double dd = 0.0;
#pragma unroll 1
    for (int k = 0; k < i; ++k) dd += SY(i, k) * S.lt[j + m * k];
    S.wt[i + m * j] = dd + S.theta * S.ss[i + m * j];
  }
#undef SY
  __syncwarp();
  return warp_factor(S.wt, m, col, col, S.rwt);
}

__device__ void d_dcstep(double& stx, double& fx, double& dx, double& sty, double& fy, double& dy,
                         double& stp, double fp, double dp, int& brackt, double stpmin,
                         double stpmax) {  // lbfgsb.f:3694-3949
  const double sgnd = dp * (dx / fabs(dx));
  double stpf, stpc, stpq;
  if (fp > fx) {
    const double th = 3.0 * (fx - fp) / (stp - stx) + dx + dp;
    const double s = fmax(fabs(th), fmax(fabs(dx), fabs(dp)));
    double gam = s * sqrt((th / s) * (th / s) - (dx / s) * (dp / s));
    if (stp < stx) gam = -gam;
    const double p = (gam - dx) + th, q = ((gam - dx) + gam) + dp, rr = p / q;
    stpc = stx + rr * (stp - stx);
    stpq = stx + ((dx / ((fx - fp) / (stp - stx) + dx)) / 2.0) * (stp - stx);
    stpf = (fabs(stpc - stx) < fabs(stpq - stx)) ? stpc : stpc + (stpq - stpc) / 2.0;
    brackt = 1;
  } else if (sgnd < 0.0) {
    const double th = 3.0 * (fx - fp) / (stp - stx) + dx + dp;
    const double s = fmax(fabs(th), fmax(fabs(dx), fabs(dp)));
    double gam = s * sqrt((th / s) * (th / s) - (dx / s) * (dp / s));
    if (stp > stx) gam = -gam;
    const double p = (gam - dp) + th, q = ((gam - dp) + gam) + dx, rr = p / q;
    stpc = stp + rr * (stx - stp);
    stpq = stp + (dp / (dp - dx)) * (stx - stp);
    stpf = (fabs(stpc - stp) > fabs(stpq - stp)) ? stpc : stpq;
    brackt = 1;
  } else if (fabs(dp) < fabs(dx)) {
    const double th = 3.0 * (fx - fp) / (stp - stx) + dx + dp;
    const double s = fmax(fabs(th), fmax(fabs(dx), fabs(dp)));
    double gam = s * sqrt(fmax(0.0, (th / s) * (th / s) - (dx / s) * (dp / s)));
    if (stp > stx) gam = -gam;
    const double p = (gam - dp) + th, q = (gam + (dx - dp)) + gam, rr = p / q;
    if (rr < 0.0 && gam != 0.0) stpc = stp + rr * (stx - stp);
    else if (stp > stx) stpc = stpmax;
    else stpc = stpmin;
    stpq = stp + (dp / (dp - dx)) * (stx - stp);
    if (brackt) {
      stpf = (fabs(stpc - stp) < fabs(stpq - stp)) ? stpc : stpq;
      stpf = (stp > stx) ? fmin(stp + 0.66 * (sty - stp), stpf) : fmax(stp + 0.66 * (sty - stp), stpf);
    } else {
      stpf = (fabs(stpc - stp) > fabs(stpq - stp)) ? stpc : stpq;
      stpf = fmin(stpmax, stpf);
      stpf = fmax(stpmin, stpf);
    }
  } else {
    if (brackt) {
      const double th = 3.0 * (fp - fy) / (sty - stp) + dy + dp;
      const double s = fmax(fabs(th), fmax(fabs(dy), fabs(dp)));
      double gam = s * sqrt((th / s) * (th / s) - (dy / s) * (dp / s));
      if (stp > sty) gam = -gam;
      const double p = (gam - dp) + th, q = ((gam - dp) + gam) + dy, rr = p / q;
      stpc = stp + rr * (sty - stp);
      stpf = stpc;
    } else {
      stpf = (stp > stx) ? stpmax : stpmin;
    }
  }
  if (fp > fx) {
    sty = stp;
    fy = fp;
    dy = dp;
  } else {
    if (sgnd < 0.0) {
      sty = stx;
      fy = fx;
      dy = dx;
    }
    stx = stp;
    fx = fp;
    dx = dp;
  }
  stp = stpf;
}

enum { CS_START = 0, CS_FG = 1, CS_CONV = 2, CS_WARN = 3, CS_ERROR = 4 };

__device__ void d_dcsrch(LbState& S, double f, double g, double stpmin, double stpmax) {
  const double ftol = 1e-3, gtol = 0.9, xtol = 0.1;  // lnsrlb parameters (lbfgsb.f:2497)
  if (S.csave == CS_START) {
    if (S.stp < stpmin || S.stp > stpmax || g >= 0.0 || stpmax < stpmin) {
      S.csave = CS_ERROR;
      return;
    }
    S.brackt = 0;
    S.stage = 1;
    S.finit = f;
    S.ginit = g;
    S.gtest = ftol * S.ginit;
    S.width = stpmax - stpmin;
    S.width1 = S.width / 0.5;
    S.stx = 0.0;
    S.fx = S.finit;
    S.gx = S.ginit;
    S.sty = 0.0;
    S.fy = S.finit;
    S.gy = S.ginit;
    S.stmin = 0.0;
    S.stmax = S.stp + 4.0 * S.stp;
    S.csave = CS_FG;
    return;
  }
  const double ftest = S.finit + S.stp * S.gtest;
  if (S.stage == 1 && f <= ftest && g >= 0.0) S.stage = 2;
  int task = CS_FG;
  if (S.brackt && (S.stp <= S.stmin || S.stp >= S.stmax)) task = CS_WARN;
  if (S.brackt && S.stmax - S.stmin <= xtol * S.stmax) task = CS_WARN;
  if (S.stp == stpmax && f <= ftest && g <= S.gtest) task = CS_WARN;
  if (S.stp == stpmin && (f > ftest || g >= S.gtest)) task = CS_WARN;
  if (f <= ftest && fabs(g) <= gtol * (-S.ginit)) task = CS_CONV;
  if (task == CS_WARN || task == CS_CONV) {
    S.csave = task;
    return;
  }
  if (S.stage == 1 && f <= S.fx && f > ftest) {
    double fm = f - S.stp * S.gtest, fxm = S.fx - S.stx * S.gtest, fym = S.fy - S.sty * S.gtest;
    double gm = g - S.gtest, gxm = S.gx - S.gtest, gym = S.gy - S.gtest;
    d_dcstep(S.stx, fxm, gxm, S.sty, fym, gym, S.stp, fm, gm, S.brackt, S.stmin, S.stmax);
    S.fx = fxm + S.stx * S.gtest;
    S.fy = fym + S.sty * S.gtest;
    S.gx = gxm + S.gtest;
    S.gy = gym + S.gtest;
  } else {
    d_dcstep(S.stx, S.fx, S.gx, S.sty, S.fy, S.gy, S.stp, f, g, S.brackt, S.stmin, S.stmax);
  }
  if (S.brackt) {
    if (fabs(S.sty - S.stx) >= 0.66 * S.width1) S.stp = S.stx + 0.5 * (S.sty - S.stx);
    S.width1 = S.width;
    S.width = fabs(S.sty - S.stx);
  }
  if (S.brackt) {
    S.stmin = fmin(S.stx, S.sty);
    S.stmax = fmax(S.stx, S.sty);
  } else {
    S.stmin = S.stp + 1.1 * (S.stp - S.stx);
    S.stmax = S.stp + 4.0 * (S.stp - S.stx);
  }
  S.stp = fmax(S.stp, stpmin);
  S.stp = fmin(S.stp, stpmax);
  if ((S.brackt && (S.stp <= S.stmin || S.stp >= S.stmax)) ||
      (S.brackt && S.stmax - S.stmin <= xtol * S.stmax))
    S.stp = S.stx;
  S.csave = CS_FG;
}

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ int lptr(const LbState& S, int m, int j) {  // logical j (0-based) -> column
  return (S.head - 1 + j) % m;
}

__device__ __forceinline__ void reset_memory(LbState& S) {
  S.info = 0;
  S.col = 0;
  S.head = 1;
  S.theta = 1.0;
  S.iupdat = 0;
  S.updatd = 0;
}

// Group-wide sums of s and maxima of x into c.red (sums first).
template <int NS, int NX, typename SY>
__device__ __forceinline__ bool lb_reduce(LbCtxT<SY>& c, double (&s)[NS], const double (&x)[NX]) {
  return group_reduce(*c.g, s, NS, x, NX, c.red, c.scratch);
}

// ---------------------------------------------------------------------------
// init: active() projection and state (lbfgsb.f:1004-1104, mainlb START)
// ---------------------------------------------------------------------------
template <typename SY>
__device__ void lb_init(LbCtxT<SY>& c, const double* x0) {
  LbState& S = *c.S;
  const ProbDesc& P = *c.P;
  if (threadIdx.x == 0) {
    S.task = LB_TASK_FG_START;
    S.done = 0;
    S.error = 0;
    S.col = 0;
    S.head = 1;
    S.itail = 0;
    S.iupdat = 0;
    S.iter = 0;
    S.nfgv = 0;
    S.ifun = 0;
    S.iback = 0;
    S.nseg = 0;
    S.nskip = 0;
    S.nintol = 0;
    S.info = 0;
    S.iword = 0;
    S.nfree = c.n;
    S.nact = 0;
    S.ileave = 0;
    S.nenter = 0;
    S.updatd = 0;
    S.wrk = 0;
    S.cnstnd = P.nonneg ? 1 : 0;
    S.boxed = 0;
    S.prjctd = 0;
    S.stage = 1;
    S.brackt = 0;
    S.csave = CS_START;
    S.nfg_total = 0;
    S.f = 0;
    S.theta = 1.0;
    S.fold = 0;
    S.epsmch = DBL_EPSILON;
    S.tol = P.factr * S.epsmch;
    S.dnorm = S.gd = S.stpmx = S.sbgnrm = S.stp = S.gdold = S.dtd = S.xstep = 0;
  }
  for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) {
    double v = x0[i];
    if (P.nonneg && v < 0.0) v = 0.0;
    c.x[i] = v;
    c.iwh[i] = P.nonneg ? 0 : -1;
    c.freef[i] = 1;
    c.d[i] = 0.0;
    for (int j = 0; j < c.m; ++j) st_sy(c, (size_t)j * c.n + i, 0.0, 0.0);
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Cauchy point
// ---------------------------------------------------------------------------
// result of the search
enum {
  CR_INFO = 0, CR_MODE, CR_TSUM, CR_NSEG, CR_BHI, CR_BLO, CR_C  // CR_C.. 6 + 6 values of c (Y and S part)
};
enum { CM_NONE_FIXED = 0, CM_BOUNDARY = 1, CM_XCP_IS_X = 2 };

__device__ __forceinline__ u128 comp_key(unsigned long long key, int idx) {
  return ((u128)key << 32) | (u128)(unsigned)idx;
}

// Breakpoint buckets.  Keys are the IEEE bits of the breakpoint times t > 0,
// which order like the times; bucket = (key - kmin) >> shift, the outermost
// buckets taking what lies outside.  2048 buckets, or 4096 for more than
// 131 072 variables, so that the crowded ones stay near a CTA's sort.
#define SMILI_NBUCKET_MAX 4096
__device__ __forceinline__ int cauchy_buckets(int n) { return n > 131072 ? 4096 : 2048; }

__device__ __forceinline__ int bucket_of(unsigned long long k, unsigned long long kmin, int shift, int nb) {
  if (k <= kmin) return 0;
  const unsigned long long q = (k - kmin) >> shift;
  return q < (unsigned long long)nb ? (int)q : nb - 1;
}

// Shared memory of the search inside the dynamic region
struct CauchySmem {
  unsigned start[SMILI_NBUCKET_MAX + 4];                // first position of each bucket; [nb] = nbreak
  u128 cand[SMILI_KC];                                  // one batch of (key, index)
  unsigned hist2[256];                                  // digits of the oversized-bucket selection
  double wtot[SMILI_MAX_WARPS][28];                     // warp totals of the scan
  double a_s[SMILI_MAX_THREADS], b_s[SMILI_MAX_THREADS];
  double Mm[144];                                       // dense middle matrix, 6 + 6 rows and columns
  double st[3];                                         // D, t, dtm at the last element passed
  double P[12], Q[12];                                  // p and sum t d w there
  double cum[32];                                       // sums over the rounds done: d^2, d w, t d w, max t
  double pre[32], tot[32];
};
// Bytes of dynamic shared memory; the launch gives every CTA at least this much.
constexpr size_t SMILI_CAUCHY_SMEM = sizeof(CauchySmem);

// Select the next batch (<= SMILI_KC elements, the smallest composites from
// first on) from the unordered range [r0, r1) of the bucketed arrays into cand,
// by radix selection on 8-bit digits of the 96-bit composite (key, index).
// Used for a bucket that holds more than SMILI_KC breakpoints.
template <typename SY>
__device__ __noinline__ int select_from_range(LbCtxT<SY>& c, const unsigned long long* sbk, const int* sbi, int r0,
                                              int r1, u128 first, u128* cand, unsigned* hist) {
  __shared__ int cnt_s, vstar_s, cum_s;
  u128 prefix = 0;
  int level = 0, budget = SMILI_KC;
  u128 sel_hi = ~(u128)0;
  bool have_hi = false;
  while (true) {
    const int shift = 96 - 8 * (level + 1);
    for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
      const u128 ck = comp_key(sbk[i], sbi[i]);
      if (ck < first) continue;
      if (level > 0 && (ck >> (96 - 8 * level)) != prefix) continue;
      atomicAdd(&hist[(unsigned)((ck >> shift) & 0xffu)], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int cum = 0, vstar = -1;
      for (int b = 0; b < 256; ++b) {
        if (cum + (int)hist[b] > budget) {
          vstar = b;
          break;
        }
        cum += hist[b];
      }
      vstar_s = vstar;
      cum_s = cum;
    }
    __syncthreads();
    const int vstar = vstar_s, cum = cum_s;
    if (vstar < 0) {
      if (level > 0) {
        sel_hi = (prefix + 1) << (96 - 8 * level);
        have_hi = true;
      }
      break;
    }
    const u128 np = (prefix << 8) | (u128)vstar;
    if (cum == budget || (cum > 0 && (4 * cum >= budget || level == 11))) {
      sel_hi = np << shift;
      have_hi = true;
      break;
    }
    budget -= cum;
    prefix = np;
    ++level;
  }
  if (threadIdx.x == 0) cnt_s = 0;
  __syncthreads();
  for (int i0 = r0; i0 < r1; i0 += blockDim.x) {
    const int i = i0 + threadIdx.x;
    bool take = false;
    u128 ck = 0;
    if (i < r1) {
      ck = comp_key(sbk[i], sbi[i]);
      take = ck >= first && !(have_hi && ck >= sel_hi);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, take);
    if (bal) {
      const int lane = threadIdx.x & 31;
      int base = 0;
      if (lane == __ffs(bal) - 1) base = atomicAdd(&cnt_s, __popc(bal));
      base = __shfl_sync(0xffffffffu, base, __ffs(bal) - 1);
      const int pos = base + __popc(bal & ((1u << lane) - 1));
      if (take && pos < SMILI_KC) cand[pos] = ck;
    }
  }
  __syncthreads();
  const int cnt = min(cnt_s, SMILI_KC);
  __syncthreads();
  return cnt;
}

// Ascending bitonic sort of cand[0..cnt), cnt <= SMILI_KC.  Up to blockDim.x
// elements it runs with one element per thread: strides below 32 by
// shuffles, the others through shared memory (256 elements: 6 of 36 steps
// need a block barrier).
__device__ __noinline__ void sort_batch(u128* cand, int cnt) {
  int np2 = 32;
  while (np2 < cnt) np2 <<= 1;
  for (int i = cnt + threadIdx.x; i < np2; i += blockDim.x) cand[i] = ~(u128)0;
  __syncthreads();
  if (np2 <= (int)blockDim.x) {
    const int i = threadIdx.x;
    const bool act = i < np2;  // whole warps: np2 is a multiple of 32
    u128 v = act ? cand[i] : ~(u128)0;
    for (int k2 = 2; k2 <= np2; k2 <<= 1) {
      for (int j2 = k2 >> 1; j2 > 0; j2 >>= 1) {
        u128 o;
        if (j2 >= 32) {
          if (act) cand[i] = v;
          __syncthreads();
          o = act ? cand[i ^ j2] : v;
          __syncthreads();
        } else {
          const unsigned lo = __shfl_xor_sync(0xffffffffu, (unsigned)v, j2);
          const unsigned mi = __shfl_xor_sync(0xffffffffu, (unsigned)(v >> 32), j2);
          const unsigned hi = __shfl_xor_sync(0xffffffffu, (unsigned)(v >> 64), j2);
          const unsigned pad = __shfl_xor_sync(0xffffffffu, (unsigned)(v >> 96), j2);
          o = ((u128)pad << 96) | ((u128)hi << 64) | ((u128)mi << 32) | lo;
        }
        const bool up = (i & k2) == 0, lower = (i & j2) == 0;
        if ((lower == up) == (o < v)) v = o;
      }
    }
    if (act) cand[i] = v;
    __syncthreads();
    return;
  }
  for (int k2 = 2; k2 <= np2; k2 <<= 1) {
    for (int j2 = k2 >> 1; j2 > 0; j2 >>= 1) {
      for (int i = threadIdx.x; i < np2; i += blockDim.x) {
        const int ixj = i ^ j2;
        if (ixj > i) {
          const u128 a = cand[i], b = cand[ixj];
          const bool up = (i & k2) == 0;
          if ((a > b) == up) {
            cand[i] = b;
            cand[ixj] = a;
          }
        }
      }
      __syncthreads();
    }
  }
}

// f1 and f2 of the segment that starts at time t, from D, p and c = W'(z - x)
// there (rows 0..5 the Y part, 6..11 the S part, zero past col), and its
// minimiser's distance -f1 / f2
__device__ __forceinline__ double segment_dtm(const double* Mm, double D, double t, const double (&Pk)[12],
                                              const double (&ck)[12], double theta, double f2_floor) {
  double cMp = 0.0, pMp = 0.0;
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    double mp = 0.0;
#pragma unroll
    for (int j = 0; j < 12; ++j) mp += Mm[i * 12 + j] * Pk[j];
    cMp += ck[i] * mp;
    pMp += Pk[i] * mp;
  }
  const double f1 = -D + theta * t * D - cMp;
  const double f2 = fmax(f2_floor, theta * D - pMp);
  return -f1 / f2;
}

// First breakpoint position of a CTA whose nominal start is p: bucket
// boundaries at or after p.
__device__ __forceinline__ int bucket_cut(int p, int nbreak, const unsigned long long* sbk, const unsigned* start,
                                          unsigned long long kmin, int shift, int nb) {
  if (p >= nbreak) return nbreak;
  const int b = bucket_of(sbk[p], kmin, shift, nb);
  return (int)start[b] == p ? p : (int)start[b + 1];
}

// The generalized Cauchy point over the bucketed breakpoints, all CTAs of the
// group together.  Each round gives every CTA the buckets of about 256
// breakpoints (later rounds 1024): the CTAs sum d^2, d w and t d w over their
// buckets, exchange the sums, and so know the state of the piecewise
// quadratic where their buckets begin; each then sorts its own breakpoints by
// (t, index), scans them and tests every segment, and the first CTA in order
// that stopped has the result.  The rounds are serial only in their number:
// one CTA that walked all breakpoints, 1024 at a time, took 130 of a 64 x 64
// solve's 387 us per evaluation, and 19 of 20 ms at 1024 x 1024, where a
// minimiser lies some 190 000 breakpoints out.  A bucket of more than SMILI_KC
// breakpoints (equal times, mostly) is taken in batches by radix selection.
// cr[] (shared): the CR_* values.  Returns 0, -1 (singular middle matrix) or
// -2 (a wait timed out).
template <typename SY>
__device__ __noinline__ int cauchy_search(LbCtxT<SY>& c, double f1_0, const double* p0, int nbreak, int bnded,
                                          const unsigned long long* sbk, const int* sbi, unsigned long long kmin,
                                          int shift, int nb, double* cr) {
  LbState& S = *c.S;
  GroupCtx& g = *c.g;
  CauchySmem& sm = *reinterpret_cast<CauchySmem*>(c.dyn);
  const int m = c.m, col = S.col, col2 = 2 * col, n = c.n;
  const int T = blockDim.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = T >> 5;
  const double theta = S.theta;
  __shared__ unsigned long long bnd_hi_s, bnd_lo_s;
  __shared__ int e_star_s, info_s, win_s;
  __shared__ double f2org_s;
  Prof& pf = *c.prof;
  // dense middle matrix: column j = M e_j, at rows / columns a (Y) and 6 + a (S)
  for (int i = threadIdx.x; i < 144; i += T) sm.Mm[i] = 0.0;
  if (threadIdx.x < 32) sm.cum[threadIdx.x] = 0.0;
  if (threadIdx.x == 0) info_s = 0;
  __syncthreads();
  for (int j = wid; j < col2; j += nw) {  // column j of M, a warp each
    double y = lane == j ? 1.0 : 0.0, s = lane == j - col ? 1.0 : 0.0;
    if (!warp_bmv(S, m, col, y, s) && lane == 0) info_s = -1;
    const int jc = j < col ? j : 6 + j - col;
    if (lane < col) {
      sm.Mm[lane * 12 + jc] = y;
      sm.Mm[(6 + lane) * 12 + jc] = s;
    }
  }
  __syncthreads();
  if (info_s) return -1;  // singular middle matrix (bmv failure)
  if (threadIdx.x < 32) {
    double s = 0;
    if (lane < 12) {
#pragma unroll
      for (int j = 0; j < 12; ++j) s += sm.Mm[lane * 12 + j] * p0[j];
      s *= p0[lane];
    }
#pragma unroll
    for (int q = 8; q >= 1; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
    if (lane == 0) {
      double f2 = -theta * f1_0;
      f2org_s = f2;
      f2 -= s;
      sm.st[0] = -f1_0;
      sm.st[1] = 0.0;
      sm.st[2] = -f1_0 / f2;
      bnd_hi_s = 0;
      bnd_lo_s = 0;
    }
  }
  if (threadIdx.x < 12) {
    sm.P[threadIdx.x] = p0[threadIdx.x];
    sm.Q[threadIdx.x] = 0.0;
  }
  __syncthreads();
  const double f2_floor = S.epsmch * f2org_s;
  if (nbreak == 0) {  // GCP in the first segment (lbfgsb.f:1433, label 888)
    if (threadIdx.x == 0) {
      const double dtm = fmax(sm.st[2], 0.0);
      cr[CR_INFO] = 0;
      cr[CR_MODE] = CM_NONE_FIXED;
      cr[CR_TSUM] = dtm;
      cr[CR_NSEG] = 1;
      cr[CR_BHI] = 0.0;
      cr[CR_BLO] = 0.0;
      for (int j = 0; j < 12; ++j) cr[CR_C + j] = dtm * sm.P[j];
    }
    __syncthreads();
    return 0;
  }
  int pj[SMILI_MAXM_DEV];
#pragma unroll
  for (int j = 0; j < SMILI_MAXM_DEV; ++j) pj[j] = j < col ? lptr(S, m, j) : 0;
  int round0 = 0;  // first position of the round
  for (int round = 0;; ++round) {
    const int B = round == 0 ? 256 : 1024;
    int r0 = 0, r1 = nbreak, rnext = nbreak;
    if (g.G > 1) {
      const long nom = (long)round0 + (long)g.rank * B;
      r0 = g.rank == 0 ? round0 : bucket_cut((int)min(nom, (long)nbreak), nbreak, sbk, sm.start, kmin, shift, nb);
      r1 = bucket_cut((int)min(nom + B, (long)nbreak), nbreak, sbk, sm.start, kmin, shift, nb);
      rnext = bucket_cut((int)min((long)round0 + (long)g.G * B, (long)nbreak), nbreak, sbk, sm.start, kmin, shift, nb);
      // ---- sums over this CTA's buckets, and what precedes them ----
      double s[32], mx[1] = {0.0};
#pragma unroll
      for (int k = 0; k < 32; ++k) s[k] = 0.0;
      for (int i = r0 + threadIdx.x; i < r1; i += T) {
        const int idx = sbi[i];
        const double te = __longlong_as_double((long long)sbk[i]);
        const double d = c.d[idx];
        s[0] += d * d;
        mx[0] = fmax(mx[0], te);
#pragma unroll
        for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
          if (j < col) {
            const double y = d * ld_wy(c, (size_t)pj[j] * n + idx);
            const double w = d * (theta * ld_ws(c, (size_t)pj[j] * n + idx));
            s[1 + j] += y;
            s[7 + j] += w;
            s[13 + j] += te * y;
            s[19 + j] += te * w;
          }
        }
      }
      block_partials(s, 32, mx, 1, group_row(g, c.red), c.scratch);
      const double* part = g.red_part + (size_t)g.parity * g.G * g.redk;
      g.parity ^= 1;
      if (!group_sync(g)) return -2;
      {
        const int k = threadIdx.x & 31, sl = threadIdx.x >> 5, S_ = T >> 5;
        const bool sum = k < 31;
        double pre = 0.0, tot = 0.0;
        constexpr int D = 4;  // rows in flight
        for (int r = sl; r < g.G; r += D * S_) {
          double v[D];
#pragma unroll
          for (int q = 0; q < D; ++q)
            v[q] = r + q * S_ < g.G ? __ldcg(part + (size_t)(r + q * S_) * g.redk + (sum ? k : 32)) : 0.0;
#pragma unroll
          for (int q = 0; q < D; ++q) {
            const double b = r + q * S_ < g.rank ? v[q] : 0.0;
            tot = sum ? tot + v[q] : fmax(tot, v[q]);
            pre = sum ? pre + b : fmax(pre, b);
          }
        }
        sm.a_s[threadIdx.x] = pre;
        sm.b_s[threadIdx.x] = tot;
        __syncthreads();
        if (threadIdx.x < 32) {
          double a = sm.a_s[k], b = sm.b_s[k];
          for (int q = 1; q < S_; ++q) {
            a = sum ? a + sm.a_s[q * 32 + k] : fmax(a, sm.a_s[q * 32 + k]);
            b = sum ? b + sm.b_s[q * 32 + k] : fmax(b, sm.b_s[q * 32 + k]);
          }
          // sums and latest time over everything before this CTA's buckets
          const double cu = sm.cum[k];
          sm.pre[k] = sum ? cu + a : fmax(cu, a);
          sm.cum[k] = sum ? cu + b : fmax(cu, b);
        }
        __syncthreads();
      }
      if (r0 > 0 && r0 < r1) {
        if (threadIdx.x < 32) {  // segment_dtm, a row of M per lane
          const double D = -f1_0 - sm.pre[0], t = sm.pre[31];
          double Pl = 0.0, cl = 0.0, mp = 0.0;
          if (lane < 12) {
            Pl = p0[lane] - sm.pre[1 + lane];
            cl = t * Pl + sm.pre[13 + lane];
            sm.P[lane] = Pl;
            sm.Q[lane] = sm.pre[13 + lane];
          }
#pragma unroll 1
          for (int j = 0; j < 12; ++j) {
            const double pj_ = __shfl_sync(0xffffffffu, Pl, j);
            if (lane < 12) mp += sm.Mm[lane * 12 + j] * pj_;
          }
          double cMp = cl * mp, pMp = Pl * mp;
#pragma unroll
          for (int q = 8; q >= 1; q >>= 1) {
            cMp += __shfl_xor_sync(0xffffffffu, cMp, q);
            pMp += __shfl_xor_sync(0xffffffffu, pMp, q);
          }
          if (lane == 0) {
            sm.st[0] = D;
            sm.st[1] = t;
            sm.st[2] = (D - theta * t * D + cMp) / fmax(f2_floor, theta * D - pMp);
            // every breakpoint before these buckets, whatever its index
            const u128 ckk = comp_key((unsigned long long)__double_as_longlong(t), -1);
            bnd_hi_s = (unsigned long long)(ckk >> 64);
            bnd_lo_s = (unsigned long long)ckk;
          }
        }
      }
      pf.mark(PR_C_GATHER);
    }
    __syncthreads();
    // ---- this CTA's breakpoints, a batch of whole buckets at a time ----
    bool finished = false;
    int pos = r0, kdone = r0;
    int big_r0 = -1, big_r1 = -1;  // an oversized bucket being consumed by radix selection
    while (pos < r1 && !finished) {
      int cnt;
      if (big_r0 < 0) {
        int e = min(pos + T, r1);
        if (e < r1) {
          const int b = bucket_of(sbk[e], kmin, shift, nb);
          e = (int)sm.start[b];                   // the batch ends where e's bucket begins,
          if (e <= pos) e = (int)sm.start[b + 1];  // or is that one bucket
        }
        cnt = e - pos;
        if (cnt > SMILI_KC) {
          big_r0 = pos;
          big_r1 = e;
        } else {
          for (int i = threadIdx.x; i < cnt; i += T) sm.cand[i] = comp_key(sbk[pos + i], sbi[pos + i]);
        }
      }
      if (big_r0 >= 0) {
        // past the last element taken; none yet: from the least composite, 0 (a
        // time that underflowed, at index 0)
        const u128 first = kdone == 0 ? 0 : (((u128)bnd_hi_s << 64) | (u128)bnd_lo_s) + 1;
        cnt = select_from_range(c, sbk, sbi, big_r0, big_r1, first, sm.cand, sm.hist2);
      }
      __syncthreads();
      pf.count(PR_C_ROUNDS);
      sort_batch(sm.cand, cnt);
      pf.mark(PR_C_SORT);
      // ---- scan in chunks of T ----
      for (int base = 0; base < cnt; base += T) {
        const int e = threadIdx.x, ge = base + e;
        const bool valid = ge < cnt;
        double vals[25];
        double te = 0.0;
        int idx = 0;
#pragma unroll
        for (int v = 0; v < 25; ++v) vals[v] = 0.0;
        if (valid) {
          const u128 ck = sm.cand[ge];
          idx = (int)(unsigned)(ck & 0xffffffffu);
          te = __longlong_as_double((long long)(unsigned long long)(ck >> 32));
          const double dibp = c.d[idx];
          vals[0] = dibp * dibp;
#pragma unroll
          for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
            if (j < col) {
              const double y = dibp * ld_wy(c, (size_t)pj[j] * n + idx);
              const double w = dibp * (theta * ld_ws(c, (size_t)pj[j] * n + idx));
              vals[1 + j] = y;
              vals[7 + j] = w;
              vals[13 + j] = te * y;
              vals[19 + j] = te * w;
            }
          }
        }
        // inclusive scan over the block: warps, then the warps' totals
#pragma unroll
        for (int v = 0; v < 25; ++v) {
          double a = vals[v];
#pragma unroll
          for (int sft = 1; sft < 32; sft <<= 1) {
            const double o = __shfl_up_sync(0xffffffffu, a, sft);
            if (lane >= sft) a += o;
          }
          vals[v] = a;
          if (lane == 31) sm.wtot[wid][v] = a;
        }
        if (threadIdx.x == 0) e_star_s = T;
        __syncthreads();
        if (threadIdx.x < 25) {
          double run = 0.0;
          for (int w = 0; w < nw; ++w) {
            const double x = sm.wtot[w][threadIdx.x];
            sm.wtot[w][threadIdx.x] = run;
            run += x;
          }
        }
        __syncthreads();
        double dtm_e = 0.0, Dk = 0.0, Pk[12], ck_[12];
        if (valid) {
          Dk = sm.st[0] - (vals[0] + sm.wtot[wid][0]);
#pragma unroll
          for (int j = 0; j < 12; ++j) {
            Pk[j] = sm.P[j] - (vals[1 + j] + sm.wtot[wid][1 + j]);
            ck_[j] = te * Pk[j] + (sm.Q[j] + (vals[13 + j] + sm.wtot[wid][13 + j]));
          }
          dtm_e = segment_dtm(sm.Mm, Dk, te, Pk, ck_, theta, f2_floor);
          sm.a_s[e] = dtm_e;
          sm.b_s[e] = te;
        }
        __syncthreads();
        // stop test for the segment ending at this element
        if (valid) {
          const double pd = (e == 0) ? sm.st[2] : sm.a_s[e - 1];
          const double pt = (e == 0) ? sm.st[1] : sm.b_s[e - 1];
          if (pd < (te - pt)) atomicMin(&e_star_s, e);
        }
        __syncthreads();
        const int es = e_star_s;
        const int nvalid = min(T, cnt - base);
        if (es < T) {
          // GCP inside the segment before element es: breakpoints up to es-1 fixed
          if ((es == 0 && threadIdx.x == 0) || (es > 0 && e == es - 1)) {
            double tsum, dtm;
            if (es == 0) {
              tsum = sm.st[1];
              dtm = fmax(sm.st[2], 0.0);
#pragma unroll
              for (int j = 0; j < 12; ++j) cr[CR_C + j] = tsum * sm.P[j] + sm.Q[j] + dtm * sm.P[j];
            } else {
              tsum = te;
              dtm = fmax(dtm_e, 0.0);
#pragma unroll
              for (int j = 0; j < 12; ++j) cr[CR_C + j] = ck_[j] + dtm * Pk[j];
              const u128 ckk = comp_key(__double_as_longlong(te), idx);
              bnd_hi_s = (unsigned long long)(ckk >> 64);
              bnd_lo_s = (unsigned long long)ckk;
            }
            cr[CR_MODE] = (kdone + es == 0) ? CM_NONE_FIXED : CM_BOUNDARY;
            cr[CR_TSUM] = tsum + dtm;
            cr[CR_NSEG] = kdone + es + 1;
          }
          finished = true;
          __syncthreads();
          break;
        }
        // no stop in this chunk: carry the state of its last element
        if (e == nvalid - 1) {
          sm.st[0] = Dk;
          sm.st[1] = te;
          sm.st[2] = dtm_e;
#pragma unroll
          for (int j = 0; j < 12; ++j) {
            sm.P[j] = Pk[j];
            sm.Q[j] = ck_[j] - te * Pk[j];
          }
          const u128 ckk = comp_key(__double_as_longlong(te), idx);
          bnd_hi_s = (unsigned long long)(ckk >> 64);
          bnd_lo_s = (unsigned long long)ckk;
        }
        __syncthreads();
        kdone += nvalid;
        if (kdone == nbreak) {
          // every breakpoint passed without a stop (lbfgsb.f:1640-1660)
          if (threadIdx.x == 0) {
            cr[CR_MODE] = CM_BOUNDARY;
            cr[CR_NSEG] = kdone;
            // all variables at their bounds: c = W'(xcp - x) = t_n P_n + Q_n
            const double dtm = (nbreak == n || bnded) ? 0.0 : fmax(sm.st[2], 0.0);
            cr[CR_TSUM] = sm.st[1] + dtm;
            for (int j = 0; j < 12; ++j) cr[CR_C + j] = sm.st[1] * sm.P[j] + sm.Q[j] + dtm * sm.P[j];
          }
          finished = true;
          __syncthreads();
          break;
        }
      }
      pf.mark(PR_C_SCAN);
      if (big_r0 >= 0) {
        if (kdone >= big_r1) {  // the oversized bucket is consumed
          pos = big_r1;
          big_r0 = big_r1 = -1;
        }
      } else {
        pos += cnt;
      }
    }
    if (finished && threadIdx.x == 0) {
      cr[CR_INFO] = 0;
      cr[CR_BHI] = __longlong_as_double((long long)bnd_hi_s);
      cr[CR_BLO] = __longlong_as_double((long long)bnd_lo_s);
    }
    __syncthreads();
    if (g.G == 1) return 0;  // one CTA has walked every breakpoint it needs
    // ---- the first CTA in order that stopped ----
    double* row = group_row(g, c.red);
    if (threadIdx.x < CR_C + 12 && finished) row[1 + threadIdx.x] = cr[threadIdx.x];
    if (threadIdx.x == 0) {
      row[0] = finished ? 1.0 : 0.0;
      win_s = g.G;
    }
    const double* part = g.red_part + (size_t)g.parity * g.G * g.redk;
    g.parity ^= 1;
    if (!group_sync(g)) return -2;
    for (int r = threadIdx.x; r < g.G; r += T)
      if (__ldcg(part + (size_t)r * g.redk) != 0.0) {
        atomicMin(&win_s, r);
        break;
      }
    __syncthreads();
    const int win = win_s;
    if (win < g.G) {
      if (threadIdx.x < CR_C + 12) cr[threadIdx.x] = __ldcg(part + (size_t)win * g.redk + 1 + threadIdx.x);
      __syncthreads();
      return 0;
    }
    round0 = rnext;
    __syncthreads();
    pf.mark(PR_C_SEL);
  }
}

// Returns 0 on success, -1 when bmv failed (info != 0).
template <typename SY>
__device__ __noinline__ int lb_cauchy(LbCtxT<SY>& c) {
  LbState& S = *c.S;
  const ProbDesc& P = *c.P;
  const int m = c.m, n = c.n, col = S.col, col2 = 2 * col;
  const bool nonneg = P.nonneg;
  unsigned long long* sbk = at<unsigned long long>(c.base, P.o_sbk);
  int* sbi = at<int>(c.base, P.o_sbi);
  int* ghist = at<int>(c.base, P.o_hist);  // [SMILI_NBUCKET_MAX] counts, [SMILI_NBUCKET_MAX] cursors
  __shared__ double cr_s[CR_C + 12], p0_s[12];
  if (S.sbgnrm <= 0.0) {
    // GCP = X (lbfgsb.f:1318-1322): z = x, iwhere untouched
    for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) c.z[i] = c.x[i];
    if (threadIdx.x == 0) cr_s[CR_MODE] = CM_XCP_IS_X;
  } else {
    int pj[SMILI_MAXM_DEV];
#pragma unroll
    for (int j = 0; j < SMILI_MAXM_DEV; ++j) pj[j] = j < col ? lptr(S, m, j) : 0;
    // sums: [0..5] Y'd, [6..11] S'd (zero past col), [12] f1, [13] nbreak,
    // [14] and [15] the first two moments of the keys' upper words (less
    // 1.0's); maxima: notbnded, -tmin, tmax, any variable without a breakpoint
    double f1a = 0.0, nbr = 0.0, k1 = 0.0, k2 = 0.0, nfr = 0.0, notb = 0.0, tmn = 1.0e308, tmx = 0.0;
    double py[SMILI_MAXM_DEV], ps[SMILI_MAXM_DEV];
#pragma unroll
    for (int j = 0; j < SMILI_MAXM_DEV; ++j) py[j] = ps[j] = 0.0;
    const int nb = cauchy_buckets(n);
    for (int i = c.g->rank * blockDim.x + threadIdx.x; i < 2 * SMILI_NBUCKET_MAX; i += c.g->G * blockDim.x)
      ghist[i] = 0;
    // U elements of a thread at a time, all loads of a step before its stores
    // (which may alias them for the compiler): the pass is bound by the latency
    // of its two dependent loads per step
    constexpr int U = sizeof(SY) == 8 ? 2 : 1;
    const int bd = blockDim.x;
    for (int i0 = c.lo + threadIdx.x; i0 < c.hi; i0 += U * bd) {
      double ng[U], xv[U];
      int iw[U];
      bool in[U], mv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * bd;
        in[u] = i < c.hi;
        ng[u] = in[u] ? -c.gv[i] : 0.0;
        xv[u] = in[u] ? c.x[i] : 0.0;
        iw[u] = in[u] ? c.iwh[i] : 3;
      }
      bool set[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        set[u] = in[u] && iw[u] != 3 && iw[u] != -1;
        if (set[u]) {
          // x - l with l = 0 (nbd = 1)
          iw[u] = xv[u] <= 0.0 ? (ng[u] <= 0.0 ? 1 : 0) : (fabs(ng[u]) <= 0.0 ? -3 : 0);
        }
        mv[u] = in[u] && (iw[u] == 0 || iw[u] == -1);
      }
      SY wy[U][SMILI_MAXM_DEV], ws[U][SMILI_MAXM_DEV];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
          const bool l = mv[u] && j < col;
          wy[u][j] = l ? c.wy[(size_t)pj[j] * n + i0 + u * bd] : (SY)0;
          ws[u][j] = l ? c.ws[(size_t)pj[j] * n + i0 + u * bd] : (SY)0;
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!in[u]) continue;
        const int i = i0 + u * bd;
        unsigned long long key = ~0ULL;
        if (mv[u]) {
          f1a -= ng[u] * ng[u];
#pragma unroll
          for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
            if (j < col) {
              py[j] += (double)wy[u][j] * ng[u];
              ps[j] += (double)ws[u][j] * ng[u];
            }
          }
          if (nonneg && ng[u] < 0.0) {
            const double tb = (set[u] ? xv[u] : 0.0) / (-ng[u]);
            nbr += 1.0;
            tmn = fmin(tmn, tb);
            tmx = fmax(tmx, tb);
            key = (unsigned long long)__double_as_longlong(tb);
            const double kh = (double)((int)(key >> 32) - 0x3ff00000);
            k1 += kh;
            k2 += kh * kh;
          } else {
            nfr = 1.0;
            if (fabs(ng[u]) > 0.0) notb = 1.0;
          }
        }
        if (set[u]) c.iwh[i] = (signed char)iw[u];
        c.d[i] = mv[u] ? ng[u] : 0.0;
        c.bkey[i] = key;
      }
    }
    double acc[16];
#pragma unroll
    for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
      acc[j] = py[j];
      acc[SMILI_MAXM_DEV + j] = ps[j];
    }
    acc[12] = f1a;
    acc[13] = nbr;
    acc[14] = k1;
    acc[15] = k2;
    const double accx[4] = {notb, -tmn, tmx, nfr};
    if (!lb_reduce(c, acc, accx)) return -2;
    const double f1 = c.red[12];
    if (threadIdx.x < 12) p0_s[threadIdx.x] = (threadIdx.x < 6 ? 1.0 : S.theta) * c.red[threadIdx.x];
    const int nbreak = (int)c.red[13];
    const int bnded = c.red[16] > 0.5 ? 0 : 1;
    const bool any_free = c.red[19] > 0.5;
    // key range of the buckets: all of it, but no more than three standard
    // deviations of the keys' exponents around their mean (a few far
    // breakpoints would otherwise leave the bulk in a few buckets)
    unsigned long long kmin = (unsigned long long)__double_as_longlong(-c.red[17]);
    unsigned long long kmax = (unsigned long long)__double_as_longlong(c.red[18]);
    if (nbreak > 0) {
      const double mu = c.red[14] / nbreak, var = c.red[15] / nbreak - mu * mu;
      const double sd = sqrt(fmax(var, 0.0)) + 64.0;
      const double lo = floor(mu - 3.0 * sd) + 0x3ff00000, hi = ceil(mu + 3.0 * sd) + 0x3ff00000;
      if (lo > 0.0 && lo < 2147483647.0) kmin = max(kmin, (unsigned long long)lo << 32);
      if (hi > 0.0 && hi < 2147483647.0) kmax = min(kmax, (unsigned long long)hi << 32);
      if (kmax < kmin) kmax = kmin;
    }
    __syncthreads();
    if (nbreak == 0 && !any_free) {
      for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) c.z[i] = c.x[i];
      if (threadIdx.x == 0) cr_s[CR_MODE] = CM_XCP_IS_X;
    } else {
      CauchySmem& sm = *reinterpret_cast<CauchySmem*>(c.dyn);
      int shift = 0;
      if (nbreak > 0) {
        // bucket the breakpoints: histogram, then scatter in bucket order
        shift = max(0, 32 + __clz(nb) - __clzll((long long)(kmax - kmin)) + 1);  // (kmax - kmin) >> shift < nb
        for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) {
          const unsigned long long k = c.bkey[i];
          if (k != ~0ULL) atomicAdd(&ghist[bucket_of(k, kmin, shift, nb)], 1);
        }
        if (!group_sync(*c.g)) return -2;
        // exclusive prefix of the bucket counts -> start offsets, in every CTA
        {
          __shared__ unsigned wsum_s[SMILI_MAX_WARPS];
          const int per = nb / blockDim.x;  // 4, 8 or 16 buckets per thread
          const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
          unsigned cnt[SMILI_NBUCKET_MAX / 256], run = 0;
#pragma unroll
          for (int q = 0; q < SMILI_NBUCKET_MAX / 256; q += 4) {
            if (q < per) {
              const int4 v = __ldcg(reinterpret_cast<const int4*>(ghist + threadIdx.x * per + q));
              cnt[q] = v.x;
              cnt[q + 1] = v.y;
              cnt[q + 2] = v.z;
              cnt[q + 3] = v.w;
              run += v.x + v.y + v.z + v.w;
            }
          }
          unsigned incl = run;
#pragma unroll
          for (int s2 = 1; s2 < 32; s2 <<= 1) {
            const unsigned o = __shfl_up_sync(0xffffffffu, incl, s2);
            if (lane >= s2) incl += o;
          }
          if (lane == 31) wsum_s[wid] = incl;
          __syncthreads();
          unsigned off = incl - run;
          for (int w = 0; w < wid; ++w) off += wsum_s[w];
#pragma unroll
          for (int q = 0; q < SMILI_NBUCKET_MAX / 256; ++q) {
            if (q < per) {
              sm.start[threadIdx.x * per + q] = off;
              off += cnt[q];
            }
          }
          if (threadIdx.x == 0) sm.start[nb] = (unsigned)nbreak;
        }
        __syncthreads();
        for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) {
          const unsigned long long k = c.bkey[i];
          if (k != ~0ULL) {
            const int b = bucket_of(k, kmin, shift, nb);
            const int q = (int)sm.start[b] + atomicAdd(&ghist[SMILI_NBUCKET_MAX + b], 1);
            sbk[q] = k;
            sbi[q] = i;
          }
        }
        if (!group_sync(*c.g)) return -2;
        c.prof->mark(PR_C_SEL);
      }
      const int rc = cauchy_search(c, f1, p0_s, nbreak, bnded, sbk, sbi, kmin, shift, nb, cr_s);
      if (rc != 0) return rc;
    }
  }
  __syncthreads();
  const int mode = (int)cr_s[CR_MODE];
  // apply the GCP and run freev (lbfgsb.f:2241-2340)
  double acc[4] = {0, 0, 0, 0};  // nfree, nenter, nleave
  const u128 bnd = ((u128)(unsigned long long)__double_as_longlong(cr_s[CR_BHI]) << 64) |
                   (u128)(unsigned long long)__double_as_longlong(cr_s[CR_BLO]);
  const double tsum = cr_s[CR_TSUM];
  const bool count_moves = S.iter > 0 && S.cnstnd;
  constexpr int UA = 2;  // elements in flight per thread
  const int bda = blockDim.x;
  const bool apply = mode == CM_BOUNDARY || mode == CM_NONE_FIXED;
  for (int i0 = c.lo + threadIdx.x; i0 < c.hi; i0 += UA * bda) {
    unsigned long long k[UA];
    double xv[UA], dv[UA];
    int iw[UA], fo[UA];
#pragma unroll
    for (int u = 0; u < UA; ++u) {
      const int i = i0 + u * bda;
      const bool in = i < c.hi;
      k[u] = in && mode == CM_BOUNDARY ? c.bkey[i] : ~0ULL;
      xv[u] = in && apply ? c.x[i] : 0.0;
      dv[u] = in && apply ? c.d[i] : 0.0;
      iw[u] = in ? c.iwh[i] : 1;
      fo[u] = in ? c.freef[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < UA; ++u) {
      const int i = i0 + u * bda;
      if (i >= c.hi) continue;
      if (k[u] != ~0ULL && comp_key(k[u], i) <= bnd) {
        c.z[i] = 0.0;  // lower bound (d < 0 at every breakpoint)
        c.iwh[i] = 1;
        iw[u] = 1;
        c.d[i] = 0.0;
      } else if (apply) {
        c.z[i] = xv[u] + tsum * dv[u];
      }
      const int fnew = iw[u] <= 0;
      if (count_moves) {
        if (fo[u] && !fnew) acc[2] += 1;
        if (!fo[u] && fnew) acc[1] += 1;
      }
      c.freef[i] = (unsigned char)fnew;
      acc[0] += fnew;
    }
  }
  const double none[1] = {0.0};
  if (!lb_reduce(c, acc, none)) return -2;
  if (threadIdx.x == 0) {
    if (mode != CM_XCP_IS_X) {
      S.nseg = (int)cr_s[CR_NSEG];
      for (int j = 0; j < col; ++j) {  // c
        S.wa[2 * m + j] = cr_s[CR_C + j];
        S.wa[2 * m + col + j] = cr_s[CR_C + 6 + j];
      }
    }
    S.nfree = (int)c.red[0];
    S.nenter = (int)c.red[1];
    S.ileave = n + 1 - (int)c.red[2];
    S.wrk = (c.red[2] > 0) || (c.red[1] > 0) || S.updatd;
    S.nact = n - S.nfree;
  }
  __syncthreads();
  return 0;
}

// ---------------------------------------------------------------------------
// formk (lbfgsb.f:1848-2172) from Gram sums over the free/active sets
// ---------------------------------------------------------------------------
template <typename SY>
__device__ __noinline__ int lb_formk(LbCtxT<SY>& c) {
  LbState& S = *c.S;
  const int m = c.m, n = c.n, col = S.col;
  // entries: Fyy (a<=b), Ass (a<=b), Fsy (a,b), Asy (a,b) over physical columns
  const int nsym = m * (m + 1) / 2;
  const int E = 2 * nsym + 2 * m * m;
  // The four masked Gram blocks W' diag(mask) W over this CTA's pixels on
  // the FP64 tensor cores: per 4 pixels, A = (masked column a at pixel k),
  // B = (column b at pixel k); lane (a = l/4, k = l%4) holds the same
  // element of both operands, so one load per matrix feeds both.
  //   Fyy = Y'FY, Fsy = S'FY (free pixels), Ass = S'AS, Asy = S'AY (active)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int ca = lane >> 2, pk = lane & 3;
  const bool cval = ca < m;  // m <= 6 < 8: one 8x8 tile per block
  const size_t colo = (size_t)(cval ? ca : 0) * n;
  double fyy[2] = {0.0, 0.0}, fsy[2] = {0.0, 0.0}, ass[2] = {0.0, 0.0}, asy[2] = {0.0, 0.0};
  const int nchunk = (c.hi - c.lo + 3) >> 2;
  constexpr int U = 4;  // chunks in flight per warp
  for (int q0 = warp; q0 < nchunk; q0 += U * nw) {
    double y[U], sv[U];
    bool fr[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = c.lo + 4 * (q0 + u * nw) + pk;
      const bool ok = i < c.hi;  // q0 + u*nw < nchunk whenever i < hi
      y[u] = (ok && cval) ? ld_wy(c, colo + i) : 0.0;
      sv[u] = (ok && cval) ? ld_ws(c, colo + i) : 0.0;
      fr[u] = ok && c.freef[i] != 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double yf = fr[u] ? y[u] : 0.0, sf = fr[u] ? sv[u] : 0.0, sa = fr[u] ? 0.0 : sv[u];
      dmma_884(fyy, yf, y[u]);
      dmma_884(fsy, sf, y[u]);
      dmma_884(ass, sa, sv[u]);
      dmma_884(asy, sa, y[u]);
    }
  }
  // combine the warps' tiles in fixed order: part[warp][tile][8x8]
  double* part = reinterpret_cast<double*>(c.dyn);
  {
    double* pw = part + (size_t)warp * 4 * 64 + ca * 8 + 2 * pk;
    pw[0] = fyy[0];
    pw[1] = fyy[1];
    pw[64] = fsy[0];
    pw[65] = fsy[1];
    pw[128] = ass[0];
    pw[129] = ass[1];
    pw[192] = asy[0];
    pw[193] = asy[1];
  }
  __syncthreads();
  double* row = group_row(*c.g, c.red);
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int t, a, b;
    if (e < 2 * nsym) {  // triangular index -> (a, b), a <= b
      t = e < nsym ? 0 : 2;
      int r = e < nsym ? e : e - nsym;
      a = 0;
      while (r >= m - a) {
        r -= m - a;
        ++a;
      }
      b = a + r;
    } else {
      const int r = e - 2 * nsym;
      t = r < m * m ? 1 : 3;
      const int q = r < m * m ? r : r - m * m;
      a = q / m;
      b = q % m;
    }
    double sum = 0.0;
    for (int w = 0; w < nw; ++w) sum += part[(size_t)w * 256 + t * 64 + a * 8 + b];
    row[e] = sum;
  }
  if (!group_combine(*c.g, E, E, c.red, c.scratch)) return -9;
  int info = 0;
  if (threadIdx.x < 32) {
    // lane j < col: column j of the Y block; lane col + j: of the S block
    const int col2 = 2 * col, jl = lane < col ? lane : lane - col;
    const int pj = lane < col2 ? lptr(S, m, jl) : 0;
    auto sym = [&](int base, int a, int b) {  // entry of a symmetric block
      const int lo = min(a, b), hi = max(a, b);
      return c.red[base + lo * m - lo * (lo - 1) / 2 + (hi - lo)];
    };
#pragma unroll 1
    for (int i = 0; i <= lane && lane < col2; ++i) {
      const int pi = lptr(S, m, i < col ? i : i - col);
      double v;
      if (lane < col) {
        v = sym(0, pj, pi) / S.theta;
        if (i == lane) v += S.sy[i + m * i];
      } else if (i < col) {
        // wn1(m + j, i): minus the active sum before j, the free sum from there
        v = i < jl ? -c.red[2 * nsym + m * m + pj * m + pi] : c.red[2 * nsym + pj * m + pi];
      } else {
        v = sym(nsym, pj, pi) * S.theta;
      }
      S.wn[i + 2 * m * lane] = v;
    }
    __syncwarp();
    info = warp_factor(S.wn, 2 * m, col2, col, S.rwn);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    c.red[0] = info;
  }
  __syncthreads();
  info = (int)c.red[0];
  __syncthreads();
  return info;
}

// ---------------------------------------------------------------------------
// cmprlb + subsm (lbfgsb.f:1720-1786, 2991-3346).  Returns 0 or an error;
// ls_ready: d, t and the sums of lb_lnsrch_start are made (c.red: g.d, d.d,
// iword, -stpmx).
// ---------------------------------------------------------------------------
template <typename SY>
__device__ __noinline__ int lb_cmprlb_subsm(LbCtxT<SY>& c, bool& ls_ready) {
  LbState& S = *c.S;
  const ProbDesc& P = *c.P;
  const int m = c.m, n = c.n, col = S.col, col2 = 2 * col;
  int pj[SMILI_MAXM_DEV];
#pragma unroll
  for (int j = 0; j < SMILI_MAXM_DEV; ++j) pj[j] = j < col ? lptr(S, m, j) : 0;
  __shared__ double a_s[2 * SMILI_MAXM_DEV], wv_s[2 * SMILI_MAXM_DEV];
  __shared__ int err_s;
  const bool unc = !S.cnstnd && col > 0;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    if (lane == 0) err_s = 0;
    if (!unc) {
      double y = lane < col ? S.wa[2 * m + lane] : 0.0, s = lane < col ? S.wa[2 * m + col + lane] : 0.0;
      if (!warp_bmv(S, m, col, y, s) && lane == 0) err_s = -8;
      if (lane < col) {
        a_s[lane] = y;
        a_s[col + lane] = s;
      }
    }
  }
  __syncthreads();
  if (err_s) return err_s;
  const double theta = S.theta;
  double ay[SMILI_MAXM_DEV], as[SMILI_MAXM_DEV];
#pragma unroll
  for (int j = 0; j < SMILI_MAXM_DEV; ++j) ay[j] = as[j] = 0.0;
  // the free flag of the next element is fetched one iteration ahead, so
  // the loads of an element wait for nothing but themselves
  const int bd = blockDim.x;
  int i = c.lo + threadIdx.x;
  bool f_next = i < c.hi && (unc || c.freef[i]);
  for (; i < c.hi; i += bd) {
    const bool fr = f_next;
    f_next = i + bd < c.hi && (unc || c.freef[i + bd]);
    if (!fr) continue;
    // the row of W at pixel i, loaded once for r_i and for W'Z r
    double wyv[SMILI_MAXM_DEV], wsv[SMILI_MAXM_DEV];
#pragma unroll
    for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
      wyv[j] = j < col ? ld_wy(c, (size_t)pj[j] * n + i) : 0.0;
      wsv[j] = j < col ? ld_ws(c, (size_t)pj[j] * n + i) : 0.0;
    }
    double ri;
    if (unc) {
      ri = -c.gv[i];
    } else {
      ri = -theta * (c.z[i] - c.x[i]) - c.gv[i];
#pragma unroll
      for (int j = 0; j < SMILI_MAXM_DEV; ++j)
        if (j < col) ri += wyv[j] * a_s[j] + wsv[j] * (theta * a_s[col + j]);
    }
    c.r[i] = ri;
#pragma unroll
    for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
      if (j < col) {
        ay[j] += wyv[j] * ri;
        as[j] += wsv[j] * ri;
      }
    }
  }
  double acc[16];
#pragma unroll
  for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
    acc[j] = ay[j];
    acc[SMILI_MAXM_DEV + j] = as[j];
  }
#pragma unroll
  for (int j = 2 * SMILI_MAXM_DEV; j < 16; ++j) acc[j] = 0.0;
  const double none[1] = {0.0};
  if (!lb_reduce(c, acc, none)) return -9;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    bool ok, ok2;
    double w = 0.0;
    if (lane < col2) w = lane < col ? c.red[lane] : theta * c.red[SMILI_MAXM_DEV + lane - col];
    w = warp_tri_solve(S.wn, 2 * m, col2, S.rwn, w, true, ok);
    w = warp_tri_solve(S.wn, 2 * m, col2, S.rwn, lane < col ? -w : w, false, ok2);
    if (!ok && lane == 0) err_s = -1;
    if (lane < col2) wv_s[lane] = w;
  }
  __syncthreads();
  if (err_s) return err_s;
  // d := (d + W wv) / theta on the free set, then project z + d.  The pass also
  // makes the line search's first step out of the result, which stands unless
  // a backtrack follows: d = z - x, t = x, their sums and the largest step
  const bool bounded_steps = S.cnstnd && S.iter > 0 && P.nonneg;
  double mx2[2] = {0.0, -1.0e10}, sm2[2] = {0.0, 0.0};  // iword, -stpmx (maxima); g.d = dd_p, d.d (sums)
  double wq[SMILI_MAXM_DEV], wr[SMILI_MAXM_DEV];
#pragma unroll
  for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
    wq[j] = j < col ? wv_s[j] : 0.0;
    wr[j] = j < col ? wv_s[col + j] : 0.0;
  }
  const double rtheta = 1.0 / theta;
  // One pass: d, the projected z and the directional derivative (z - x).g;
  // all loads of an element before its stores (which may alias them for the
  // compiler), the free flag one element ahead.  With the line search's start in
  // it: FP64 at 64^2 to 1024^2 a group sum and a pass less; FP32 (74 problems of
  // 256 x 256) 320 us for this and the line search against 322 apart, the
  // launch 72.9 against 73.2 ms.
  i = c.lo + threadIdx.x;
  f_next = i < c.hi && (unc || c.freef[i]);
  for (; i < c.hi; i += bd) {
    const bool fr = f_next;
    f_next = i + bd < c.hi && (unc || c.freef[i + bd]);
    const double zi = c.z[i], xv = c.x[i], gvi = c.gv[i];
    double ri = fr ? c.r[i] : 0.0;
    SY wyr[SMILI_MAXM_DEV], wsr[SMILI_MAXM_DEV];
#pragma unroll
    for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
      wyr[j] = (fr && j < col) ? c.wy[(size_t)pj[j] * n + i] : (SY)0;
      wsr[j] = (fr && j < col) ? c.ws[(size_t)pj[j] * n + i] : (SY)0;
    }
    c.xp[i] = zi;
    double zn = zi;
    if (fr) {
#pragma unroll
      for (int j = 0; j < SMILI_MAXM_DEV; ++j)
        if (j < col) ri += (double)wyr[j] * wq[j] / theta + (double)wsr[j] * wr[j];
      ri *= rtheta;
      c.r[i] = ri;
      if (P.nonneg) {
        zn = fmax(0.0, zi + ri);
        if (zn == 0.0) mx2[0] = 1.0;
      } else {
        zn = zi + ri;
      }
      c.z[i] = zn;
    }
    const double di = zn - xv;
    c.d[i] = di;
    c.t[i] = xv;
    sm2[0] += di * gvi;
    sm2[1] += di * di;
    if (bounded_steps && di < 0.0) {
      const double a2 = -xv;  // l - x with l = 0
      mx2[1] = fmax(mx2[1], a2 >= 0.0 ? 0.0 : -(a2 / di));
    }
  }
  if (!lb_reduce(c, sm2, mx2)) return -9;
  const int iword = c.red[2] > 0.5;
  const double dd_p = c.red[0];
  if (threadIdx.x == 0) S.iword = iword;
  __syncthreads();
  if (!iword || dd_p <= 0.0) {
    ls_ready = true;
    return 0;
  }
  // backtrack: z = xp, alpha = largest feasible step along d (lbfgsb.f:3270-3330)
  double zero[1] = {0.0}, acc3[1] = {-1.0};  // minima as maxima of the negated values
  for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) {
    c.z[i] = c.xp[i];
    if ((c.freef[i] || unc) && P.nonneg) {
      const double dk = c.r[i];
      if (dk < 0.0) {
        const double t2 = -c.z[i];
        acc3[0] = fmax(acc3[0], t2 >= 0.0 ? 0.0 : -(t2 / dk));
      }
    }
  }
  if (!lb_reduce(c, zero, acc3)) return -9;
  const double alpha = -c.red[1];
  __syncthreads();
  double acc4[1] = {-(double)n};
  if (alpha < 1.0) {
    for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) {
      if ((c.freef[i] || unc) && P.nonneg && c.r[i] < 0.0) {
        const double t2 = -c.z[i];
        const double v = t2 >= 0.0 ? 0.0 : t2 / c.r[i];
        if (v == alpha) acc4[0] = fmax(acc4[0], -(double)i);
      }
    }
    zero[0] = 0.0;
    if (!lb_reduce(c, zero, acc4)) return -9;
  }
  const int ibd = alpha < 1.0 ? -(int)c.red[1] : -1;
  __syncthreads();
  for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) {
    if (c.freef[i] || unc) {
      if (i == ibd) {
        c.z[i] = 0.0;
        c.r[i] = 0.0;
      }
      c.z[i] += alpha * c.r[i];
    }
  }
  __syncthreads();
  return 0;
}

// ---------------------------------------------------------------------------
// mainlb control flow (lbfgsb.f:287-1003) between function evaluations
// ---------------------------------------------------------------------------
enum { LB_RET_DONE = 0, LB_RET_FG = 1, LB_RET_RESTART = 2, LB_RET_ABORT = -9 };

template <typename SY>
__device__ int lb_abort(LbCtxT<SY>& c) {
  if (threadIdx.x == 0) {
    c.S->error = 1;
    c.S->task = LB_TASK_ERROR;
    c.S->done = 1;
  }
  __syncthreads();
  return LB_RET_DONE;
}

// x = t + stp d, or z when stp == 1 (lnsrlb, lbfgsb.f:2562-2570); at the start
// of a line search also r = g
template <typename SY>
__device__ void lb_set_trial_x(LbCtxT<SY>& c, bool start) {
  const double stp = c.S->stp;
  constexpr int U = 4;
  const int bd = blockDim.x;
  for (int i0 = c.lo + threadIdx.x; i0 < c.hi; i0 += U * bd) {
    double v[U], gi[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * bd;
      v[u] = i >= c.hi ? 0.0 : (stp == 1.0) ? c.z[i] : stp * c.d[i] + c.t[i];
      gi[u] = start && i < c.hi ? c.gv[i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * bd;
      if (i >= c.hi) continue;
      c.x[i] = v[u];
      if (start) c.r[i] = gi[u];
    }
  }
  __syncthreads();
}

// "info /= 0 or iback >= 20" branch of mainlb (lbfgsb.f:888-920)
template <typename SY>
__device__ int lb_ls_fail(LbCtxT<SY>& c, bool restore) {
  for (int i = c.lo + threadIdx.x; restore && i < c.hi; i += blockDim.x) {
    c.x[i] = c.t[i];
    c.gv[i] = c.r[i];
  }
  __shared__ int res_s;
  if (threadIdx.x == 0) {
    LbState& S = *c.S;
    S.f = S.fold;
    if (S.col == 0) {
      if (S.info == 0) {
        S.info = -9;
        S.nfgv--;
        S.ifun--;
        S.iback--;
      }
      S.task = LB_TASK_ABNORMAL;
      S.iter++;
      S.done = 1;
      res_s = LB_RET_DONE;
    } else {
      if (S.info == 0) S.nfgv--;
      reset_memory(S);
      res_s = LB_RET_RESTART;
    }
  }
  __syncthreads();
  const int r = res_s;
  __syncthreads();
  return r;
}

// label 555 + the first part of lnsrlb (lbfgsb.f:2480-2575)
template <typename SY>
__device__ __noinline__ int lb_lnsrch_start(LbCtxT<SY>& c, bool ready) {
  LbState& S = *c.S;
  const bool bounded_steps = S.cnstnd && S.iter > 0;
  // gd, dtd; (unused), -stpmx (maxima): the places lb_cmprlb_subsm leaves them in
  double acc[2] = {0.0, 0.0}, stm[2] = {0.0, -1.0e10};
  constexpr int U = 2;  // elements in flight per thread
  const int bd = blockDim.x;
  for (int i0 = ready ? c.hi : c.lo + threadIdx.x; i0 < c.hi; i0 += U * bd) {
    double zv[U], xv[U], gi[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * bd;
      const bool in = i < c.hi;
      zv[u] = in ? c.z[i] : 0.0;
      xv[u] = in ? c.x[i] : 0.0;
      gi[u] = in ? c.gv[i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * bd;
      if (i >= c.hi) continue;
      const double di = zv[u] - xv[u];
      c.d[i] = di;
      c.t[i] = xv[u];
      acc[1] += di * di;
      acc[0] += gi[u] * di;
      if (bounded_steps && c.P->nonneg && di < 0.0) {
        const double a2 = -xv[u];  // l - x with l = 0
        stm[1] = fmax(stm[1], a2 >= 0.0 ? 0.0 : -(a2 / di));
      }
    }
  }
  if (!ready && !lb_reduce(c, acc, stm)) return LB_RET_ABORT;
  __shared__ int act_s;
  if (threadIdx.x == 0) {
    S.dtd = c.red[1];
    S.dnorm = sqrt(S.dtd);
    S.stpmx = 1.0e10;
    if (S.cnstnd) S.stpmx = (S.iter == 0) ? 1.0 : -c.red[3];
    S.stp = (S.iter == 0 && !S.boxed) ? fmin(1.0 / S.dnorm, S.stpmx) : 1.0;
    S.fold = S.f;
    S.ifun = 0;
    S.iback = 0;
    S.csave = CS_START;
    S.gd = c.red[0];
    S.gdold = S.gd;
    if (S.gd >= 0.0) {
      S.info = -4;  // ascent direction in projection
      act_s = 0;
    } else {
      d_dcsrch(S, S.f, S.gd, 0.0, S.stpmx);
      S.xstep = S.stp * S.dnorm;
      S.ifun++;
      S.nfgv++;
      S.iback = S.ifun - 1;
      act_s = 1;
    }
  }
  __syncthreads();
  const int act = act_s;
  __syncthreads();
  if (!act) {
    const int r = lb_ls_fail(c, false);  // x and g have not changed yet
    return r == LB_RET_RESTART ? LB_RET_RESTART : LB_RET_DONE;
  }
  lb_set_trial_x(c, true);
  if (threadIdx.x == 0) S.task = LB_TASK_FG_LN;
  __syncthreads();
  return LB_RET_FG;
}

// label 222 onwards: Cauchy point, subspace minimisation, line-search start
template <typename SY>
__device__ __noinline__ int lb_iter(LbCtxT<SY>& c) {
  LbState& S = *c.S;
  for (int guard = 0; guard < 4; ++guard) {
    if (threadIdx.x == 0) S.iword = -1;
    __syncthreads();
    if (!S.cnstnd && S.col > 0) {
      for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) c.z[i] = c.x[i];
      if (threadIdx.x == 0) {
        S.wrk = S.updatd;
        S.nseg = 0;
      }
      __syncthreads();
    } else {
      c.prof->mark(PR_LB_POST);
      const int rc = lb_cauchy(c);
      c.prof->mark(PR_CAUCHY);
      if (rc == -2) return lb_abort(c);
      if (rc != 0) {
        if (threadIdx.x == 0) reset_memory(S);
        __syncthreads();
        continue;
      }
      if (threadIdx.x == 0) S.nintol += S.nseg;
      __syncthreads();
    }
    bool ls_ready = false;
    if (S.nfree != 0 && S.col != 0) {
      if (S.wrk) {
        c.prof->mark(PR_LB_POST);
        const int rc = lb_formk(c);
        c.prof->mark(PR_FORMK);
        if (rc == -9) return lb_abort(c);
        if (rc != 0) {
          if (threadIdx.x == 0) reset_memory(S);
          __syncthreads();
          continue;
        }
      }
      c.prof->mark(PR_LB_POST);
      const int rc = lb_cmprlb_subsm(c, ls_ready);
      c.prof->mark(PR_SUBSM);
      if (rc == -9) return lb_abort(c);
      if (rc != 0) {
        if (threadIdx.x == 0) reset_memory(S);
        __syncthreads();
        continue;
      }
    }
    c.prof->mark(PR_LB_POST);
    const int r = lb_lnsrch_start(c, ls_ready);
    c.prof->mark(PR_LNSRCH);
    if (r == LB_RET_ABORT) return lb_abort(c);
    if (r == LB_RET_RESTART) continue;
    return r;
  }
  return lb_abort(c);  // repeated restarts: not reachable with an empty memory
}

// Called after every function/gradient evaluation with the group-reduced
// f, g.d and projected-gradient norm.  Returns LB_RET_FG when x holds the next
// point to evaluate, LB_RET_DONE when the solve is over.
template <typename SY>
__device__ __noinline__ int lb_after_fg(LbCtxT<SY>& c, double f, double gd_fg, double sbg) {
  LbState& S = *c.S;
  const ProbDesc& P = *c.P;
  const int m = c.m;
  __shared__ int act_s;
  if (threadIdx.x == 0) {
    S.f = f;
    S.nfg_total++;
  }
  __syncthreads();
  if (S.task == LB_TASK_FG_START) {
    if (threadIdx.x == 0) {
      S.nfgv = 1;
      S.sbgnrm = sbg;
      if (S.sbgnrm <= P.pgtol) {
        S.task = LB_TASK_CONV;
        S.done = 1;
      }
    }
    __syncthreads();
    if (S.done) return LB_RET_DONE;
    return lb_iter(c);
  }
  // FG_LN: lnsrlb from label 556
  if (threadIdx.x == 0) {
    S.gd = gd_fg;
    d_dcsrch(S, S.f, S.gd, 0.0, S.stpmx);
    S.xstep = S.stp * S.dnorm;
    if (S.csave != CS_CONV && S.csave != CS_WARN) {
      S.ifun++;
      S.nfgv++;
      S.iback = S.ifun - 1;
      act_s = (S.iback >= 20) ? 2 : 1;
    } else {
      act_s = 0;
    }
  }
  __syncthreads();
  const int act = act_s;
  __syncthreads();
  if (act == 1) {
    lb_set_trial_x(c, false);
    return LB_RET_FG;
  }
  if (act == 2) {
    const int r = lb_ls_fail(c, true);
    return r == LB_RET_RESTART ? lb_iter(c) : LB_RET_DONE;
  }
  // NEW_X: iteration finished (lbfgsb.f:931-944), driver test, label 777
  if (threadIdx.x == 0) {
    S.iter++;
    S.sbgnrm = sbg;
    if (c.g->rank == 0 && S.iter - 1 < P.niter + 2) c.trace[S.iter - 1] = S.f;
    if (S.f <= P.ftarget) {
      S.task = LB_TASK_TARGET;  // requested objective reached (no reference counterpart)
      S.done = 1;
    } else if (S.iter > P.niter) {
      S.task = LB_TASK_STOP;  // fftim2d.f90:324-325
      S.done = 1;
    } else if (S.sbgnrm <= P.pgtol) {
      S.task = LB_TASK_CONV;
      S.done = 1;
    } else {
      const double ddum = fmax(fabs(S.fold), fmax(fabs(S.f), 1.0));
      if ((S.fold - S.f) <= S.tol * ddum) {
        S.task = LB_TASK_CONV;
        S.done = 1;
      }
    }
    if (!S.done) {
      double dr, dd;
      if (S.stp == 1.0) {
        dr = S.gd - S.gdold;
        dd = -S.gdold;
      } else {
        dr = (S.gd - S.gdold) * S.stp;
        dd = -S.gdold * S.stp;
      }
      S.wa[0] = dr;  // keep dr for matupd below
      if (dr <= S.epsmch * dd) {
        S.nskip++;
        S.updatd = 0;
        act_s = 0;
      } else {
        S.updatd = 1;
        S.iupdat++;
        if (S.iupdat <= m) {
          S.col = S.iupdat;
          S.itail = (S.head + S.iupdat - 2) % m + 1;
        } else {
          S.itail = S.itail % m + 1;
          S.head = S.head % m + 1;
        }
        act_s = 1;
      }
    }
  }
  __syncthreads();
  if (S.done) return LB_RET_DONE;
  if (act_s) {
    // matupd (lbfgsb.f:2584-2670) fused with r = g - r, d = stp d and rr
    const int n = c.n, itail = S.itail - 1;
    const double sc = (S.stp == 1.0) ? 1.0 : S.stp;
    // per-column partial sums in registers: the column loops are unrolled
    // to the largest memory with a guard, so no array is indexed at run time
    double rr_acc = 0.0, ay[SMILI_MAXM_DEV], as[SMILI_MAXM_DEV];
#pragma unroll
    for (int j = 0; j < SMILI_MAXM_DEV; ++j) ay[j] = as[j] = 0.0;
    // FP32 (64 registers): one element at a time, its loads where they are
    // used.  With all 13 loads of an element before its arithmetic every
    // stage of the launch came out slower: 74 problems of 256 x 256, 20
    // iterations, 74.5 ms against 72.8; 0.5 to 1.5 % at 1 to 12 CTAs per problem.
    if constexpr (sizeof(SY) == 4) {
      for (int i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) {
        const double ri = c.gv[i] - c.r[i];
        const double di = c.d[i] * sc;
        rr_acc += ri * ri;
#pragma unroll
        for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
          if (j < m) {
            ay[j] += di * ld_wy(c, (size_t)j * n + i);
            as[j] += ld_ws(c, (size_t)j * n + i) * di;
          }
        }
        st_sy(c, (size_t)itail * n + i, di, ri);
        c.r[i] = ri;
        c.d[i] = di;
      }
    } else {
      constexpr int U = 2;  // elements in flight per thread
      const int bd = blockDim.x;
      for (int i0 = c.lo + threadIdx.x; i0 < c.hi; i0 += U * bd) {
        double ri[U], di[U];
        SY wy[U][SMILI_MAXM_DEV], ws[U][SMILI_MAXM_DEV];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = i0 + u * bd;
          const bool in = i < c.hi;
          ri[u] = in ? c.gv[i] - c.r[i] : 0.0;
          di[u] = in ? c.d[i] * sc : 0.0;
#pragma unroll
          for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
            wy[u][j] = in && j < m ? c.wy[(size_t)j * n + i] : (SY)0;
            ws[u][j] = in && j < m ? c.ws[(size_t)j * n + i] : (SY)0;
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = i0 + u * bd;
          if (i >= c.hi) continue;
          rr_acc += ri[u] * ri[u];
#pragma unroll
          for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
            if (j < m) {
              ay[j] += di[u] * (double)wy[u][j];
              as[j] += (double)ws[u][j] * di[u];
            }
          }
          st_sy(c, (size_t)itail * n + i, di[u], ri[u]);
          c.r[i] = ri[u];
          c.d[i] = di[u];
        }
      }
    }
    double acc[16];
#pragma unroll
    for (int j = 0; j < SMILI_MAXM_DEV; ++j) {
      acc[j] = ay[j];
      acc[SMILI_MAXM_DEV + j] = as[j];
    }
    acc[12] = rr_acc;
#pragma unroll
    for (int j = 13; j < 16; ++j) acc[j] = 0.0;
    const double none[1] = {0.0};
    if (!lb_reduce(c, acc, none)) return lb_abort(c);
    if (threadIdx.x < 32) {
      const double rr = c.red[12], dr = S.wa[0];
      const int col = S.col, lane = threadIdx.x;
      // shift the matrices when the oldest pair leaves, then the new row and column
      constexpr int NE = (SMILI_MAXM_DEV * SMILI_MAXM_DEV + 31) / 32;
      double ns[NE], ny[NE];
#pragma unroll
      for (int q = 0; q < NE; ++q) {
        const int e = lane + 32 * q, i = e % col, j = e / col;
        if (e >= col * col) continue;
        const int sh = (S.iupdat > m && i < col - 1 && j < col - 1) ? 1 + m : 0;
        ns[q] = S.ss[i + m * j + sh];
        ny[q] = S.sy[i + m * j + sh];
        if (j == col - 1 && i < col - 1) ns[q] = c.red[SMILI_MAXM_DEV + (S.head - 1 + i) % m];
        if (i == col - 1 && j < col - 1) ny[q] = c.red[(S.head - 1 + j) % m];
        if (i == col - 1 && j == col - 1) {
          ns[q] = (S.stp == 1.0) ? S.dtd : S.stp * S.stp * S.dtd;
          ny[q] = dr;
        }
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < NE; ++q) {
        const int e = lane + 32 * q, i = e % col, j = e / col;
        if (e >= col * col) continue;
        if (i <= j) S.ss[i + m * j] = ns[q];
        if (i >= j) S.sy[i + m * j] = ny[q];
      }
      if (lane == 0) S.theta = rr / dr;
      __syncwarp();
      if (warp_formt(S, m) != 0 && lane == 0) reset_memory(S);
    }
    __syncthreads();
  }
  return lb_iter(c);
}
