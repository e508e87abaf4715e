// Common device helpers: complex arithmetic, block reductions and the
// intra-group barrier of the persistent solver.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "layout.h"

// CTA shape of the solver kernel per precision.  FP32 runs 512 threads
// (two CTAs per SM at 64 registers: 32 resident warps to hide the latency of
// the gather-heavy stages), FP64 256 threads (two CTAs per SM at 128
// registers; its shared-memory staging is twice as large).  Device code
// strides by blockDim.x; buffers shared by both shapes are sized for the
// larger one.
template <typename R>
struct Shape {
  static constexpr int threads = sizeof(R) == 4 ? 512 : 256;
  static constexpr int warps = threads / 32;
  static constexpr int min_blocks = 2;
};
#define SMILI_MAX_THREADS 512
#define SMILI_MAX_WARPS (SMILI_MAX_THREADS / 32)

template <typename R>
struct cpx {
  R x, y;
};
template <typename R>
__device__ __forceinline__ cpx<R> cmk(R a, R b) {
  cpx<R> c;
  c.x = a;
  c.y = b;
  return c;
}
template <typename R>
__device__ __forceinline__ cpx<R> cadd(cpx<R> a, cpx<R> b) {
  return cmk(a.x + b.x, a.y + b.y);
}
template <typename R>
__device__ __forceinline__ cpx<R> csub(cpx<R> a, cpx<R> b) {
  return cmk(a.x - b.x, a.y - b.y);
}
template <typename R>
__device__ __forceinline__ cpx<R> cmul(cpx<R> a, cpx<R> b) {
  return cmk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename R>
__device__ __forceinline__ cpx<R> cscale(cpx<R> a, R s) {
  return cmk(a.x * s, a.y * s);
}
// multiply by +i
template <typename R>
__device__ __forceinline__ cpx<R> cmul_i(cpx<R> a) {
  return cmk(-a.y, a.x);
}

template <typename T>
__device__ __forceinline__ T* at(char* base, int64_t off) {
  return reinterpret_cast<T*>(base + off);
}

// ---------------------------------------------------------------------------
// Group context: the CTAs that cooperate on one problem.
// ---------------------------------------------------------------------------
struct GroupCtx {
  int rank, G;
  unsigned* bar;       // arrivals of the group's CTAs since the launch began (never reset)
  unsigned target;     // arrival count that completed the last barrier
  double* red_part;    // [2][G][redk] partials of the group reductions, used in turn
  int redk;            // values one CTA may contribute to a reduction
  int parity;          // half of red_part the next reduction uses
  int* abort_flag;     // global abort (set on a barrier timeout)
  long long spin_limit;
};

// largest reduction: the Gram blocks of formk, 2 m (m + 1) / 2 + 2 m m at m = 6
#define SMILI_REDK 128
// reductions of one evaluation (no L-BFGS-B step): at most 16 sums and one maximum
#define SMILI_REDK_FG 32

// Spin budget of one barrier wait.  A healthy barrier completes in
// microseconds; the limit only ends a wait that can never complete.
#define SMILI_SPIN_LIMIT (1LL << 24)

__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Wait until the group's arrival count reaches g.target (compared modulo
// 2^32).  The polls are relaxed and one fence follows them: an acquire load
// per poll would drop the SM's L1 lines each time, also those of the other
// CTA on the SM (an FP32 batch ran 4 % slower).  Polls without sleeping for a short while (barriers normally
// complete within microseconds), then backs off; gives up after spin_limit
// polls or when another CTA aborted.
__device__ __forceinline__ bool wait_arrivals(GroupCtx& g) {
  long long spins = 0;
  while ((int)(ld_relaxed(g.bar) - g.target) < 0) {
    ++spins;
    if (spins > g.spin_limit || ((spins & 63) == 0 && *((volatile int*)g.abort_flag))) {
      atomicExch(g.abort_flag, 1);
      return false;
    }
    if (spins > 4096) __nanosleep(64);
  }
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  return true;
}

// Group barrier.  Returns false when the wait timed out (abort flag set):
// callers stop work.  The count only grows, so a CTA's arrival is one release
// reduction (cumulative over the block's earlier writes, which bar.sync
// orders before it) and the wait polls that same count: two trips to L2.  A
// barrier whose last arriver resets a counter and then releases a generation
// takes four: 2.4 against 1.2 us at 2 to 64 CTAs, 2.8 against 1.5 at 296 (B200).
__device__ bool group_sync(GroupCtx& g) {
  __syncthreads();
  if (g.G == 1) return true;
  __shared__ int ok_s;
  g.target += (unsigned)g.G;
  if (threadIdx.x == 0) {
    red_release_add(g.bar, 1u);
    ok_s = wait_arrivals(g) ? 1 : 0;
  }
  __syncthreads();
  return ok_s != 0;
}

// ---------------------------------------------------------------------------
// Reductions over the group (deterministic, the same value in every CTA)
// ---------------------------------------------------------------------------
// One FP64 tensor-core product D = A B + D of an 8x4 by 4x8 tile
// (mma.sync m8n8k4 f64).  Lane l holds A[l/4][l%4], B[l%4][l/4] and
// D[l/4][2(l%4) + {0,1}].
__device__ __forceinline__ void dmma_884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Maximum over the warp (as fmax: a NaN only where all are): the doubles as
// unsigned integers of the same order, their words one after the other.
__device__ __forceinline__ double warp_max(double a) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a), top = 1ULL << 63;
  const unsigned long long k = a != a ? 0 : ((b & top) ? ~b : (b | top));
  const unsigned hi = (unsigned)(k >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)k : 0u);
  const unsigned long long m = ((unsigned long long)mh << 32) | ml;
  return __longlong_as_double((long long)((m & top) ? (m & ~top) : ~m));
}

// Sum (or maximum) of one value over the rows r0, r0 + step, ... < G, D loads
// in flight.
template <int D>
__device__ __forceinline__ double fold_rows(const double* col, int r0, int step, int G, int redk, bool sum) {
  const double none = sum ? 0.0 : -INFINITY;
  double a = none;
#pragma unroll 1
  for (int r = r0; r < G; r += D * step) {
    double v[D];
#pragma unroll
    for (int q = 0; q < D; ++q) v[q] = r + q * step < G ? __ldcg(col + (size_t)(r + q * step) * redk) : none;
#pragma unroll
    for (int q = 0; q < D; ++q) a = sum ? a + v[q] : fmax(a, v[q]);
  }
  return a;
}

// Second half of a group reduction: every CTA has its partials (ns sums,
// then maxima, K in all) in its row of the current half of red_part, or in
// out when G == 1.  After the barrier each CTA combines all rows itself, in
// the same order: T / Kp slices of ranks in parallel, then the slices.  (A
// last arriver that combines the rows one after another and publishes the
// result adds a second barrier trip and a load latency per row.)  The halves
// alternate, so a row is rewritten only after a later barrier has shown that
// every CTA has read it.  scratch: blockDim.x doubles of shared memory.
__device__ __noinline__ bool group_combine(GroupCtx& g, int K, int ns, double* out, double* scratch) {
  if (g.G == 1) {
    __syncthreads();
    return true;
  }
  const double* part = g.red_part + (size_t)g.parity * g.G * g.redk;
  g.parity ^= 1;
  if (!group_sync(g)) return false;
  const int sh = K <= 16 ? 4 : (K <= 32 ? 5 : (K <= 64 ? 6 : 7));
  const int k = threadIdx.x & ((1 << sh) - 1), sl = threadIdx.x >> sh, S = blockDim.x >> sh;
  const bool sum = k < ns;
  double a = sum ? 0.0 : -INFINITY;
  if (k < K) {
    const double* col = part + k;
    if (g.G <= 4 * S) a = fold_rows<4>(col, sl, S, g.G, g.redk, sum);  // one trip, little code
    else a = fold_rows<8>(col, sl, S, g.G, g.redk, sum);
  }
  scratch[threadIdx.x] = a;
  __syncthreads();
  if (threadIdx.x < K) {
    const int n = min(S, g.G);
    double t = scratch[threadIdx.x];
#pragma unroll 4
    for (int q = 1; q < n; ++q) {
      const double v = scratch[(q << sh) + threadIdx.x];
      t = sum ? t + v : fmax(t, v);
    }
    out[threadIdx.x] = t;
  }
  __syncthreads();
  return true;
}

// doubles of shared scratch the reductions need with T threads: one per
// thread, or up to 40 values per warp
#define SMILI_SCRATCH(T) ((T) / 32 * 40)

// the row this CTA writes before group_combine
__device__ __forceinline__ double* group_row(GroupCtx& g, double* out) {
  return g.G == 1 ? out : g.red_part + ((size_t)g.parity * g.G + g.rank) * g.redk;
}

// Sums of each thread's s[0..ns) and maxima of its x[0..nx) over the block,
// into row[0..ns) and row[ns..ns+nx); ns + nx <= 40.  A warp sums a value with
// a tensor-core product by ones: 8 lanes per product, two exchanges for eight
// values.  One routine with rolled loops for every reduction of the kernel:
// each size unrolled (31 exchanges of two words for 16 values) spent most of
// its time on fetching its instructions, 6.6 us per group sum of 16 values and
// 4 maxima where the barrier in it takes 2 (B200).
__device__ __noinline__ void block_partials(const double* s, int ns, const double* x, int nx, double* row,
                                            double* scratch) {
  const int K = ns + nx, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5, q = lane >> 2;
  double* w = scratch + wid * K;
#pragma unroll 1
  for (int v0 = 0; v0 < ns; v0 += 8) {
    const int nv = min(8, ns - v0);
    double r = 0.0;
#pragma unroll 4
    for (int i = 0; i < nv; ++i) {
      double d[2] = {0.0, 0.0};
      dmma_884(d, 1.0, s[v0 + i]);
      const double t = d[0] + d[1];
      r = q == i ? t : r;
    }
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    if ((lane & 3) == 0 && q < nv) w[v0 + q] = r;
  }
#pragma unroll 1
  for (int k = 0; k < nx; ++k) {
    const double a = warp_max(x[k]);
    if (lane == 0) w[ns + k] = a;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double a = scratch[threadIdx.x];
#pragma unroll 4
    for (int v = 1; v < nw; ++v) {
      const double b = scratch[v * K + threadIdx.x];
      a = (int)threadIdx.x < ns ? a + b : fmax(a, b);
    }
    row[threadIdx.x] = a;
  }
}

// Group-wide sums of s[0..ns) and maxima of x[0..nx) over all threads:
// out[0..ns) and out[ns..ns+nx) (shared) in every CTA.
// scratch: SMILI_SCRATCH(blockDim.x) doubles of shared memory.
__device__ __noinline__ bool group_reduce(GroupCtx& g, const double* s, int ns, const double* x, int nx, double* out,
                                          double* scratch) {
  block_partials(s, ns, x, nx, group_row(g, out), scratch);
  return group_combine(g, ns + nx, ns, out, scratch);
}

// ---------------------------------------------------------------------------
// Stage profiler: CTA 0 (thread 0) accumulates the time between consecutive
// marks into acc[stage] (nanoseconds, from %globaltimer).  Off when acc is 0.
// ---------------------------------------------------------------------------
enum {
  PR_F1 = 0, PR_F2, PR_F3, PR_F4, PR_F5, PR_F6, PR_F7, PR_F8, PR_LB_POST, PR_CAUCHY, PR_FORMK,
  PR_SUBSM, PR_LNSRCH, PR_INIT, PR_OTHER, PR_COUNT, PR_C_SEL, PR_C_GATHER, PR_C_SORT, PR_C_SCAN,
  PR_C_ROUNDS, PR_NSTAGE
};

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

struct Prof {
  unsigned long long* acc;
  unsigned long long t;
  __device__ void start() {
    if (acc) t = gtimer();
  }
  __device__ void mark(int st) {
    if (acc) {
      const unsigned long long now = gtimer();
      acc[st] += now - t;
      t = now;
    }
  }
  __device__ void count(int st) {
    if (acc) acc[st] += 1;
  }
};
