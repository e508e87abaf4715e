// Points of a bare transform sorted on the device.
//
// nufft_fwd_real and nufft_adj_real1d get their points in the caller's order
// and use them once.  Sorted on one host core, 200 000 points took 12 of the
// call's 14 ms; as a counting sort here (count, scan, scatter, work items)
// they take 0.1 ms beside the copy of u and v.  Sorted by bin x bin tile of
// the band and inside a tile by cell, as the host sorts the points of a
// solve; the order inside a cell is not fixed (a forward transform does not
// depend on it, an adjoint adds its tiles with atomics anyway).
// Bound by the launches: 16 bytes per point read, 40 written.
#pragma once

// where a bare transform's sort keeps its arrays (arena offsets)
struct UvSort {
  int64_t o_u = 0, o_v = 0;      // as given (double); a forward transform's result afterwards
  int64_t o_cre = 0, o_cim = 0;  // visibilities of an adjoint transform (double)
  int64_t o_key = 0, o_perm = 0, o_hist = 0, o_sums = 0;
  int nb1 = 0, ntile = 0, nkey = 0;  // tiles of the band per row and in all, cells in all
};

constexpr int UVSORT_T = 1024, UVSORT_CHUNK = 4 * UVSORT_T;  // threads, cells per scan block

// exclusive sum of v over the block's UVSORT_T threads; total in every thread
__device__ __forceinline__ int block_exclusive(int v, int& total) {
  __shared__ int ws[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int s = v;
#pragma unroll
  for (int q = 1; q < 32; q <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, s, q);
    if (lane >= q) s += t;
  }
  if (lane == 31) ws[warp] = s;
  __syncthreads();
  if (warp == 0) {
    int t = ws[lane];
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, t, q);
      if (lane >= q) t += o;
    }
    ws[lane] = t;
  }
  __syncthreads();
  total = ws[31];
  const int before = warp ? ws[warp - 1] : 0;
  __syncthreads();
  return before + s - v;
}

// fine-grid coordinate in the kernel precision, as the host computes it
template <typename R>
__device__ __forceinline__ R grid_coord(double u, int nf) {
  return (R)(u * nf / (2.0 * 3.14159265358979323846));
}

template <typename R>
__global__ void uvsort_count(const ProbDesc* desc, char* base, UvSort q) {
  const ProbDesc& P = *desc;
  const double *u = at<double>(base, q.o_u), *v = at<double>(base, q.o_v);
  int *key = at<int>(base, q.o_key), *hist = at<int>(base, q.o_hist);
  const R half = (R)0.5 * (R)P.w;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < P.nuv; j += gridDim.x * blockDim.x) {
    const int c1 = imod((int)ceil(grid_coord<R>(u[j], P.nf1) - half) - P.b1s, P.nf1);  // inside the band
    const int c2 = imod((int)ceil(grid_coord<R>(v[j], P.nf2) - half) - P.b2s, P.nf2);
    const int t1 = c1 / P.bin, t2 = c2 / P.bin;
    const int k = ((t2 * q.nb1 + t1) * P.bin + (c2 - t2 * P.bin)) * P.bin + (c1 - t1 * P.bin);
    key[j] = k;
    atomicAdd(hist + k, 1);
  }
}

// sums of the chunks of UVSORT_CHUNK cells
__global__ void __launch_bounds__(UVSORT_T) uvsort_sums(char* base, UvSort q) {
  const int* hist = at<int>(base, q.o_hist);
  int s = 0, total;
  for (int k = 0; k < 4; ++k) {
    const int i = blockIdx.x * UVSORT_CHUNK + k * UVSORT_T + threadIdx.x;
    if (i < q.nkey) s += hist[i];
  }
  block_exclusive(s, total);
  if (threadIdx.x == 0) at<int>(base, q.o_sums)[blockIdx.x] = total;
}

// hist -> first position of every cell.  Every block adds up the chunks before
// its own (about 1000 of them at most: 2056^2 cells).
__global__ void __launch_bounds__(UVSORT_T) uvsort_scan(char* base, UvSort q) {
  int* hist = at<int>(base, q.o_hist);
  const int* sums = at<int>(base, q.o_sums);
  int b = 0, first, total;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += UVSORT_T) b += sums[i];
  block_exclusive(b, first);
  const int i0 = blockIdx.x * UVSORT_CHUNK + 4 * threadIdx.x;
  int h[4], s = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    h[k] = i0 + k < q.nkey ? hist[i0 + k] : 0;
    s += h[k];
  }
  int at_ = first + block_exclusive(s, total);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (i0 + k < q.nkey) hist[i0 + k] = at_;
    at_ += h[k];
  }
}

// points to their places; afterwards hist[k] is the end of cell k
template <typename R>
__global__ void uvsort_scatter(const ProbDesc* desc, char* base, UvSort q) {
  const ProbDesc& P = *desc;
  const double *u = at<double>(base, q.o_u), *v = at<double>(base, q.o_v);
  const double *cre = at<double>(base, q.o_cre), *cim = at<double>(base, q.o_cim);
  const int* key = at<int>(base, q.o_key);
  int *hist = at<int>(base, q.o_hist), *perm = at<int>(base, q.o_perm);
  R *su = at<R>(base, P.o_u), *sv = at<R>(base, P.o_v);
  cpx<R>* contrib = at<cpx<R>>(base, P.o_contrib);
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < P.nuv; j += gridDim.x * blockDim.x) {
    const int p = atomicAdd(hist + key[j], 1);
    perm[p] = j;
    su[p] = grid_coord<R>(u[j], P.nf1);
    sv[p] = grid_coord<R>(v[j], P.nf2);
    if (q.o_cre) contrib[p] = cmk<R>((R)cre[j], (R)(-cim[j]));  // c = (Re, -Im)
  }
}

// spreading work items: <= 128 consecutive points of one tile.  One block.
__global__ void __launch_bounds__(UVSORT_T) uvsort_items(ProbDesc* desc, char* base, UvSort q) {
  const int bin = desc->bin, cells = bin * bin;
  const int* ends = at<int>(base, q.o_hist);
  int4* items = at<int4>(base, desc->o_items);
  int done = 0;
  for (int t0 = 0; t0 < q.ntile; t0 += UVSORT_T) {
    const int t = t0 + (int)threadIdx.x;
    int a = 0, e = 0;
    if (t < q.ntile) {
      a = t ? ends[t * cells - 1] : 0;
      e = ends[t * cells + cells - 1];
    }
    int total;
    int o = done + block_exclusive((e - a + 127) / 128, total);
    for (int j = a; j < e; j += 128, ++o)
      items[o] = make_int4(j, min(j + 128, e), t / q.nb1 * bin, t % q.nb1 * bin);
    done += total;
  }
  if (threadIdx.x == 0) desc->nitems = done;
}

// a forward transform's visibilities in the caller's order, over u and v
template <typename R>
__global__ void uvsort_result(const ProbDesc* desc, char* base, UvSort q) {
  const cpx<R>* V = at<cpx<R>>(base, desc->o_V);
  const int* perm = at<int>(base, q.o_perm);
  double *re = at<double>(base, q.o_u), *im = at<double>(base, q.o_v);
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < desc->nuv; j += gridDim.x * blockDim.x) {
    re[perm[j]] = (double)V[j].x;
    im[perm[j]] = (double)V[j].y;
  }
}
