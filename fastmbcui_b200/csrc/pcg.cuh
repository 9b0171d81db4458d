// Batched PCG kernels (kl_chol.cu:891-1088 for one column, here R columns at
// once with per-column alpha, beta and stopping).  Vectors are n x R
// row-major in the new (fine-to-coarse) order, arithmetic type T; every PCG
// scalar and every dot product is FP64 (partial sums per block, then one
// deterministic reduction).  Elementwise kernels use a 2-D block: x over RHS
// columns, y over points.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mbc {

// COL_STAGNANT: replacement mode only -- three consecutive replacements
// found the true residual less than halved: the FP32 recursion has reached
// its attainable accuracy and the column is finished in FP64.
enum ColStatus : int32_t { COL_ACTIVE = -1, COL_OK = 0, COL_MAXIT = 1, COL_BREAKDOWN = 2, COL_STAGNANT = 3 };

struct PcgScalars {
  double *rz, *b2, *thr, *alpha, *beta, *rr, *pt;
  double *rr_ref;  // residual replacement: |r|^2 at the last replacement
  int32_t *stall;  // residual replacement: consecutive replacements without progress
  int32_t *status, *iters;
  int32_t *done;   // 1 when no column is active
  int32_t *want;   // residual replacement requested (set by RED_CHECK)
  int32_t *tick;   // [blocks arrived, any column active] of the reduction in flight; zero between kernels
  int32_t maxit;
  double tol2;
  double drop2;    // > 0: replacement mode, replace once |r|^2 < drop2 * rr_ref
  int32_t stall_check;  // replacement mode: 1 = mark columns stagnant (COL_STAGNANT)
};

enum ReduceMode : int32_t {
  RED_NONE = -1,
  RED_STORE = 0,   // out[c] = s
  RED_INIT_B = 1,  // b2 = s, thr = tol^2 s, status ACTIVE unless |b|^2 < 1e-16
  RED_ALPHA = 2,   // alpha = rz / s (breakdown if s <= 0 or NaN)
  RED_CHECK = 3,   // rr = s, iters++, converge / max-iteration test, done flag
  RED_BETA = 4,    // beta = s / rz, rz = s
  RED_REPLACE = 5  // true |r|^2 after a residual replacement: rr = rr_ref = s, converge test
};

// a column's step for its reduced sum s (one thread)
__device__ __forceinline__ void apply_sum(int32_t mode, int c, double s, const PcgScalars &sc, double *out)
{
  switch (mode) {
    case RED_STORE:
      out[c] = s;
      break;
    case RED_INIT_B:
      sc.b2[c] = s;
      sc.thr[c] = sc.tol2 * s;
      if (sc.rr_ref) sc.rr_ref[c] = s;
      if (sc.stall) sc.stall[c] = 0;
      if (sc.status[c] == COL_ACTIVE && s < 1e-16) {
        sc.status[c] = COL_OK;  // kl_chol.cu:950-953: zero right-hand side
        sc.rr[c] = 0.0;
      }
      break;
    case RED_ALPHA:
      if (sc.status[c] == COL_ACTIVE) {
        sc.pt[c] = s;
        if (!(s > 0.0) || !(sc.rz[c] == sc.rz[c])) {
          sc.status[c] = COL_BREAKDOWN;
          sc.alpha[c] = 0.0;
        } else {
          sc.alpha[c] = sc.rz[c] / s;
        }
      } else {
        sc.alpha[c] = 0.0;
      }
      break;
    case RED_CHECK:
      if (sc.status[c] == COL_ACTIVE) {
        sc.rr[c] = s;
        sc.iters[c] += 1;
        if (!(s == s)) {
          sc.status[c] = COL_BREAKDOWN;
        } else if (sc.drop2 > 0.0) {
          // replacement mode: convergence is only declared on a true
          // FP64 residual, so ask for one
          if (s < sc.thr[c] || s < sc.drop2 * sc.rr_ref[c]) *sc.want = 1;
          if (sc.iters[c] >= sc.maxit) sc.status[c] = COL_MAXIT;
        } else if (s < sc.thr[c]) {
          sc.status[c] = COL_OK;
        } else if (sc.iters[c] >= sc.maxit) {
          sc.status[c] = COL_MAXIT;
        }
      }
      break;
    case RED_REPLACE:
      if (sc.status[c] == COL_ACTIVE || sc.status[c] == COL_MAXIT) {
        const double prev = sc.rr_ref[c];
        sc.rr[c] = s;
        sc.rr_ref[c] = s;
        if (!(s == s)) {
          sc.status[c] = COL_BREAKDOWN;
        } else if (s < sc.thr[c]) {
          sc.status[c] = COL_OK;
        } else if (sc.stall_check) {
          sc.stall[c] = s > 0.25 * prev ? sc.stall[c] + 1 : 0;
          if (sc.stall[c] >= 3 && sc.status[c] == COL_ACTIVE) sc.status[c] = COL_STAGNANT;
        }
      }
      break;
    case RED_BETA:
      if (sc.status[c] == COL_ACTIVE) {
        sc.beta[c] = s / sc.rz[c];
        sc.rz[c] = s;
      } else {
        sc.beta[c] = 0.0;
      }
      break;
  }
}

// Sums of the partials of columns warp0, warp0 + nwarps, ... (lanes over the
// partial blocks, a fixed order) and their steps; returns whether one of them
// is still active.
__device__ __forceinline__ int reduce_columns(int nblk, int R, const double *part, int32_t mode, const PcgScalars &sc,
                                              double *out, int warp0, int nwarps)
{
  const int lane = threadIdx.x + threadIdx.y * blockDim.x & 31;
  int any = 0;
  for (int c = warp0; c < R; c += nwarps) {
    double s = 0.0;
#pragma unroll 4
    for (int b = lane; b < nblk; b += 32) s += __ldcg(part + (size_t)b * R + c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      apply_sum(mode, c, s, sc, out);
      if (sc.status && sc.status[c] == COL_ACTIVE) any = 1;
    }
  }
  return any;
}

__device__ __forceinline__ bool sets_done(int32_t mode)
{
  return mode == RED_CHECK || mode == RED_INIT_B || mode == RED_ALPHA || mode == RED_REPLACE;
}

// 8 columns per block of 256 threads; the last block to finish writes the
// stop flag.
__global__ void __launch_bounds__(256) reduce_kernel(int nblk, int R, const double *__restrict__ part, int32_t mode,
                                                     PcgScalars sc, double *__restrict__ out)
{
  if (mode != RED_INIT_B && mode != RED_STORE && mode != RED_REPLACE && sc.done && *sc.done) return;
  int any = reduce_columns(nblk, R, part, mode, sc, out, blockIdx.x * 8 + (threadIdx.x >> 5), gridDim.x * 8);
  if (!sets_done(mode) || !sc.done) return;
  any = __syncthreads_or(any);
  if (threadIdx.x != 0) return;
  if (any) atomicOr(sc.tick + 1, 1);
  __threadfence();
  if (atomicAdd(sc.tick, 1) == (int)gridDim.x - 1) {
    *sc.done = atomicAdd(sc.tick + 1, 0) ? 0 : 1;
    sc.tick[0] = 0;
    sc.tick[1] = 0;
  }
}

// The reduction inside the kernel that wrote the partials (RED_NONE: left to
// reduce_kernel): the last block to arrive sums them.  For few partials, where
// the launch of a kernel of its own costs more.  The block has 256 threads.
__device__ __forceinline__ void reduce_by_last_block(int nblk, int R, const double *part, int32_t mode,
                                                     const PcgScalars &sc)
{
  if (mode == RED_NONE) return;
  __shared__ int s_last;
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(sc.tick, 1) == (int)(gridDim.x * gridDim.y) - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  int any = reduce_columns(nblk, R, part, mode, sc, nullptr, tid >> 5, 8);
  any = __syncthreads_or(any);
  if (tid == 0) {
    sc.tick[0] = 0;
    if (sets_done(mode)) *sc.done = any ? 0 : 1;
  }
}

// Block reduction over threadIdx.y of one double per thread; thread (x, 0)
// returns the block sum for column x.
__device__ __forceinline__ double block_sum_y(double v, double *red)
{
  const int tx = threadIdx.x, ty = threadIdx.y;
  red[ty * blockDim.x + tx] = v;
  __syncthreads();
  for (int h = blockDim.y / 2; h > 0; h >>= 1) {
    if (ty < h) red[ty * blockDim.x + tx] += red[(ty + h) * blockDim.x + tx];
    __syncthreads();
  }
  return red[tx];
}

// One half of the preconditioner z = L (L^T r): out_j = sum over the entries k
// of row (or column) j of val[k] in[ind[k]], n x R, optionally with the
// partials of rv . out.  L^T walks the columns of L, L its rows (val in row
// order).
// What bounds it: the gathers, by latency in small scenes, whose longest rows
// (the coarse points', hundreds of entries) a thread per row walked alone, by
// L2 traffic in large ones.  A row's entries are spread over the lanes left
// beside its columns (32 / cx, cx the columns' power of two) and over wpr
// warps, four gathers in flight each; blocks stride over the rows, so that
// the partials stay few.
template <typename T, typename LT>
__global__ void __launch_bounds__(256) precond_kernel(int n, int R, int cx, int wpr, const int32_t *__restrict__ ptr,
                                                      const int32_t *__restrict__ ind, const LT *__restrict__ val,
                                                      const T *__restrict__ in, T *__restrict__ out,
                                                      const T *__restrict__ rv, double *__restrict__ part,
                                                      int32_t mode, PcgScalars sc, const int32_t *__restrict__ done)
{
  if (done && *done) return;
  __shared__ T sacc[8][32];
  __shared__ double sdot[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cl = lane & (cx - 1), el = lane / cx, le = 32 / cx;
  const int w = warp % wpr, slot = warp / wpr, rows = 8 / wpr;
  const int c = blockIdx.y * cx + cl;
  const bool col = c < R;
  const int step = le * wpr;
  double d = 0.0;
  for (int base = blockIdx.x * rows; base < n; base += gridDim.x * rows) {
    const int j = base + slot;
    T acc = T(0);
    if (j < n && col) {
      const int k1 = ptr[j + 1];
      int k = ptr[j] + w * le + el;
      for (; k + 3 * step < k1; k += 4 * step) {
        T x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = in[(size_t)ind[k + q * step] * R + c];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc = fma((T)val[k + q * step], x[q], acc);
      }
      T x[3], v[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int kq = k + q * step;
        v[q] = kq < k1 ? (T)val[kq] : T(0);
        x[q] = kq < k1 ? in[(size_t)ind[kq] * R + c] : T(0);
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) acc = fma(v[q], x[q], acc);
    }
    for (int o = cx; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (wpr > 1) {
      sacc[warp][lane] = acc;
      __syncthreads();
      if (w == 0)
        for (int q = 1; q < wpr; ++q) acc += sacc[warp + q][lane];
    }
    if (w == 0 && el == 0 && col && j < n) {
      out[(size_t)j * R + c] = acc;
      if (part) d += (double)rv[(size_t)j * R + c] * (double)acc;
    }
    if (wpr > 1) __syncthreads();
  }
  if (!part) return;
  sdot[warp][lane] = d;  // zero but for the first warp and entry lane of a row
  __syncthreads();
  if (warp == 0 && el == 0 && col) {
    for (int q = wpr; q < 8; q += wpr) d += sdot[q][lane];
    part[(size_t)blockIdx.x * R + c] = d;
  }
  reduce_by_last_block(gridDim.x, R, part, mode, sc);
}

// the values of L in row order
template <typename LT>
__global__ void row_values_kernel(int64_t nnz, const int32_t *__restrict__ rmap, const LT *__restrict__ lval,
                                  LT *__restrict__ lrow)
{
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nnz) lrow[t] = lval[rmap[t]];
}

// part = a . b per block (a, b n x R); blocks stride over the rows
template <typename T>
__global__ void __launch_bounds__(256) dot_partial_kernel(int n, int R, const T *__restrict__ a,
                                                          const T *__restrict__ b, double *__restrict__ part)
{
  extern __shared__ double red[];
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  double d = 0.0;
  if (c < R)
    for (int i = blockIdx.x * blockDim.y + threadIdx.y; i < n; i += gridDim.x * blockDim.y)
      d += (double)a[(size_t)i * R + c] * (double)b[(size_t)i * R + c];
  const double s = block_sum_y(d, red);
  if (threadIdx.y == 0 && c < R) part[(size_t)blockIdx.x * R + c] = s;
}

// x += alpha p; r -= alpha t; part = r . r   (x may be FP64 while p, r are T)
template <typename T, typename XT>
__global__ void __launch_bounds__(256) update_xr_kernel(int n, int R, const double *__restrict__ alpha,
                                                        const T *__restrict__ p, const T *__restrict__ t,
                                                        XT *__restrict__ x, T *__restrict__ r,
                                                        double *__restrict__ part, int32_t mode, PcgScalars sc,
                                                        const int32_t *__restrict__ done)
{
  if (done && *done) return;
  extern __shared__ double red[];
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  double d = 0.0;
  if (c < R) {
    const double a = alpha[c];
    for (int i = blockIdx.x * blockDim.y + threadIdx.y; i < n; i += gridDim.x * blockDim.y) {
      const size_t o = (size_t)i * R + c;
      const XT xv = (XT)((double)x[o] + a * (double)p[o]);
      const T rv = (T)((double)r[o] - a * (double)t[o]);
      x[o] = xv;
      r[o] = rv;
      d += (double)rv * (double)rv;
    }
  }
  const double s = block_sum_y(d, red);
  if (threadIdx.y == 0 && c < R) part[(size_t)blockIdx.x * R + c] = s;
  reduce_by_last_block(gridDim.x, R, part, mode, sc);
}

// p = z + beta p (active columns only)
template <typename T>
__global__ void __launch_bounds__(256) update_p_kernel(int n, int R, const double *__restrict__ beta,
                                                       const int32_t *__restrict__ status, const T *__restrict__ z,
                                                       T *__restrict__ p, const int32_t *__restrict__ done)
{
  if (done && *done) return;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= R || status[c] != COL_ACTIVE) return;
  const double b = beta[c];
  for (int i = blockIdx.x * blockDim.y + threadIdx.y; i < n; i += gridDim.x * blockDim.y) {
    const size_t o = (size_t)i * R + c;
    p[o] = (T)((double)z[o] + b * (double)p[o]);
  }
}

// ---- small helpers --------------------------------------------------------

// dst[P[o], c] = (T) src[o, c]  (original order -> new order, type change)
template <typename S, typename D>
__global__ void permute_in_kernel(int n, int R, const int32_t *__restrict__ P,
                                  const S *__restrict__ src, D *__restrict__ dst)
{
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * R) return;
  const int o = (int)(idx / R), c = (int)(idx - (int64_t)o * R);
  dst[(size_t)P[o] * R + c] = (D)src[idx];
}

// dst[o, c] = (D) src[P[o], c]   (new order -> original order)
template <typename S, typename D>
__global__ void permute_out_kernel(int n, int R, const int32_t *__restrict__ P,
                                   const S *__restrict__ src, D *__restrict__ dst)
{
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * R) return;
  const int o = (int)(idx / R), c = (int)(idx - (int64_t)o * R);
  dst[idx] = (D)src[(size_t)P[o] * R + c];
}

template <typename S, typename D>
__global__ void convert_kernel(int64_t count, const S *__restrict__ src, D *__restrict__ dst)
{
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < count) dst[idx] = (D)src[idx];
}

// y = a - b elementwise (count entries)
template <typename T>
__global__ void sub_kernel(int64_t count, const T *__restrict__ a, const T *__restrict__ b,
                           T *__restrict__ y)
{
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < count) y[idx] = a[idx] - b[idx];
}

// x64 += (double) d for columns whose status says they took part
template <typename T>
__global__ void accumulate_kernel(int n, int R, const T *__restrict__ d, double *__restrict__ x)
{
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < (int64_t)n * R) x[idx] += (double)d[idx];
}

// dst[i, k] = src[i, idx[k]]   (n rows, R -> Rs columns)
template <typename T>
__global__ void gather_cols_kernel(int n, int R, int Rs, const int32_t *__restrict__ idx,
                                   const T *__restrict__ src, T *__restrict__ dst)
{
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)n * Rs) return;
  const int i = (int)(t / Rs), k = (int)(t - (int64_t)i * Rs);
  dst[t] = src[(size_t)i * R + idx[k]];
}

// dst[i, idx[k]] = src[i, k]
template <typename T>
__global__ void scatter_cols_kernel(int n, int R, int Rs, const int32_t *__restrict__ idx,
                                    const T *__restrict__ src, T *__restrict__ dst)
{
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)n * Rs) return;
  const int i = (int)(t / Rs), k = (int)(t - (int64_t)i * Rs);
  dst[(size_t)i * R + idx[k]] = src[t];
}

// Column compaction of a batched PCG: the per-column state of the columns
// idx[0 .. Rs) moves to columns 0 .. Rs of dst (the iteration temporaries
// alpha, beta and p.t are recomputed; the stop flags start clear)
__global__ void gather_scalars_kernel(int Rs, const int32_t *__restrict__ idx, PcgScalars src, PcgScalars dst)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) {
    *dst.done = 0;
    *dst.want = 0;
    dst.tick[0] = dst.tick[1] = 0;
  }
  if (k >= Rs) return;
  const int c = idx[k];
  dst.rz[k] = src.rz[c];
  dst.b2[k] = src.b2[c];
  dst.thr[k] = src.thr[c];
  dst.rr[k] = src.rr[c];
  dst.rr_ref[k] = src.rr_ref[c];
  dst.stall[k] = src.stall[c];
  dst.status[k] = src.status[c];
  dst.iters[k] = src.iters[c];
}

// ... and back: the outcome of compacted column k to column idx[k] of dst
__global__ void scatter_scalars_kernel(int Rs, const int32_t *__restrict__ idx, PcgScalars src, PcgScalars dst)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= Rs) return;
  const int c = idx[k];
  dst.rz[c] = src.rz[k];
  dst.rr[c] = src.rr[k];
  dst.rr_ref[c] = src.rr_ref[k];
  dst.stall[c] = src.stall[k];
  dst.status[c] = src.status[k];
  dst.iters[c] = src.iters[k];
}

// points (n x 3 float, stride 3) -> float4, optionally gathered by `order`
__global__ void pack_points_kernel(int n, const float *__restrict__ src,
                                   const int32_t *__restrict__ order, float4 *__restrict__ dst)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int o = order ? order[i] : i;
  dst[i] = make_float4(src[3 * (size_t)o], src[3 * (size_t)o + 1], src[3 * (size_t)o + 2], 0.f);
}

}  // namespace mbc
