// Matvec kernels for the MFS operator K (nf collocation rows x n sources).
//
//  * point kernel, evaluated in registers (FP32 here; the FP64 products are
//    matvec64.cuh's):
//      K(i,j) = coef ((x_i - y_j).n_i) / |x_i - y_j|^3   (src/kernels.h:24-40)
//    rows   : W[i, r] = sum_j K(i,j) V[j, r]   (one row per thread, sources
//             staged through shared memory in tiles, R columns per chunk)
//    columns: T[j, r] = sum_i K(i,j) W[i, r]   (one source per thread, rows
//             staged through shared memory)
//
// Coordinates are float4 (x, y, z, 0) so every point is one 16-byte load.
// Vectors are row-major with leading dimension `ld` (the RHS count R); a
// launch handles columns [r0, r0 + RC).  T is the arithmetic type.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mbc {

// The hardware estimate without rsqrtf's scaling of denormal arguments (four
// instructions of sixteen in an evaluation): for those the kernel value
// itself is beyond FP32's range.
__device__ __forceinline__ float rsqrt_ftz(float a)
{
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}

template <typename T>
struct PointKernel;

template <>
struct PointKernel<float> {
  __device__ __forceinline__ static float eval(const float4 &x, const float4 &nx, const float4 &y)
  {
    const float dx = x.x - y.x, dy = x.y - y.y, dz = x.z - y.z;
    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    const float ir = rsqrt_ftz(r2);
    const float rn = fmaf(dz, nx.z, fmaf(dy, nx.y, dx * nx.x));
    return rn * (ir * ir * ir);
  }
};

// FP64 kernel value rn a^(-3/2), a = |x - y|^2, in 16 FP64 instructions: the
// FP32 hardware estimate y0 of a^(-1/2) has e = 1 - a y0^2 with |e| < 1e-6
// (its own error and the rounding of a to FP32), and
// a^(-3/2) = y0^3 (1 - e)^(-3/2) = y0^3 (1 + 3/2 e + 15/8 e^2 + O(e^3)), the
// dropped term below 3e-18.  Two Newton-Raphson steps on a^(-1/2) and its
// cube take 20.  Valid for a in FP32 range; a = 0 gives NaN.
template <>
struct PointKernel<double> {
  __device__ __forceinline__ static double eval(const double3 &x, const double3 &nx, const double3 &y)
  {
    const double dx = x.x - y.x, dy = x.y - y.y, dz = x.z - y.z;
    const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
    const double rn = fma(dz, nx.z, fma(dy, nx.y, dx * nx.x));
    const double y0 = (double)rsqrtf((float)r2);
    const double y2 = y0 * y0;
    const double e = fma(-r2, y2, 1.0);
    const double s = rn * y0 * y2;
    return fma(s, e * fma(e, 1.875, 1.5), s);
  }
  __device__ __forceinline__ static double eval(const float4 &x, const float4 &nx, const float4 &y)
  {
    return eval(make_double3(x.x, x.y, x.z), make_double3(nx.x, nx.y, nx.z), make_double3(y.x, y.y, y.z));
  }
};

// Single-layer potential kernel 1/|x - y| in FP64 (the normal is unused):
// the potential of the solved strengths, utils/torch_utils.py:254-276.  The
// same expansion: a^(-1/2) = y0 (1 + e/2 + 3/8 e^2 + O(e^3)).
struct SingleLayer64 {
  __device__ __forceinline__ static double eval(const double3 &x, const double3 &, const double3 &y)
  {
    const double dx = x.x - y.x, dy = x.y - y.y, dz = x.z - y.z;
    const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
    const double y0 = (double)rsqrtf((float)r2);
    const double e = fma(-r2, y0 * y0, 1.0);
    return fma(y0, e * fma(e, 0.375, 0.5), y0);
  }
};

// Rows direction.  Block = TI threads, one row each; grid.x over rows,
// grid.y over RC-column chunks.  `done` (may be NULL) lets an iteration that
// has nothing left to do exit at once.
template <typename T, int RC, int TI, int TJ>
__global__ void __launch_bounds__(TI) pk_rows_kernel(
    const float4 *__restrict__ xr, const float4 *__restrict__ nr, int nf,
    const float4 *__restrict__ ys, int n, const T *__restrict__ v, int ldv,
    T coef, T *__restrict__ w, int ldw, int R, const int *__restrict__ done)
{
  if (done && *done) return;
  __shared__ float4 sy[TJ];
  __shared__ T sv[TJ * RC];
  const int i = blockIdx.x * TI + threadIdx.x;
  const int r0 = blockIdx.y * RC;
  const int rc = min(RC, R - r0);
  float4 xi = make_float4(0.f, 0.f, 0.f, 0.f), ni = xi;
  if (i < nf) {
    xi = xr[i];
    ni = nr[i];
  }
  T acc[RC];
#pragma unroll
  for (int r = 0; r < RC; ++r) acc[r] = T(0);
  for (int j0 = 0; j0 < n; j0 += TJ) {
    const int jm = min(TJ, n - j0);
    __syncthreads();
    for (int t = threadIdx.x; t < jm; t += TI) sy[t] = ys[j0 + t];
    for (int t = threadIdx.x; t < jm * RC; t += TI) {
      const int jj = t / RC, rr = t - jj * RC;
      sv[t] = rr < rc ? v[(size_t)(j0 + jj) * ldv + r0 + rr] : T(0);
    }
    __syncthreads();
    if (jm == TJ) {
#pragma unroll 2
      for (int jj = 0; jj < TJ; ++jj) {
        const T k = PointKernel<T>::eval(xi, ni, sy[jj]);
#pragma unroll
        for (int r = 0; r < RC; ++r) acc[r] = fma(k, sv[jj * RC + r], acc[r]);
      }
    } else {
      for (int jj = 0; jj < jm; ++jj) {
        const T k = PointKernel<T>::eval(xi, ni, sy[jj]);
#pragma unroll
        for (int r = 0; r < RC; ++r) acc[r] = fma(k, sv[jj * RC + r], acc[r]);
      }
    }
  }
  if (i < nf) {
#pragma unroll
    for (int r = 0; r < RC; ++r)
      if (r < rc) w[(size_t)i * ldw + r0 + r] = coef * acc[r];
  }
}

// Columns direction: T[j, r] = coef * sum_i K(i,j) W[i, r].  Optionally fused
// with the PCG curvature partial sums: part[blockIdx.x * R + r] =
// sum over this block's sources of p[j, r] * T[j, r] (FP64).
template <typename T, int RC, int TI, int TJ>
__global__ void __launch_bounds__(TI) pk_cols_kernel(
    const float4 *__restrict__ xr, const float4 *__restrict__ nr, int nf,
    const float4 *__restrict__ ys, int n, const T *__restrict__ wv, int ldw,
    T coef, T *__restrict__ t_out, int ldt, int R, const T *__restrict__ pdot,
    double *__restrict__ part, const int *__restrict__ done)
{
  if (done && *done) return;
  __shared__ float4 sx[TJ], sn[TJ];
  __shared__ T sw[TJ * RC];
  __shared__ double sred[RC][TI / 32];
  const int j = blockIdx.x * TI + threadIdx.x;
  const int r0 = blockIdx.y * RC;
  const int rc = min(RC, R - r0);
  float4 yj = make_float4(0.f, 0.f, 0.f, 0.f);
  if (j < n) yj = ys[j];
  T acc[RC];
#pragma unroll
  for (int r = 0; r < RC; ++r) acc[r] = T(0);
  for (int i0 = 0; i0 < nf; i0 += TJ) {
    const int im = min(TJ, nf - i0);
    __syncthreads();
    for (int t = threadIdx.x; t < im; t += TI) {
      sx[t] = xr[i0 + t];
      sn[t] = nr[i0 + t];
    }
    for (int t = threadIdx.x; t < im * RC; t += TI) {
      const int ii = t / RC, rr = t - ii * RC;
      sw[t] = rr < rc ? wv[(size_t)(i0 + ii) * ldw + r0 + rr] : T(0);
    }
    __syncthreads();
    if (im == TJ) {
#pragma unroll 2
      for (int ii = 0; ii < TJ; ++ii) {
        const T k = PointKernel<T>::eval(sx[ii], sn[ii], yj);
#pragma unroll
        for (int r = 0; r < RC; ++r) acc[r] = fma(k, sw[ii * RC + r], acc[r]);
      }
    } else {
      for (int ii = 0; ii < im; ++ii) {
        const T k = PointKernel<T>::eval(sx[ii], sn[ii], yj);
#pragma unroll
        for (int r = 0; r < RC; ++r) acc[r] = fma(k, sw[ii * RC + r], acc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RC; ++r) acc[r] *= coef;
  if (j < n) {
#pragma unroll
    for (int r = 0; r < RC; ++r)
      if (r < rc) t_out[(size_t)j * ldt + r0 + r] = acc[r];
  }
  if (part) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int r = 0; r < RC; ++r) {
      double d = 0.0;
      if (j < n && r < rc) d = (double)pdot[(size_t)j * ldt + r0 + r] * (double)acc[r];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      if (lane == 0) sred[r][wid] = d;
    }
    __syncthreads();
    if (threadIdx.x < RC && threadIdx.x < rc) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < TI / 32; ++k) s += sred[threadIdx.x][k];
      part[(size_t)blockIdx.x * R + r0 + threadIdx.x] = s;
    }
  }
}

}  // namespace mbc

