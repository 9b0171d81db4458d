// Theta_s = K(:, I_s)^T K(:, I_s) of the supernodes with at most 64 entries,
// FP32 or FP64, before factor_kernel factors them (gram_ready).
//
// A block takes one supernode and one part of the collocation rows; a panel
// of rows x entries is evaluated into shared memory and multiplied from there.
// What bounds it: the evaluations (one per row and entry, 5 n nf of them over a
// scene's overlapping sets) and the n_s (n_s + 1) / 2 multiply-adds per row.
// A thread per entry of Theta_s needs two shared-memory loads per
// multiply-add and is bound by those, 8 times slower than the arithmetic.
//   FP32: threads own 8 x 8 tiles of the upper triangle and every G-th row of
//     the panel (G = threads / tiles): four 128-bit loads per 64 multiply-adds.
//   FP64: mma.sync m16n8k8.f64, a warp owns every eighth group of 8 rows and all
//     tiles of the upper triangle; the A fragments are the B fragments of the
//     same columns, so a panel value is loaded once.  Coordinates are staged as
//     doubles: nine conversions per evaluation would cost more than its 16
//     FP64 instructions.
// Few supernodes (a small scene, the FP64 retries of an FP32 factor) are cut
// into parts of the rows, whose blocks factor_kernel adds in order.  All sums
// have a fixed order.
// Measured (B200): the FP32 factor of 24000 points (rho 3) with its FP64 retries
// 49 -> 16 ms, the FP64 factor of 3000 points 3.1 -> 2.0 ms, against one thread per
// entry inside factor_kernel.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "factor.cuh"
#include "matvec64.cuh"

namespace mbc {
namespace gram {

constexpr int kMaxNs = 64;
constexpr int kThreads = 256;
constexpr int kMaxParts = 16;

// panel rows and padded width of a set of ns entries
template <typename T>
__host__ __device__ constexpr int rows_for(int ns)
{
  return sizeof(T) == 4 && ns <= 32 ? 128 : 64;
}
template <typename T>
__host__ __device__ constexpr int width_for(int ns)
{
  return sizeof(T) == 4 ? (ns + 7) / 8 * 8 : (ns + 15) / 16 * 16;
}
template <typename T>
__host__ __device__ constexpr int ld_for(int ns)
{
  return width_for<T>(ns) + 4;
}
// panel, row points (x, n, z) and entry points; FP64 point kernels keep them as doubles
template <typename T>
__host__ __device__ constexpr int smem_bytes(int ns_max)
{
  constexpr int pt = sizeof(T) == 4 ? 16 : 24;
  return rows_for<T>(ns_max) * ld_for<T>(ns_max) * (int)sizeof(T) + (3 * 128 + kMaxNs) * pt;
}

struct Args {
  FactorArgs f;
  int parts;           // parts of the rows: grid.y
  int64_t part_stride; // entries between the parts' copies of theta
  const int64_t *off;  // a supernode's entries in a copy
  int rows, ld;        // panel rows and stride of the launch
};

// acc of 8 x 8 tile (p0, q0) += outer products of panel row k
__device__ __forceinline__ void rank1(const float *row, int p0, int q0, float (&acc)[8][8])
{
  float p[8], q[8];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float4 a = *reinterpret_cast<const float4 *>(row + p0 + 4 * h);
    const float4 b = *reinterpret_cast<const float4 *>(row + q0 + 4 * h);
    p[4 * h] = a.x, p[4 * h + 1] = a.y, p[4 * h + 2] = a.z, p[4 * h + 3] = a.w;
    q[4 * h] = b.x, q[4 * h + 1] = b.y, q[4 * h + 2] = b.z, q[4 * h + 3] = b.w;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(p[i], q[j], acc[i][j]);
}

// MT: 16-entry tiles of an FP64 set (1 .. 4); unused in FP32
template <typename T, int MT>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 4 || MT <= 2 ? 2 : 1) gram_kernel(Args a, T *__restrict__ theta)
{
  extern __shared__ __align__(16) unsigned char smg[];
  const FactorArgs &f = a.f;
  const int s = f.list[blockIdx.x];
  const int sb = f.set_ptr[s];
  const int ns = f.set_ptr[s + 1] - sb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int TR = a.rows, LD = a.ld;
  const int W = width_for<T>(ns);  // <= LD - 4
  constexpr bool dbl = sizeof(T) == 8;
  T *panel = reinterpret_cast<T *>(smg);
  unsigned char *pts = smg + (size_t)TR * LD * sizeof(T);
  // points: float4 arrays, or (FP64 point kernel) doubles [3][..]
  float4 *rx = reinterpret_cast<float4 *>(pts), *rn = rx + 128, *rz = rn + 128, *src = rz + 128;
  double *drx = reinterpret_cast<double *>(pts), *dsrc = drx + 6 * 128;
  int32_t *scol = reinterpret_cast<int32_t *>(src);
  const bool dpk = dbl && f.kind == 1;

  for (int p = tid; p < ns; p += kThreads) {
    const int c = f.set_ind[sb + p];
    if (f.kind == 0) scol[p] = f.Pinv[c];
    else if (dpk) {
      const float4 y = f.ys[c];
      dsrc[p] = y.x;
      dsrc[kMaxNs + p] = y.y;
      dsrc[2 * kMaxNs + p] = y.z;
    } else {
      src[p] = f.ys[c];
    }
  }
  for (int e = tid; e < TR * LD; e += kThreads) panel[e] = T(0);  // the padding stays zero

  // FP32 tiles
  const int nb = W >> 3, ntile = nb * (nb + 1) / 2;
  const int G = min(kThreads / ntile, 64);
  const int g = tid / ntile;
  int p0 = 0, q0 = 0;
  float acc[8][8];
  // FP64 fragments of the tiles (mi, nj) with 8 nj + 7 >= 16 mi
  constexpr int NF = MT * (MT + 1);
  double accd[NF][4];
  if constexpr (!dbl) {
    tri_decode(tid % ntile, p0, q0);
    p0 *= 8;
    q0 *= 8;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  } else {
#pragma unroll
    for (int i = 0; i < NF; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) accd[i][j] = 0.0;
  }
  const T coef = (T)f.coef;
  const uint32_t inv = ((1u << 20) + ns - 1) / ns;  // t / ns = t inv >> 20 for t < TR ns <= 8192
  const int r0 = (int)((int64_t)f.nf * blockIdx.y / a.parts), r1 = (int)((int64_t)f.nf * (blockIdx.y + 1) / a.parts);

  // the next tile's row points, fetched before the products of this one
  float4 fx, fn, fz;
  auto fetch = [&](int i0) {
    if (tid < TR && f.kind != 0) {
      const int i = min(i0 + tid, f.nf - 1);
      fx = f.xr[i];
      fn = f.nr[i];
      if (f.kind == 2) fz = f.zr[i];
    }
  };
  fetch(r0);
  for (int i0 = r0; i0 < r1; i0 += TR) {
    const int im = min(TR, r1 - i0);
    __syncthreads();  // the last tile's panel and points are read
    if (tid < TR && f.kind != 0) {
      if (dpk) {
        drx[tid] = fx.x;
        drx[128 + tid] = fx.y;
        drx[256 + tid] = fx.z;
        drx[384 + tid] = fn.x;
        drx[512 + tid] = fn.y;
        drx[640 + tid] = fn.z;
      } else {
        rx[tid] = fx;
        rn[tid] = fn;
        if (f.kind == 2) rz[tid] = fz;
      }
    }
    __syncthreads();
    for (int t = tid; t < TR * ns; t += kThreads) {
      const int rr = (int)((uint32_t)t * inv >> 20), p = t - rr * ns;
      T v = T(0);
      if (rr < im) {
        if (f.kind == 1) {
          if constexpr (dbl)
            v = coef * PointKernel<double>::eval(make_double3(drx[rr], drx[128 + rr], drx[256 + rr]),
                                                 make_double3(drx[384 + rr], drx[512 + rr], drx[640 + rr]),
                                                 make_double3(dsrc[p], dsrc[kMaxNs + p], dsrc[2 * kMaxNs + p]));
          else
            v = coef * PointKernel<float>::eval(rx[rr], rn[rr], src[p]);
        } else if (f.kind == 2) {
          v = coef * SolidAngle<T>::eval(rx[rr], rn[rr], rz[rr], src[p]);
        } else {
          v = (T)__ldg(f.M + (size_t)(i0 + rr) * f.ldm + scol[p]);
        }
      }
      panel[rr * LD + p] = v;
    }
    fetch(i0 + TR);
    __syncthreads();
    if constexpr (!dbl) {
      if (g < G)
        for (int k = g; k < im; k += G) rank1(panel + k * LD, p0, q0, acc);
    } else {
      for (int k8 = warp * 8; k8 < im; k8 += 64) {
        const double *row = panel + (k8 + (lane & 3)) * LD + (lane >> 2);
        double b0[2 * MT], b1[2 * MT];
#pragma unroll
        for (int j = 0; j < 2 * MT; ++j) {
          b0[j] = row[8 * j];
          b1[j] = row[4 * LD + 8 * j];
        }
        int q = 0;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          const double af[4] = {b0[2 * i], b0[2 * i + 1], b1[2 * i], b1[2 * i + 1]};
#pragma unroll
          for (int j = 2 * i; j < 2 * MT; ++j) p64::mma_f64(accd[q++], af, b0[j], b1[j]);
        }
      }
    }
  }

  // sum over the G row groups (FP32) or 8 warps (FP64) in order, as many W x W
  // blocks at a time as the panel holds; entries tid, tid + 256, ... per thread
  T *slot = panel;
  const int per = max(1, TR * LD / (W * W));
  const int holders = dbl ? kThreads / 32 : G;
  const int me = dbl ? warp : g;
  T fin[kMaxNs * kMaxNs / kThreads];
#pragma unroll
  for (int i = 0; i < kMaxNs * kMaxNs / kThreads; ++i) fin[i] = T(0);
  for (int h0 = 0; h0 < holders; h0 += per) {
    const int cnt = min(per, holders - h0);
    __syncthreads();
    if (me >= h0 && me < h0 + cnt) {
      T *d = slot + (size_t)(me - h0) * W * W;
      if constexpr (!dbl) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) d[(p0 + i) * W + q0 + j] = acc[i][j];
      } else {
        int q = 0;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 2 * i; j < 2 * MT; ++j, ++q)
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int p = 16 * i + (lane >> 2) + 8 * (h >> 1), c = 8 * j + 2 * (lane & 3) + (h & 1);
              if (p < W && c < W) d[p * W + c] = accd[q][h];
            }
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kMaxNs * kMaxNs / kThreads; ++i) {
      const int e = tid + i * kThreads;
      if (e < W * W && e / W <= e % W)
        for (int h = 0; h < cnt; ++h) fin[i] += slot[(size_t)h * W * W + e];
    }
  }
  T *A = theta + a.part_stride * blockIdx.y + a.off[s];
#pragma unroll
  for (int i = 0; i < kMaxNs * kMaxNs / kThreads; ++i) {
    const int e = tid + i * kThreads, p = e / W, q = e % W;
    if (e < W * W && p <= q && q < ns) {
      const int rp = ns - 1 - p, rq = ns - 1 - q;
      A[rp + (size_t)rq * ns] = fin[i];
      A[rq + (size_t)rp * ns] = fin[i];
    }
  }
}

}  // namespace gram
}  // namespace mbc
