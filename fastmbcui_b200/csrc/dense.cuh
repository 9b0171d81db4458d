// Products with a caller-provided dense matrix M (nf x n, row-major FP32), the
// mfs_torch operator's input, in FP32 or FP64.
//
//   DIR 0: W[i, r] = sum_o M[i, o] V[P[o], r]     DIR 1: T[P[o], r] = sum_i M[i, o] W[i, r]
//
// (the vector blocks on the source side are in the plan's order, P[o] the
// position of column o).  What bounds it: one pass over M from HBM (73 us for
// the 15360 x 7686 matrix of three mesh bodies) and, from about 20 FP32 columns
// or 8 FP64 ones on, the multiply-adds.  So:
//   * M is read once for up to 32 columns, 64 outputs x 64 reduction positions
//     per tile, by cp.async three tiles deep (16-, 8- or 4-byte copies by what
//     the row stride and the base address allow), rows of M contiguous in
//     both directions.
//   * The 8 warps of a block share every tile by reduction position, 8 each,
//     and every warp holds the block's whole 64 x np outputs in registers:
//     FP32 8 x np/4 per lane (four positions at a time from 128-bit shared
//     loads), FP64 as mma.sync m16n8k8.f64 fragments, M converted on load.
//     One sum over the warps at the end replaces a barrier-bound small tile.
//   * A matrix with few rows of blocks is cut over a cluster of up to 8 blocks
//     along the reduction axis; the cluster adds its tiles through distributed
//     shared memory, in order, so that no second kernel is needed.
// Measured (B200, 15360 x 7686, 18 columns): FP32 K 2.76 -> 0.23 ms and K^T 2.09
// -> 0.24 ms, FP64 3.79 -> 0.38 and 6.02 -> 0.41 ms, against a warp per row and a
// thread per column with the columns re-read in chunks of 4 to 32.
// All sums have a fixed order.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "matvec64.cuh"

namespace mbc {
namespace dns {

constexpr int kBM = 64;     // outputs per block
constexpr int kBK = 64;     // reduction positions per tile
constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kStages = 3;
constexpr int kMaxCluster = 8;

struct Args {
  const float *M;
  int64_t ldm;
  int nf, n;
  const int32_t *P;
  const void *in;      // K x R
  void *out;
  int R;
  int vec;             // bytes per copy of M: 16, 8 or 4
  int vecv;            // bytes per copy of the vector block: 16, 8 or 4
  const void *pdot;    // DIR 1: p (n x R, plan order) for the curvature partials, or NULL
  double *part;        // part[(blockIdx.x * gridDim.z + cluster rank) * R + r]
  const int32_t *done;
};

// columns per block of NT units: FP32 NT columns per lane x 4, FP64 NT mma tiles of 8
template <typename T>
__host__ __device__ constexpr int cols(int nt)
{
  return sizeof(T) == 4 ? 4 * nt : 8 * nt;
}
template <typename T>
__host__ __device__ constexpr int ldv(int nt)  // row stride of the staged vector tile
{
  return sizeof(T) == 4 ? cols<T>(nt) : p64::lds_for(nt);
}
// row stride of the staged M tile: [output][position] (DIR 0) or [position][output]
template <int DIR>
__host__ __device__ constexpr int ldt()
{
  return DIR == 0 ? kBK + 4 : kBM + 8;
}
template <typename T, int DIR>
__host__ __device__ constexpr int smem_bytes(int nt)
{
  const int stages = kStages * (64 * ldt<DIR>() * (int)sizeof(float) + kBK * ldv<T>(nt) * (int)sizeof(T));
  const int sums = 5 * kBM * cols<T>(nt) * (int)sizeof(T);  // four warps' blocks and the block's sum
  return stages > sums ? stages : sums;
}

template <int B>
__device__ __forceinline__ void cp_async(void *smem, const void *gmem, int bytes)
{
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  if (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(B), "r"(bytes) : "memory");
}

template <int V>
struct Int {
  static constexpr int value = V;
};

// N consecutive floats from shared memory, aligned as N allows
template <int N>
__device__ __forceinline__ void load_row(const float *p, float (&v)[N])
{
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
      const float4 x = reinterpret_cast<const float4 *>(p)[q];
      v[4 * q] = x.x;
      v[4 * q + 1] = x.y;
      v[4 * q + 2] = x.z;
      v[4 * q + 3] = x.w;
    }
  } else if constexpr (N % 2 == 0) {
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
      const float2 x = reinterpret_cast<const float2 *>(p)[q];
      v[2 * q] = x.x;
      v[2 * q + 1] = x.y;
    }
  } else {
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = p[q];
  }
}

template <typename T, int DIR, int NT>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 4 || NT <= 2 ? 2 : 1) dense_kernel(Args a)
{
  if (a.done && *a.done) return;
  namespace cg = cooperative_groups;
  constexpr int NP = cols<T>(NT), LDV = ldv<T>(NT), LDT = ldt<DIR>();
  constexpr int MT_FLOATS = 64 * LDT;
  extern __shared__ __align__(16) unsigned char smd[];
  float *sm_m = reinterpret_cast<float *>(smd);                                       // [kStages][64][LDT]
  T *sm_v = reinterpret_cast<T *>(smd + kStages * MT_FLOATS * sizeof(float));         // [kStages][kBK][LDV]
  const int M = DIR == 0 ? a.nf : a.n, K = DIR == 0 ? a.n : a.nf;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int o0 = blockIdx.x * kBM, c0 = blockIdx.y * NP;
  const int tiles = (K + kBK - 1) / kBK;
  const int tb = (int)((int64_t)tiles * blockIdx.z / gridDim.z), te = (int)((int64_t)tiles * (blockIdx.z + 1) / gridDim.z);
  const T *in = reinterpret_cast<const T *>(a.in);

  // Copies of M: CP per row, this thread's rows rm, rm + 256 / CP, ...; tile
  // tl starts at mp + tl * adv.  Tiles inside the matrix take no checks.
  const int per = a.vec >> 2, cp_log = a.vec == 16 ? 4 : a.vec == 8 ? 5 : 6;
  const int rm = tid >> cp_log, cm = (tid & ((1 << cp_log) - 1)) * per, rstep = kThreads >> cp_log;
  const float *mp = a.M + (DIR == 0 ? (size_t)(o0 + rm) * a.ldm + cm : (size_t)rm * a.ldm + o0 + cm);
  const int64_t adv = DIR == 0 ? kBK : (int64_t)kBK * a.ldm;
  const bool out_full = o0 + kBM <= M;
  auto copy_m = [&](float *dst, int tl, auto bytes_of) {
    constexpr int B = decltype(bytes_of)::value;
    const int k0 = tl * kBK;
    const float *src = mp + tl * adv;
    if (out_full && k0 + kBK <= K) {
#pragma unroll
      for (int i = 0; i < 64 / B; ++i)
        cp_async<B>(dst + (rm + i * rstep) * LDT + cm, src + (size_t)(i * rstep) * a.ldm, B);
    } else {
      const int r0 = DIR == 0 ? o0 : k0, q0 = DIR == 0 ? k0 : o0;
#pragma unroll
      for (int i = 0; i < 64 / B; ++i) {
        const int r = r0 + rm + i * rstep, left = 4 * (a.n - q0 - cm);
        const int bytes = r < a.nf && left > 0 ? min(B, left) : 0;
        cp_async<B>(dst + (rm + i * rstep) * LDT + cm, bytes ? src + (size_t)(i * rstep) * a.ldm : a.M, bytes);
      }
    }
  };
  // Copies of the vector block: units of vecv bytes, ur per row; this thread's
  // unit u of a tile is row kk[u], column cv[u].  Columns past the last unit
  // are zeroed once.  The permuted rows of DIR 0 are looked up a tile ahead.
  constexpr int kUnits = NP * (int)sizeof(T) / 4 / 4;  // per thread at most (4-byte copies)
  constexpr int U = sizeof(T) == 8 ? kUnits / 2 : kUnits;
  const int ev = a.vecv / (int)sizeof(T);  // elements per copy
  const int ur = (min(NP, a.R - c0) + ev - 1) / ev;
  int kk[U], cv[U], pk[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int e = tid + u * kThreads;
    kk[u] = e < kBK * ur ? e / ur : -1;
    cv[u] = (e - kk[u] * ur) * ev;
    pk[u] = 0;
  }
  for (int e = tid; e < kStages * kBK * LDV; e += kThreads)
    if (e % LDV >= ur * ev) sm_v[e] = T(0);
  auto lookup = [&](int tl) {
    if (DIR == 0 && tl < te) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (kk[u] >= 0) pk[u] = __ldg(a.P + min(tl * kBK + kk[u], K - 1));
    }
  };
  auto stage = [&](int tl) {
    if (tl < te) {
      const int b = (tl - tb) % kStages, k0 = tl * kBK;
      float *dm = sm_m + b * MT_FLOATS;
      if (a.vec == 16) copy_m(dm, tl, Int<16>{});
      else if (a.vec == 8) copy_m(dm, tl, Int<8>{});
      else copy_m(dm, tl, Int<4>{});
      T *dv = sm_v + b * kBK * LDV;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (kk[u] >= 0) {
          const bool ok = k0 + kk[u] < K;
          const T *src = in + (size_t)(DIR == 0 ? pk[u] : min(k0 + kk[u], K - 1)) * a.R + c0 + cv[u];
          T *dst = dv + kk[u] * LDV + cv[u];
          if (a.vecv == 16) cp_async<16>(dst, src, ok ? 16 : 0);
          else if (a.vecv == 8) cp_async<8>(dst, src, ok ? 8 : 0);
          else if constexpr (sizeof(T) == 4) cp_async<4>(dst, src, ok ? 4 : 0);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // FP32: acc[j][q], output j of the lane's 8, column q of its NT.
  // FP64: acc[(m * NT + q)][4], mma fragments of the four 16-output tiles.
  constexpr int NA = sizeof(T) == 4 ? 8 * NT : 16 * NT;
  T acc[NA];
#pragma unroll
  for (int q = 0; q < NA; ++q) acc[q] = T(0);
  const int g = lane >> 2, t = lane & 3;

  lookup(tb);
  stage(tb);
  lookup(tb + 1);
  stage(tb + 1);
  lookup(tb + 2);
  for (int tl = tb; tl < te; ++tl) {
    stage(tl + 2);
    lookup(tl + 3);
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncthreads();
    const int b = (tl - tb) % kStages;
    const float *tm = sm_m + b * MT_FLOATS;
    const T *tv = sm_v + b * kBK * LDV;
    const int kw = warp * 8;  // this warp's positions of the tile
    if constexpr (sizeof(T) == 4) {
      if constexpr (DIR == 0) {
#pragma unroll
        for (int k4 = 0; k4 < 8; k4 += 4) {
          float4 m[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) m[j] = *reinterpret_cast<const float4 *>(tm + (j * 8 + g) * LDT + kw + k4);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float v[NT];
            load_row<NT>(tv + (kw + k4 + u) * LDV + t * NT, v);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float mj = u == 0 ? m[j].x : u == 1 ? m[j].y : u == 2 ? m[j].z : m[j].w;
#pragma unroll
              for (int q = 0; q < NT; ++q) acc[j * NT + q] = fmaf(mj, v[q], acc[j * NT + q]);
            }
          }
        }
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float *row = tm + (kw + u) * LDT + g * 4;
          const float4 m0 = *reinterpret_cast<const float4 *>(row), m1 = *reinterpret_cast<const float4 *>(row + 32);
          const float m[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
          float v[NT];
          load_row<NT>(tv + (kw + u) * LDV + t * NT, v);
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int q = 0; q < NT; ++q) acc[j * NT + q] = fmaf(m[j], v[q], acc[j * NT + q]);
        }
      }
    } else {
      const T *bv = tv + (kw + t) * LDV + g;
      T b0[NT], b1[NT];
#pragma unroll
      for (int q = 0; q < NT; ++q) {
        b0[q] = bv[q * 8];
        b1[q] = bv[4 * LDV + q * 8];
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        // A fragment: outputs g, g + 8 of tile m, positions t, t + 4
        const float *p = DIR == 0 ? tm + (m * 16 + g) * LDT + kw + t : tm + (kw + t) * LDT + m * 16 + g;
        constexpr int dr = DIR == 0 ? 8 * LDT : 8, dk = DIR == 0 ? 4 : 4 * LDT;
        const double af[4] = {(double)p[0], (double)p[dr], (double)p[dk], (double)p[dr + dk]};
#pragma unroll
        for (int q = 0; q < NT; ++q) {
          double (&c)[4] = *reinterpret_cast<double (*)[4]>(&acc[(m * NT + q) * 4]);
          p64::mma_f64(c, af, b0[q], b1[q]);
        }
      }
    }
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // the block's sum: warps 4..7 hand theirs to warps 0..3, whose four blocks
  // are then added in order (there and over the cluster in 64 bits, with one
  // rounding each, as every rounding of a whole sum weighs as much as a
  // warp's chain).  slot[w][output][column]
  T *slot = reinterpret_cast<T *>(smd);
  constexpr int SL = kBM * NP;
  auto visit = [&](auto f) {  // f(element of the 64 x NP block, accumulator index)
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int o = DIR == 0 ? j * 8 + g : (j < 4 ? g * 4 + j : 32 + g * 4 + j - 4);
#pragma unroll
        for (int q = 0; q < NT; ++q) f(o * NP + t * NT + q, j * NT + q);
      }
    } else {
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int q = 0; q < NT; ++q)
#pragma unroll
          for (int h = 0; h < 4; ++h)
            f((m * 16 + g + 8 * (h >> 1)) * NP + q * 8 + 2 * t + (h & 1), (m * NT + q) * 4 + h);
    }
  };
  T *mine = slot + (warp & 3) * SL;
  if (warp >= 4) visit([&](int e, int q) { mine[e] = acc[q]; });
  __syncthreads();
  if (warp < 4) visit([&](int e, int q) { mine[e] += acc[q]; });
  __syncthreads();
  T *fin = slot + 4 * SL;
  for (int e = tid; e < SL; e += kThreads)
    fin[e] = (T)(((double)slot[e] + (double)slot[SL + e]) + ((double)slot[2 * SL + e] + (double)slot[3 * SL + e]));

  // the cluster's blocks hold the shares of the reduction axis: each adds and
  // stores a slice of the outputs
  const int z = gridDim.z;
  int rank = 0, ra = 0, rb = kBM;
  if (z > 1) {
    cg::cluster_group cl = cg::this_cluster();
    rank = (int)cl.block_rank();
    ra = kBM * rank / z;
    rb = kBM * (rank + 1) / z;
    cl.sync();
  } else {
    __syncthreads();
  }
  __shared__ double red[kThreads];
  constexpr int RG = kThreads / NP;  // row groups of the store
  const int c = tid % NP, rg = tid / NP;
  double d = 0.0;
  if (rg < RG && c0 + c < a.R) {
    for (int o = ra + rg; o < rb && o0 + o < M; o += RG) {
      T s;
      if (z > 1) {
        cg::cluster_group cl = cg::this_cluster();
        double sum = *cl.map_shared_rank(fin + o * NP + c, 0);
        for (int k = 1; k < z; ++k) sum += (double)*cl.map_shared_rank(fin + o * NP + c, k);
        s = (T)sum;
      } else {
        s = fin[o * NP + c];
      }
      const size_t at = (size_t)(DIR == 0 ? o0 + o : __ldg(a.P + o0 + o)) * a.R + c0 + c;
      reinterpret_cast<T *>(a.out)[at] = s;
      if (a.part) d += (double)reinterpret_cast<const T *>(a.pdot)[at] * (double)s;
    }
  }
  if (a.part) {
    red[tid] = d;
    __syncthreads();
    if (rg == 0 && c0 + c < a.R) {
      for (int k = 1; k < RG; ++k) d += red[k * NP + c];
      a.part[((size_t)blockIdx.x * z + rank) * a.R + c0 + c] = d;
    }
  }
  if (z > 1) cg::this_cluster().sync();  // no block leaves while others read its sums
}

}  // namespace dns
}  // namespace mbc
