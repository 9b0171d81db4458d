// FP64 point-kernel products on the FP64 matrix instructions (mma.sync
// m16n8k8 f64): one kernel for both directions and for every column count.
//
//   DIR 0: W[i, r] = coef sum_j G(x_i, n_i, y_j) V[j, r]   (outputs: rows,    reduction: sources)
//   DIR 1: T[j, r] = coef sum_i G(x_i, n_i, y_j) W[i, r]   (outputs: sources, reduction: rows)
//
// What bounds it: the FP64 pipe (DFMA and DMMA share it: both measured
// 36 to 37 TFLOP/s on the B200).  A kernel value costs 16 FP64 instructions
// and each column one multiply-add, so a value must serve as many columns as
// possible, and the operands of the multiply-adds must not cost issue slots.
//   * A warp owns 16 outputs x up to 64 columns.  Each lane evaluates exactly
//     the four entries of its m16n8k8 A fragment in registers (rows g and
//     g + 8, reduction positions t and t + 4, g = lane / 4, t = lane % 4), so
//     nothing is evaluated twice inside 64 columns and no kernel value passes
//     through shared memory; the 16 x 8 values then meet all the warp's
//     column tiles.  More than 64 columns: column groups (grid.y), each
//     evaluating again.  96 columns a warp would evaluate less (7 % of the
//     work at 192) but leave one block per SM, and evaluations and matrix
//     instructions of too few warps to overlap: 47 % of the FP64 pipe, against
//     73 % with two blocks (24000 points, 192 columns: 14.9 ms, against 10.8).
//   * The vector block's tile (kKT positions x columns, FP64) is staged by
//     cp.async two deep; its row stride is 4 modulo 16 doubles, which makes
//     the B fragment loads free of bank conflicts.
//   * A block is 8 warps: kMT = 4 tiles of 16 outputs x KS = 2 shares of every
//     staged tile (16 or 32 outputs a block, with more shares, read the tiles
//     from L2 more often and sum more: 10 to 40 % slower at every size but the
//     smallest).  The shares of a tile are summed through shared memory at the
//     end.  Where blocks are too few, or fill a last wave badly, the
//     reduction axis is further cut over a cluster of up to 8 blocks, which add
//     their results through distributed shared memory.  All sums have a fixed
//     order.
// Positions past the end carry the last point and zero vector entries: their
// kernel values are finite wherever that point's own are.
// Measured (B200, K then K^T): 20000 x 20000, 60 columns 4.90 ms, against
// 10.92 ms for one thread per output with FP64 FMAs and one evaluation per 32
// columns; the FP64 pipe's floor is 3.5 ms.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "matvec.cuh"

namespace mbc {
namespace p64 {

constexpr int kKT = 64;        // reduction positions per staged tile
constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kMT = 4;         // tiles of 16 outputs per block
constexpr int kRows = 16 * kMT;
constexpr int kNtMax = 8;      // column tiles of 8 per warp: two blocks per SM

struct Args {
  const float4 *xr, *nr;  // collocation rows, normals (float4)
  const float4 *ys;       // sources
  int nf, n;
  const double *in;       // K x R vector block (row stride R)
  double *out;            // M x R
  int R;
  double coef;
  const double *pdot;     // curvature partials: p, M x R, or NULL
  double *part;           // per slice of outputs: part[(blockIdx.x * cluster size + rank) * R + r]
  const int32_t *done;
};

__host__ __device__ constexpr int lds_for(int nt) { return nt * 8 + (nt % 2 == 0 ? 4 : 12); }
static_assert(lds_for(6) % 16 == 4 && lds_for(3) % 16 == 4 && lds_for(1) % 16 == 4 && lds_for(8) % 16 == 4,
              "stride of the staged tile");
template <int DIR>
__host__ __device__ constexpr int coords()
{
  return DIR == 0 ? 3 : 6;
}
template <int DIR>
__host__ __device__ constexpr int smem_bytes(int nt)
{
  return 2 * kKT * (lds_for(nt) + coords<DIR>()) * (int)sizeof(double);
}

__device__ __forceinline__ void mma_f64(double (&c)[4], const double (&a)[4], double b0, double b1)
{
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, bool valid)
{
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(s), "l"(gmem), "r"(valid ? 8 : 0) : "memory");
}

// grid (output blocks of kRows, column groups, cluster size)
template <int DIR, int NT, class Ker>
__global__ void __launch_bounds__(kThreads, 2) pk64_kernel(Args a)
{
  if (a.done && *a.done) return;
  constexpr int MT = kMT;
  constexpr int KS = kWarps / MT;   // shares of a staged tile
  constexpr int KW = kKT / KS;      // positions of a share
  constexpr int LDS = lds_for(NT);
  constexpr int NC = coords<DIR>();
  constexpr int NP = NT * 8;
  extern __shared__ __align__(16) double sm64[];
  double *sv = sm64;                    // [2][kKT][LDS]
  double *sc = sm64 + 2 * kKT * LDS;    // [2][NC][kKT]
  const int M = DIR == 0 ? a.nf : a.n;
  const int K = DIR == 0 ? a.n : a.nf;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int mt = warp % MT, ks = warp / MT;
  const int c0 = blockIdx.y * NP;
  const int row0 = (blockIdx.x * MT + mt) * 16 + g;
  // this block's tiles
  const int tiles = (K + kKT - 1) / kKT;
  const int tb = (int)((int64_t)tiles * blockIdx.z / gridDim.z), te = (int)((int64_t)tiles * (blockIdx.z + 1) / gridDim.z);

  double3 ox[2], on[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = row0 + 8 * h;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
    if (i < M) {
      if (DIR == 0) {
        p = a.xr[i];
        q = a.nr[i];
      } else {
        p = a.ys[i];
      }
    }
    ox[h] = make_double3(p.x, p.y, p.z);
    on[h] = make_double3(q.x, q.y, q.z);
  }

  // stage tile `tl` of the vector block into buffer b (asynchronously)
  auto stage = [&](int tl, int b) {
    const int k0 = tl * kKT;
    double *dst = sv + b * kKT * LDS;
    for (int e = tid; e < kKT * NP; e += kThreads) {
      const int kk = e / NP, c = e - kk * NP;
      const bool ok = k0 + kk < K && c0 + c < a.R;
      cp_async8(dst + kk * LDS + c, ok ? a.in + (size_t)(k0 + kk) * a.R + c0 + c : a.in, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the tile's coordinates: fetched early into registers, converted and
  // stored once the other buffer's readers are done
  float4 fp, fq = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fetch = [&](int tl) {
    if (tid < kKT) {
      const int k = min(tl * kKT + tid, K - 1);
      if (DIR == 0) {
        fp = a.ys[k];
      } else {
        fp = a.xr[k];
        fq = a.nr[k];
      }
    }
  };
  auto put = [&](int b) {
    if (tid < kKT) {
      double *d = sc + b * NC * kKT + tid;
      d[0] = fp.x;
      d[kKT] = fp.y;
      d[2 * kKT] = fp.z;
      if (DIR == 1) {
        d[3 * kKT] = fq.x;
        d[4 * kKT] = fq.y;
        d[5 * kKT] = fq.z;
      }
    }
  };

  double acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[j][q] = 0.0;

  if (tb < te) {
    stage(tb, 0);
    fetch(tb);
    put(0);
  }
  for (int tl = tb; tl < te; ++tl) {
    const int b = (tl - tb) & 1;
    const bool more = tl + 1 < te;
    if (more) {
      stage(tl + 1, b ^ 1);
      fetch(tl + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const double *tv = sv + b * kKT * LDS;
    const double *tc = sc + b * NC * kKT;
#pragma unroll(KW / 8 < 4 ? KW / 8 : 4)
    for (int k8 = 0; k8 < KW; k8 += 8) {
      const int kk = ks * KW + k8 + t;
      double af[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // reduction positions t and t + 4
        const double *c = tc + kk + 4 * h;
        const double3 p = make_double3(c[0], c[kKT], c[2 * kKT]);
        double3 q = make_double3(0.0, 0.0, 0.0);
        if (DIR == 1) q = make_double3(c[3 * kKT], c[4 * kKT], c[5 * kKT]);
#pragma unroll
        for (int u = 0; u < 2; ++u)
          af[2 * h + u] = DIR == 0 ? Ker::eval(ox[u], on[u], p) : Ker::eval(p, q, ox[u]);
      }
      const double *bv = tv + kk * LDS + g;
#pragma unroll
      for (int j = 0; j < NT; ++j) mma_f64(acc[j], af, bv[j * 8], bv[4 * LDS + j * 8]);
    }
    if (more) put(b ^ 1);
    __syncthreads();
  }

  // sum the shares of the tiles in order: share s adds its block to slot mt
  // of [MT][16][NP] once share s - 1 has
  double *slot = sm64;
  constexpr int ROWS = MT * 16;
#pragma unroll 1
  for (int s = 0; s < KS; ++s) {
    if (ks == s) {
      double *d = slot + mt * 16 * NP;
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          double *e = d + (g + 8 * (q >> 1)) * NP + j * 8 + 2 * t + (q & 1);
          *e = s == 0 ? acc[j][q] : *e + acc[j][q];
        }
    }
    __syncthreads();
  }
  // the cluster's blocks hold their parts of the reduction: each adds and
  // stores a slice of the outputs
  namespace cg = cooperative_groups;
  const int z = gridDim.z;
  int rank = 0, ra = 0, rb = ROWS;
  if (z > 1) {
    cg::cluster_group cl = cg::this_cluster();
    rank = (int)cl.block_rank();
    ra = ROWS * rank / z;
    rb = ROWS * (rank + 1) / z;
    cl.sync();
  }
  __shared__ double red[kThreads];
  constexpr int RG = kThreads / NP;  // row groups of the store
  const int c = tid % NP, rg = tid / NP, o0 = blockIdx.x * ROWS;
  double d = 0.0;
  if (rg < RG && c0 + c < a.R) {
    for (int o = ra + rg; o < rb && o0 + o < M; o += RG) {
      double v = z > 1 ? *cg::this_cluster().map_shared_rank(slot + o * NP + c, 0) : slot[o * NP + c];
      for (int k = 1; k < z; ++k) v += *cg::this_cluster().map_shared_rank(slot + o * NP + c, k);
      v *= a.coef;
      const size_t at = (size_t)(o0 + o) * a.R + c0 + c;
      a.out[at] = v;
      if (a.part) d += a.pdot[at] * v;
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

}  // namespace p64
}  // namespace mbc
