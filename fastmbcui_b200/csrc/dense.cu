// Dispatch of the dense products (dense.cuh).
#include <algorithm>
#include <cstdint>

#include <cuda_runtime.h>

#include "cuda_util.h"
#include "dense.cuh"
#include "dense.h"
#include "solver.h"

namespace mbc {

namespace {

// Blocks of a cluster along the reduction axis.  The blocks of an SM share
// its issue slots, so a launch lasts as long as the SM with the most blocks,
// a block as long as its tiles plus about two tiles' time to fill the
// pipeline and to sum over its warps and its cluster.  The smallest estimate
// wins: 5 blocks of 3 tiles (one coarse mesh body) are cut to single tiles,
// the 240 row blocks of three fine bodies into clusters of 4.
// FP32 rows (short) take at least 4 blocks, and up to 16 tiles one block per
// one or two: a warp's chain of roundings is then no longer than the K / 32 of
// a lane of a warp per output, and the error against 64 bits no larger
// (30000 x 3000, 12 columns: 1.85e-7, with one block 2.52e-7).  The time is the
// same to a few percent at every size.
int pick_cluster(int M, int K, int groups, bool short_chains)
{
  const int64_t blocks = (int64_t)cdiv(M, dns::kBM) * groups;
  const int tiles = (int)cdiv(K, dns::kBK);
  const int zmin = !short_chains ? 1 : tiles > 16 ? 4 : std::min(tiles, dns::kMaxCluster);
  int best = zmin;
  double tbest = 1e300;
  for (int z = zmin; z <= dns::kMaxCluster && z <= tiles; z *= 2) {
    const double t = (double)cdiv(blocks * z, 148) * ((double)cdiv(tiles, z) + (z > 1 ? 2.25 : 2.0));
    if (t < tbest) {
      tbest = t;
      best = z;
    }
  }
  return best;
}

template <typename T, int DIR, int NT>
void launch(const Solver &S, const dns::Args &a, unsigned blocks, unsigned groups, int z, cudaStream_t st)
{
  constexpr int smem = dns::smem_bytes<T, DIR>(NT);
  constexpr int id = ((sizeof(T) == 8) * 2 + DIR) * 8 + NT - 1;
  if (!S.dense_smem[id]) {  // once per solver
    allow_max_smem(dns::dense_kernel<T, DIR, NT>, smem);
    S.dense_smem[id] = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks, groups, z);
  cfg.blockDim = dim3(dns::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = z;
  cfg.attrs = at;
  cfg.numAttrs = z > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, dns::dense_kernel<T, DIR, NT>, a);  // an error stays pending for the caller's check
}

template <typename T, int DIR>
int product(const Solver &S, int R, const T *in, T *out, const T *pdot, double *part, const int32_t *done,
            cudaStream_t st)
{
  const int M = DIR == 0 ? S.nf : S.n, K = DIR == 0 ? S.n : S.nf;
  constexpr int unit = sizeof(T) == 4 ? 4 : 8;
  const int groups = (int)cdiv(R, 32);
  int nt = (int)cdiv(cdiv(R, groups), unit);
  if (nt == 7) nt = 8;
  dns::Args a{};
  a.M = S.op.M;
  a.ldm = S.op.ldm;
  a.nf = S.nf;
  a.n = S.n;
  a.P = S.dP();
  a.in = in;
  a.out = out;
  a.R = R;
  const uintptr_t at = (uintptr_t)S.op.M;
  a.vec = at % 16 == 0 && S.op.ldm % 4 == 0 ? 16 : at % 8 == 0 && S.op.ldm % 2 == 0 ? 8 : 4;
  // a row of the vector block is R elements: copies of several need R (and so
  // every row and column group, a multiple of 4 units) to be a multiple too
  constexpr int et = (int)sizeof(T);
  a.vecv = (uintptr_t)in % 16 == 0 && R % (16 / et) == 0 ? 16 : et == 4 && (uintptr_t)in % 8 == 0 && R % 2 == 0 ? 8 : et;
  a.pdot = pdot;
  a.part = part;
  a.done = done;
  const int z = pick_cluster(M, K, groups, sizeof(T) == 4 && DIR == 0);
  const unsigned blocks = cdiv(M, dns::kBM);
  switch (nt) {
    case 1: launch<T, DIR, 1>(S, a, blocks, groups, z, st); break;
    case 2: launch<T, DIR, 2>(S, a, blocks, groups, z, st); break;
    case 3: launch<T, DIR, 3>(S, a, blocks, groups, z, st); break;
    case 4: launch<T, DIR, 4>(S, a, blocks, groups, z, st); break;
    default:
      if constexpr (sizeof(T) == 4) {
        if (nt == 5) launch<T, DIR, 5>(S, a, blocks, groups, z, st);
        else if (nt == 6) launch<T, DIR, 6>(S, a, blocks, groups, z, st);
        else launch<T, DIR, 8>(S, a, blocks, groups, z, st);
      }
  }
  ++S.launches;
  return (int)blocks * z;
}

}  // namespace

template <typename T>
void dense_launch_rows(const Solver &S, int R, const T *v, T *w, const int32_t *done, cudaStream_t st)
{
  product<T, 0>(S, R, v, w, nullptr, nullptr, done, st);
}

template <typename T>
int dense_launch_cols(const Solver &S, int R, const T *w, T *t, const T *pdot, double *part, const int32_t *done,
                      cudaStream_t st)
{
  return product<T, 1>(S, R, w, t, pdot, part, done, st);
}

template void dense_launch_rows<float>(const Solver &, int, const float *, float *, const int32_t *, cudaStream_t);
template void dense_launch_rows<double>(const Solver &, int, const double *, double *, const int32_t *, cudaStream_t);
template int dense_launch_cols<float>(const Solver &, int, const float *, float *, const float *, double *,
                                      const int32_t *, cudaStream_t);
template int dense_launch_cols<double>(const Solver &, int, const double *, double *, const double *, double *,
                                       const int32_t *, cudaStream_t);

}  // namespace mbc
