// Dispatch of the FP64 point-kernel products (matvec64.cuh).
#include <type_traits>

#include <cuda_runtime.h>

#include "cuda_util.h"
#include "matvec64.cuh"
#include "matvec64.h"
#include "solver.h"

namespace mbc {

namespace {

struct Cfg {
  int nt, groups, z;
};

// The split of an M x K product over R columns: the fewest column groups of at
// most 64, and the smallest cluster (1, 2, 4, 8 blocks along the reduction)
// that gives a thousand blocks, seven per SM: fewer leave SMs idle or a last
// wave short, larger clusters cost more to start and to add up.  Measured
// (B200, us of K; clusters of 1 / 2 / 4 / 8): 3000 x 3000, 12 columns 123 / 82 /
// 75 / 71; 20000, 60 columns 3351 / 2716 / 2432 / 2669; 32000, 96 columns
// 10666 / 10564 / 10913 / 11651.
Cfg pick(int M, int K, int R)
{
  Cfg c{};
  c.groups = (int)cdiv(R, 8 * p64::kNtMax);
  const int need = (int)cdiv(cdiv(R, c.groups), 8);
  c.nt = need == 5 ? 6 : need == 7 ? 8 : need;
  const int64_t blocks = (int64_t)cdiv(M, p64::kRows) * c.groups;
  for (c.z = 1; c.z < 8 && blocks * c.z < 1000 && (int)cdiv(K, p64::kKT) >= 4 * c.z; c.z *= 2) {
  }
  return c;
}

template <int DIR, int NT, class Ker>
void launch(const Solver &S, const p64::Args &a, const Cfg &c, int M, cudaStream_t st)
{
  constexpr int smem = p64::smem_bytes<DIR>(NT);
  constexpr int id = (std::is_same<Ker, SingleLayer64>::value * 2 + DIR) * p64::kNtMax + NT - 1;
  if (!S.p64_smem[id]) {  // once per solver: the attribute calls cost more than a small product
    allow_max_smem(p64::pk64_kernel<DIR, NT, Ker>, smem);
    S.p64_smem[id] = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(cdiv(M, p64::kRows), c.groups, c.z);
  cfg.blockDim = dim3(p64::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = c.z;
  cfg.attrs = at;
  cfg.numAttrs = c.z > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, p64::pk64_kernel<DIR, NT, Ker>, a);  // an error stays pending for the caller's check
}

// the product; returns the rows of the curvature partials
template <int DIR, class Ker>
int product(const Solver &S, int R, const double *in, double *out, double coef, const double *pdot, double *part,
            const int32_t *done, cudaStream_t st)
{
  const int M = DIR == 0 ? S.nf : S.n, K = DIR == 0 ? S.n : S.nf;
  const Cfg c = pick(M, K, R);
  p64::Args a{};
  a.xr = S.x4();
  a.nr = S.n4();
  a.ys = S.y4();
  a.nf = S.nf;
  a.n = S.n;
  a.in = in;
  a.out = out;
  a.R = R;
  a.coef = coef;
  a.pdot = pdot;
  a.part = part;
  a.done = done;
  switch (c.nt) {
    case 1: launch<DIR, 1, Ker>(S, a, c, M, st); break;
    case 2: launch<DIR, 2, Ker>(S, a, c, M, st); break;
    case 3: launch<DIR, 3, Ker>(S, a, c, M, st); break;
    case 4: launch<DIR, 4, Ker>(S, a, c, M, st); break;
    case 6: launch<DIR, 6, Ker>(S, a, c, M, st); break;
    default: launch<DIR, 8, Ker>(S, a, c, M, st); break;
  }
  ++S.launches;
  return (int)cdiv(M, p64::kRows) * c.z;
}

}  // namespace

void p64_launch_rows(const Solver &S, int R, const double *v, double *w, const int32_t *done, cudaStream_t st)
{
  product<0, PointKernel<double>>(S, R, v, w, S.op.coef, nullptr, nullptr, done, st);
}

int p64_launch_cols(const Solver &S, int R, const double *w, double *t, const double *pdot, double *part,
                    const int32_t *done, cudaStream_t st)
{
  return product<1, PointKernel<double>>(S, R, w, t, S.op.coef, pdot, part, done, st);
}

void p64_launch_potential(const Solver &S, int R, const double *x, double *phi, cudaStream_t st)
{
  product<0, SingleLayer64>(S, R, x, phi, 1.0 / (4.0 * 3.14159265358979323846), nullptr, nullptr, nullptr, st);
}

}  // namespace mbc
