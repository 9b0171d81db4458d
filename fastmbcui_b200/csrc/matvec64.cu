// Dispatch of the FP64 point-kernel products (matvec64.cuh).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include <cuda_runtime.h>

#include "cuda_util.h"
#include "matvec64.cuh"
#include "matvec64.h"
#include "solver.h"

namespace mbc {

namespace {

constexpr double kSMs = 148.0;
constexpr size_t kPartsBytes = (size_t)64 << 20;  // most that the partial blocks of a split may take

struct Cfg {
  int nt, groups, mt, parts;
};

// The split of an M x K product over R columns.  Blocks of one SM share its
// FP64 pipe, so a launch lasts as long as the SM with the most blocks:
// ceil(blocks parts / 148) blocks of 16 mt K / parts entries at 16 + 8 nt
// FP64 multiply-adds each, plus ~2 us a block to start and to sum its shares,
// and no shorter than its reads of the vector block from L2 (~6 TB/s).
// Splitting the reduction (parts > 1) costs a second kernel and the partial
// blocks' round trip.  The shape with the smallest estimate is taken: at
// R = 12 and 3000 points 16 outputs per block and no split, at R = 60 and
// 20000 points 64 outputs and a split that fills the last wave.
Cfg pick(int M, int K, int R)
{
  Cfg c{};
  c.groups = (int)cdiv(R, 8 * p64::kNtMax);
  const int need = (int)cdiv(cdiv(R, c.groups), 8);
  for (int nt : {1, 2, 3, 4, 6, 8})
    if (nt >= need) {
      c.nt = nt;
      break;
    }
  const double np = 8.0 * c.nt, rate = 64.0 * 1.8e3;  // multiply-adds per us and SM
  double best = 1e300;
  for (int mt : {4, 2, 1})
    for (int parts = 1; parts <= 8; ++parts) {
      if (parts > 1 && ((size_t)parts * M * R * sizeof(double) > kPartsBytes || (int)cdiv(K, p64::kKT) < 4 * parts)) break;
      const double blocks = (double)cdiv(M, 16 * mt) * c.groups;
      const double work = 16.0 * mt * K * (16.0 + np) / rate / parts;
      const double l2 = blocks * K * np * 8.0 / 6e6;
      double t = std::max(std::ceil(blocks * parts / kSMs) * (work + 2.0), l2);
      if (parts > 1) t += 4.0 + 2.0 * parts * (double)M * R * 8.0 / 5e6;
      if (t < 0.98 * best) {
        best = t;
        c.mt = mt;
        c.parts = parts;
      }
    }
  return c;
}

template <int DIR, int NT, int MT, class Ker>
void launch(const Solver &S, const p64::Args &a, const Cfg &c, int M, cudaStream_t st)
{
  constexpr int smem = p64::smem_bytes<DIR>(NT);
  constexpr int id = ((std::is_same<Ker, SingleLayer64>::value * 2 + DIR) * 3 + MT / 2) * p64::kNtMax + NT - 1;
  if (!S.p64_smem[id]) {  // once per solver: the attribute calls cost more than a small product
    allow_max_smem(p64::pk64_kernel<DIR, NT, MT, Ker>, smem);
    S.p64_smem[id] = true;
  }
  p64::pk64_kernel<DIR, NT, MT, Ker><<<dim3(cdiv(M, 16 * MT), c.groups, c.parts), p64::kThreads, smem, st>>>(a);
}

template <int DIR, int NT, class Ker>
void by_mt(const Solver &S, const p64::Args &a, const Cfg &c, int M, cudaStream_t st)
{
  switch (c.mt) {
    case 4: launch<DIR, NT, 4, Ker>(S, a, c, M, st); break;
    case 2: launch<DIR, NT, 2, Ker>(S, a, c, M, st); break;
    default: launch<DIR, NT, 1, Ker>(S, a, c, M, st); break;
  }
}

// the product; returns the rows of the curvature partials
template <int DIR, class Ker>
int product(const Solver &S, int R, const double *in, double *out, double coef, const double *pdot, double *part,
            const int32_t *done, cudaStream_t st)
{
  const int M = DIR == 0 ? S.nf : S.n, K = DIR == 0 ? S.n : S.nf;
  Cfg c = pick(M, K, R);
  if (c.parts > 1 && S.m_p64.reserve((size_t)c.parts * M * R * sizeof(double)) != MBC_OK) c.parts = 1;
  p64::Args a{};
  a.xr = S.x4();
  a.nr = S.n4();
  a.ys = S.y4();
  a.nf = S.nf;
  a.n = S.n;
  a.in = in;
  a.out = out;
  a.parts = (double *)S.m_p64.ptr;
  a.nparts = c.parts;
  a.R = R;
  a.groups = c.groups;
  a.coef = coef;
  a.pdot = pdot;
  a.part = part;
  a.done = done;
  switch (c.nt) {
    case 1: by_mt<DIR, 1, Ker>(S, a, c, M, st); break;
    case 2: by_mt<DIR, 2, Ker>(S, a, c, M, st); break;
    case 3: by_mt<DIR, 3, Ker>(S, a, c, M, st); break;
    case 4: by_mt<DIR, 4, Ker>(S, a, c, M, st); break;
    case 6: by_mt<DIR, 6, Ker>(S, a, c, M, st); break;
    default: by_mt<DIR, 8, Ker>(S, a, c, M, st); break;
  }
  ++S.launches;
  if (c.parts == 1) return (int)cdiv(M, 16 * c.mt);
  const unsigned blocks = cdiv(M, p64::kSumRows);
  p64::pk64_sum_kernel<<<blocks, 256, 0, st>>>(M, R, c.parts, a.parts, coef, out, pdot, part, done);
  ++S.launches;
  return (int)blocks;
}

}  // namespace

mbc_status p64_reserve(const Solver &S, int R)
{
  if (S.op.kind != MBC_OP_POINT_KERNEL) return MBC_OK;
  size_t b = 0;
  for (int dir = 0; dir < 2; ++dir) {
    const int M = dir == 0 ? S.nf : S.n, K = dir == 0 ? S.n : S.nf;
    const Cfg c = pick(M, K, R);
    if (c.parts > 1) b = std::max(b, (size_t)c.parts * M * R * sizeof(double));
  }
  return b ? S.m_p64.reserve(b) : MBC_OK;
}

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
