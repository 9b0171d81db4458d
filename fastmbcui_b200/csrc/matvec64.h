// FP64 point-kernel products of a solver (matvec64.cu).
#pragma once

#include <cuda_runtime.h>

#include "solver.h"

namespace mbc {

// most rows of curvature partials a columns product of n sources writes
inline int p64_part_rows(int n) { return (n + 63) / 64 * 8; }
// w (nf x R) = K v
void p64_launch_rows(const Solver &S, int R, const double *v, double *w, const int32_t *done, cudaStream_t st);
// t (n x R) = K^T w, optionally with the partials of p . t; returns their rows
int p64_launch_cols(const Solver &S, int R, const double *w, double *t, const double *pdot, double *part,
                    const int32_t *done, cudaStream_t st);
// phi (nf x R) = single-layer potential of x (n x R) over 4 pi
void p64_launch_potential(const Solver &S, int R, const double *x, double *phi, cudaStream_t st);

}  // namespace mbc
