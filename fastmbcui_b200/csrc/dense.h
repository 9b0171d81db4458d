// Products of a solver's dense operator (dense.cu).
#pragma once

#include <cuda_runtime.h>

#include "solver.h"

namespace mbc {

// most rows of curvature partials a columns product of n sources writes
inline int dense_part_rows(int n) { return (n + 63) / 64 * 8; }
// w (nf x R) = K v
template <typename T>
void dense_launch_rows(const Solver &S, int R, const T *v, T *w, const int32_t *done, cudaStream_t st);
// t (n x R) = K^T w, optionally with the partials of p . t; returns their rows
template <typename T>
int dense_launch_cols(const Solver &S, int R, const T *w, T *t, const T *pdot, double *part, const int32_t *done,
                      cudaStream_t st);

}  // namespace mbc
