// Completion of the left vectors of negligible singular values, by one CTA.
#pragma once

#include "common.cuh"

namespace fpls {

// Makes u (L entries) orthogonal to the first j columns of U, two Gram-Schmidt
// passes, and returns its squared norm; one CTA.
__device__ inline double orthogonal_to_first(double* u, int L, const double* U, int ldu, int j, double* scratch) {
  for (int pass = 0; pass < 2; ++pass) {
    for (int jj = 0; jj < j; ++jj) {
      const double* uo = U + (size_t)jj * ldu;
      double d = 0.0;
      for (int i = threadIdx.x; i < L; i += blockDim.x) d += uo[i] * u[i];
      d = block_sum(d, scratch);
      for (int i = threadIdx.x; i < L; i += blockDim.x) u[i] -= d * uo[i];
      __syncthreads();
    }
  }
  double nn = 0.0;
  for (int i = threadIdx.x; i < L; i += blockDim.x) nn += u[i] * u[i];
  return block_sum(nn, scratch);
}

// Column j of U (L rows) = a unit vector made orthogonal to the columns before it.
// Candidates: the unit vectors that keep half their length, then any that keeps its
// share (one does: the squared lengths left of all unit vectors add up to the
// dimensions left).
__device__ inline void complete_null_column(int L, int j, double* U, int ldu, double* scratch) {
  double* uj = U + (size_t)j * ldu;
  for (int e = 0; e < 2 * L; ++e) {
    for (int i = threadIdx.x; i < L; i += blockDim.x) uj[i] = (i == e % L) ? 1.0 : 0.0;
    __syncthreads();
    const double nn = orthogonal_to_first(uj, L, U, ldu, j, scratch);
    if (!isfinite(nn)) break;   // a column before it is not finite, and none of the candidates would be
    if (nn > (e < L ? 0.25 : 0.5 / L)) {
      const double inv = 1.0 / sqrt(nn);
      for (int i = threadIdx.x; i < L; i += blockDim.x) uj[i] *= inv;
      __syncthreads();
      if (nn <= 0.25) {   // more length was lost: once more
        const double n2 = orthogonal_to_first(uj, L, U, ldu, j, scratch);
        for (int i = threadIdx.x; i < L; i += blockDim.x) uj[i] /= sqrt(n2);
        __syncthreads();
      }
      break;
    }
  }
}

}  // namespace fpls
