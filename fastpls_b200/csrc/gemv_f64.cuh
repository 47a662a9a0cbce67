// FP64 matrix-vector product bodies, shared by the GEMV kernels and the one-launch
// SIMPLS loop: the order of every sum is theirs, not the caller's.
#pragma once

#include "common.cuh"

namespace fpls {

constexpr int kGemvRows = 256;   // rows (threads) of one block of y = A x

// Column ranges of y = A x (rows x cols): blocks of kGemvRows rows times `splits`
// ranges of kps columns, partials added in range order.
struct GemvRanges { int row_blocks, splits, kps; };
inline GemvRanges gemv_ranges(int rows, int cols, int sm_count) {
  GemvRanges g{ceil_div(rows, kGemvRows), 1, cols};
  const int target = 4 * sm_count;
  if (g.row_blocks < target) {
    const int a = ceil_div(target, g.row_blocks), b = ceil_div(cols, 256);
    g.splits = a < b ? a : b;
    if (g.splits < 1) g.splits = 1;
  }
  g.kps = ceil_div(cols, g.splits);
  g.splits = ceil_div(cols, g.kps);
  return g;
}

// Row ranges of y = A^T x that SIMPLS takes for one fit: a warp a column leaves a
// tall matrix of few columns with too few loads in flight (50000 x 1000: 214 us
// for 400 MB, five ranges 66 us), so columns get ranges until there are 32 warps
// an SM, each of at least 8192 rows.  One range up to 2^22 elements, where the
// one-launch loop takes whole columns and the sums have to be its.
inline GemvRanges gemv_t_ranges(int rows, int cols, int sm_count) {
  GemvRanges g{cols, 1, rows};
  if ((long long)rows * cols > (1ll << 22)) {
    const int a = ceil_div(32 * sm_count, cols), b = rows / 8192;
    g.splits = a < b ? a : b;
    if (g.splits < 1) g.splits = 1;
  }
  g.kps = ceil_div(ceil_div(rows, g.splits), 32) * 32;
  g.splits = ceil_div(rows, g.kps);
  return g;
}

// acc += sum_k a[k * lda] xs[k], k < kn in order; AHEAD loads go out before they
// are multiplied (one after another, a 400 x 2000 product waited 63 times for L2).
template <int AHEAD>
__device__ __forceinline__ double gemv_row(const double* __restrict__ a, size_t lda, const double* xs, int kn, double acc) {
  for (int k = 0; k < kn; k += AHEAD) {
    double v[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) v[u] = k + u < kn ? __ldg(a + (size_t)(k + u) * lda) : 0.0;
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (k + u < kn) acc = fma(v[u], xs[k + u], acc);
  }
  return acc;
}

// a . x over K entries by one warp: lane l takes l, l + 32, ... in order, then a
// shuffle tree (every lane has the result).  x by plain loads.
template <int AHEAD>
__device__ __forceinline__ double gemv_column(const double* __restrict__ a, const double* x, int K) {
  double acc = 0.0;
  for (int k0 = threadIdx.x & 31; k0 < K; k0 += 32 * AHEAD) {
    double v[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) v[u] = k0 + 32 * u < K ? __ldg(a + k0 + 32 * u) : 0.0;
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (k0 + 32 * u < K) acc = fma(v[u], x[k0 + 32 * u], acc);
  }
  return warp_sum(acc);
}

}  // namespace fpls
