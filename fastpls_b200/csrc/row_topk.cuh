// The largest entries of every row of a score matrix (class scores, candidate
// scores): descending values, the earlier class first on ties, NaN never.
#pragma once

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "context.cuh"

namespace fpls {

constexpr int kRowTopkMax = 32;

// S (w x C, column-major, ld w), bias (C) or null added to every row.  A block
// takes 32 rows; lane = row, so every load of a warp is 256 contiguous bytes,
// and warp g scans the classes g, g + G, ... four loads at a time into a sorted
// list of K in registers.  The G lists of a row are then merged in shared
// memory.  (One thread a row with its list in local memory left 157 blocks
// waiting for dependent local stores: 20000 x 1000, top 5: 818 us against 58 us.)
// Entries that no class fills: index `empty`, score -inf.  first_nan: a row
// whose first score is NaN yields `empty` (the argmax rule: nothing exceeds it).
template <int K>
__global__ void __launch_bounds__(K <= 8 ? 1024 : 256) row_topk_kernel(const double* __restrict__ S, int w, int C,
                                                        const double* __restrict__ bias, int top_k, int empty,
                                                        bool first_nan, int* __restrict__ idx,
                                                        double* __restrict__ score) {
  extern __shared__ double sv[];   // [G][K][32] values, then the classes
  constexpr int kNone = 0x7fffffff;
  const int G = blockDim.x >> 5, g = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* si = reinterpret_cast<int*>(sv + (size_t)G * K * 32);
  const int i = blockIdx.x * 32 + lane;
  double vals[K];
  int ids[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    vals[j] = -INFINITY;
    ids[j] = kNone;
  }
  auto insert = [&](double v, int c) {
    if (v > vals[K - 1]) {
      vals[K - 1] = v;
      ids[K - 1] = c + 1;
#pragma unroll
      for (int j = K - 1; j > 0; --j) {
        if (vals[j] > vals[j - 1]) {
          const double tv = vals[j];
          vals[j] = vals[j - 1];
          vals[j - 1] = tv;
          const int ti = ids[j];
          ids[j] = ids[j - 1];
          ids[j - 1] = ti;
        }
      }
    }
  };
  if (i < w) {
    const double* row = S + i;
    int c = g;
    for (; c + 3 * G < C; c += 4 * G) {
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldg(row + (size_t)(c + u * G) * w);
#pragma unroll
      for (int u = 0; u < 4; ++u) insert(bias ? v[u] + bias[c + u * G] : v[u], c + u * G);
    }
    for (; c < C; c += G) {
      const double v = __ldg(row + (size_t)c * w);
      insert(bias ? v + bias[c] : v, c);
    }
  }
#pragma unroll
  for (int j = 0; j < K; ++j) {
    sv[(g * K + j) * 32 + lane] = vals[j];
    si[(g * K + j) * 32 + lane] = ids[j];
  }
  __syncthreads();
  // pairwise merges: warp g takes the lists g and g + half, the better K of both
  for (int half = G / 2; half >= 1; half /= 2) {
    if (g < half) {
      int p = 0, q = 0;
      const double *va = sv + (size_t)g * K * 32 + lane, *vb = sv + (size_t)(g + half) * K * 32 + lane;
      const int *ia = si + (size_t)g * K * 32 + lane, *ib = si + (size_t)(g + half) * K * 32 + lane;
      double x = va[0], y = vb[0];
      int xi = ia[0], yi = ib[0];
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const bool a = x > y || (x == y && xi <= yi);
        vals[j] = a ? x : y;
        ids[j] = a ? xi : yi;
        if (a) {
          ++p;
          x = p < K ? va[p * 32] : -INFINITY;
          xi = p < K ? ia[p * 32] : kNone;
        } else {
          ++q;
          y = q < K ? vb[q * 32] : -INFINITY;
          yi = q < K ? ib[q * 32] : kNone;
        }
      }
    }
    __syncthreads();
    if (g < half) {
#pragma unroll
      for (int j = 0; j < K; ++j) {
        sv[(g * K + j) * 32 + lane] = vals[j];
        si[(g * K + j) * 32 + lane] = ids[j];
      }
    }
    __syncthreads();
  }
  if (g == 0 && i < w) {
    bool none = false;
    if (first_nan) none = isnan(bias ? S[i] + bias[0] : S[i]);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (j >= top_k) break;
      const bool take = !none && ids[j] != kNone;
      idx[i + (size_t)j * w] = take ? ids[j] : empty;
      if (score) score[i + (size_t)j * w] = take ? vals[j] : -INFINITY;
    }
  }
}

// idx / score: w x top_k (ld w); top_k up to kRowTopkMax.  The list length is
// rounded up to one of eight.  Up to 8 warps for 32 rows; 32 where the rows alone
// do not give every SM two blocks and the lists fit the registers of 1024 threads
// (then the scan, not the merge, is the time), but no warp without a class, and 8
// classes a warp at least where the rows fill the GPU by themselves.
inline void row_topk_launch(const double* S, int w, int C, const double* bias, int top_k, int empty, bool first_nan,
                            int* idx, double* score) {
  Context& ctx = Context::get();
  auto go = [&](auto kernel, int K) {
    const bool many = ceil_div(w, 32) >= 2 * ctx.sm_count;
    int G = K > 8 || many ? 8 : 32;
    while (G > 1 && C < (many ? 8 * G : G)) G /= 2;
    const size_t smem = (size_t)G * K * 32 * 12;
    if (smem > 48 * 1024)
      FPLS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    kernel<<<ceil_div(w, 32), 32 * G, smem, ctx.stream>>>(S, w, C, bias, top_k, empty, first_nan, idx, score);
  };
  if (top_k <= 1) go(row_topk_kernel<1>, 1);
  else if (top_k <= 3) go(row_topk_kernel<3>, 3);
  else if (top_k <= 5) go(row_topk_kernel<5>, 5);
  else if (top_k <= 8) go(row_topk_kernel<8>, 8);
  else if (top_k <= 12) go(row_topk_kernel<12>, 12);
  else if (top_k <= 16) go(row_topk_kernel<16>, 16);
  else if (top_k <= 20) go(row_topk_kernel<20>, 20);
  else go(row_topk_kernel<32>, 32);
  note_launch();
  FPLS_CHECK_LAUNCH();
}

}  // namespace fpls
