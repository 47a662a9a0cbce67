// The largest entries of every row of a score matrix (class scores, candidate
// scores): descending values, the earlier class first on ties, NaN never.
#pragma once

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "context.cuh"

namespace fpls {

constexpr int kRowTopkMax = 32;

// S (w x C, column-major, ld w), bias (C) or null added to every row.  G warps
// take 32 rows; lane = row, so every load of a warp is 256 contiguous bytes,
// and warp g scans the classes g, g + G, ... four loads at a time into a sorted
// list of K in registers.  The G lists of a row are then merged in shared
// memory; one list (few classes) is the result, and a block takes several such
// groups of rows.  (One thread a row with its list in local memory left 157 blocks
// waiting for dependent local stores: 20000 x 1000, top 5: 818 us against 58 us.)
// Entries that no class fills: index `empty`, score -inf.  first_nan: a row
// whose first score is NaN yields `empty` (the argmax rule: nothing exceeds it).
template <int K>
__global__ void __launch_bounds__(K <= 8 ? 1024 : 256) row_topk_kernel(const double* __restrict__ S, int w, int C,
                                                        const double* __restrict__ bias, int top_k, int empty,
                                                        bool first_nan, int G, int* __restrict__ idx,
                                                        double* __restrict__ score) {
  extern __shared__ double shared_lists[];   // a group: [G][K][32] values, then the classes
  constexpr int kNone = 0x7fffffff;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = warp / G, g = warp - group * G;
  double* sv = shared_lists + (size_t)group * G * K * 48;
  int* si = reinterpret_cast<int*>(sv + (size_t)G * K * 32);
  const int i = (blockIdx.x * (static_cast<int>(blockDim.x >> 5) / G) + group) * 32 + lane;
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
  if (G > 1) {
#pragma unroll
    for (int j = 0; j < K; ++j) {
      sv[(g * K + j) * 32 + lane] = vals[j];
      si[(g * K + j) * 32 + lane] = ids[j];
    }
    __syncthreads();
  }
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
// (then the scan, not the merge, is the time), but never fewer than 16 classes a
// warp: the best 2 of 3 classes for 3000 rows took 6.0 us with 8 warps for 32 rows,
// 4.4 with one.
inline void row_topk_launch(const double* S, int w, int C, const double* bias, int top_k, int empty, bool first_nan,
                            int* idx, double* score) {
  Context& ctx = Context::get();
  auto go = [&](auto kernel, int K) {
    int G = K > 8 || ceil_div(w, 32) >= 2 * ctx.sm_count ? 8 : 32;
    while (G > 1 && C < 16 * G) G /= 2;
    const int groups = G >= 8 ? 1 : ceil_div(w, 256) >= 2 * ctx.sm_count ? 8 / G : 1;
    const size_t smem = G > 1 ? (size_t)groups * G * K * 32 * 12 : 0;
    if (smem > 48 * 1024)
      FPLS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    kernel<<<ceil_div(w, 32 * groups), 32 * G * groups, smem, ctx.stream>>>(S, w, C, bias, top_k, empty, first_nan, G, idx,
                                                                           score);
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
