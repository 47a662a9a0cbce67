// FP64 tensor-core (DMMA) GEMM tiles: C = alpha op(A) op(B) (+ beta C, + a row
// vector), column-major.
//
// FP64 has no tcgen05 kind; mma.sync m8n8k4 is the FP64 tensor path, 64
// multiply-adds a clock and SM.  What a product loses against that is padding
// (the product's column counts are those of components, classes, fits: 5, 30,
// 50, 100), an uneven last wave and, in short contractions, the wait for the
// first tiles.  So a CTA takes 64 rows by 8 NT columns with NT picked for the
// column count, four warps of 16 x 8 NT, and tiles of 16 contraction steps come
// in by cp.async through kStages buffers, 16 bytes at a time where the operands
// are aligned for it.  A K-contiguous operand keeps its rows contiguous in
// shared memory (stride 20), the other its columns (stride width + 4): fills and
// fragment loads of both are free of bank conflicts, so no transposed copies
// are made.
//
// The sum over a K range runs in the order of the contraction, four terms a
// DMMA, whatever NT is: results do not depend on the tile shape.
#pragma once

#include "common.cuh"

namespace fpls {
namespace gemm64 {

constexpr int kBM = 64;
constexpr int kBK = 16;
constexpr int kThreads = 128;

struct Args {
  int M, N, K;
  double alpha;
  const double* A;
  int lda;
  const double* B;
  int ldb;
  double beta;
  double* C;
  int ldc;
  int k_per_split;
  long long split_stride;   // > 0: K range z stores its own partial at C + z * stride
  int upper;                // skip tiles entirely below the diagonal
  const double* row_add;    // added to every row of the result (null: nothing), no splits
};

template <bool KC, int MN>
struct Tile {
  static constexpr int kStride = KC ? kBK + 4 : MN + 4;
  static constexpr int kSize = KC ? MN * kStride : kBK * kStride;
  static __device__ __forceinline__ int at(int mn, int k) { return KC ? mn * kStride + k : k * kStride + mn; }
};

template <int BYTES>
__device__ __forceinline__ void copy_async(double* dst, const double* src, int valid) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(BYTES), "r"(valid) : "memory");
}

// Fills one tile (MN x kBK); elements outside the operand or the K range read as zero.
template <bool KC, int MN, int V>   // V doubles a copy
__device__ __forceinline__ void fill_tile(double* S, const double* __restrict__ P, int ld, int mn0, int k0, int limit,
                                          int kend) {
  constexpr int kChunks = MN * kBK / V;
#pragma unroll
  for (int t0 = 0; t0 < kChunks; t0 += kThreads) {
    const int t = t0 + threadIdx.x;
    if (kChunks % kThreads && t >= kChunks) break;
    int mn, k, left;
    if (KC) {
      k = (t % (kBK / V)) * V;
      mn = t / (kBK / V);
      left = mn0 + mn < limit ? kend - (k0 + k) : 0;
    } else {
      mn = (t % (MN / V)) * V;
      k = t / (MN / V);
      left = k0 + k < kend ? limit - (mn0 + mn) : 0;
    }
    const int n = left < 0 ? 0 : left < V ? left : V;
    const double* src = n ? (KC ? P + (size_t)(mn0 + mn) * ld + k0 + k : P + mn0 + mn + (size_t)(k0 + k) * ld) : P;
    copy_async<8 * V>(S + Tile<KC, MN>::at(mn, k), src, 8 * n);
  }
}

template <int NT>
constexpr int kStages = NT <= 2 ? 6 : NT <= 5 ? 4 : 3;

template <bool TA, bool TB, int NT>
constexpr size_t smem_bytes() {
  return sizeof(double) * kStages<NT> * (Tile<TA, kBM>::kSize + Tile<!TB, 8 * NT>::kSize);
}

// op(A) (m,k): TA ? A[k + m*lda] : A[m + k*lda]   -> K-contiguous when TA
// op(B) (k,n): TB ? B[n + k*ldb] : B[k + n*ldb]   -> K-contiguous when !TB
template <bool TA, bool TB, int NT, int V>
__global__ void __launch_bounds__(kThreads) gemm_f64_dmma(Args g) {
  extern __shared__ __align__(16) double gemm_sm[];
  constexpr int BN = 8 * NT, S = kStages<NT>;
  using TileA = Tile<TA, kBM>;
  using TileB = Tile<!TB, BN>;
  double* As = gemm_sm;
  double* Bs = gemm_sm + S * TileA::kSize;
  const int bm = blockIdx.x * kBM, bn = blockIdx.y * BN;
  if (g.upper && bm >= bn + BN) return;
  const int kbeg = blockIdx.z * g.k_per_split;
  const int kend = min(g.K, kbeg + g.k_per_split);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int wm = warp * 16;
  double acc[2][NT][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int nblk = kbeg < kend ? (kend - kbeg + kBK - 1) / kBK : 0;
  auto load = [&](int b) {
    if (b < nblk) {
      const int st = b % S;
      fill_tile<TA, kBM, V>(As + st * TileA::kSize, g.A, g.lda, bm, kbeg + b * kBK, g.M, kend);
      fill_tile<!TB, BN, V>(Bs + st * TileB::kSize, g.B, g.ldb, bn, kbeg + b * kBK, g.N, kend);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int b = 0; b < S - 1; ++b) load(b);
  for (int b = 0; b < nblk; ++b) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
    __syncthreads();
    load(b + S - 1);
    const double* a_s = As + (b % S) * TileA::kSize;
    const double* b_s = Bs + (b % S) * TileB::kSize;
    const int kleft = kend - (kbeg + b * kBK);
    double fa[2][2], fb[2][NT];
    auto load_step = [&](int s4, int buf) {
#pragma unroll
      for (int i = 0; i < 2; ++i) fa[buf][i] = a_s[TileA::at(wm + i * 8 + gid, 4 * s4 + tig)];
#pragma unroll
      for (int j = 0; j < NT; ++j) fb[buf][j] = b_s[TileB::at(j * 8 + gid, 4 * s4 + tig)];
    };
    auto multiply = [&](int buf) {
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) dmma_8x8x4(acc[i][j][0], acc[i][j][1], fa[buf][i], fb[buf][j]);
    };
    if (kleft >= kBK) {
      // the next step's fragments load under this step's products: one warp a
      // scheduler is enough to keep the tensor pipe busy
      load_step(0, 0);
#pragma unroll
      for (int s4 = 0; s4 < kBK / 4; ++s4) {
        if (s4 + 1 < kBK / 4) load_step(s4 + 1, (s4 + 1) & 1);
        multiply(s4 & 1);
      }
    } else {   // the range's last tile: nothing but zeros after kleft
      for (int s4 = 0; 4 * s4 < kleft; ++s4) {
        load_step(s4, 0);
        multiply(0);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = bm + wm + i * 8 + gid;
    if (m >= g.M) continue;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = bn + j * 8 + tig * 2 + e;
        if (n >= g.N) continue;
        // split-K: each K range stores its own partial (summed in range order
        // by splitk_reduce_kernel, so runs repeat bit for bit)
        double* cp = g.C + (size_t)blockIdx.z * g.split_stride + m + (size_t)n * g.ldc;
        double v = g.alpha * acc[i][j][e];
        if (!g.split_stride && g.beta != 0.0) v += g.beta * *cp;
        if (g.row_add) v += g.row_add[n];
        *cp = v;
      }
    }
  }
}

// Launches the tile kernel of (TA, TB) for 8 nt columns a tile (one of kWidths).
constexpr int kWidths[] = {1, 2, 4, 5, 7, 8, 10, 13};
template <bool TA, bool TB>
void launch(const Args& g, int nt, bool vec, dim3 grid, cudaStream_t st);

template <bool TA, bool TB, int NT>
void launch_width(const Args& g, bool vec, dim3 grid, cudaStream_t st) {
  constexpr size_t smem = smem_bytes<TA, TB, NT>();
  static const bool once = [] {
    FPLS_CUDA(cudaFuncSetAttribute(gemm_f64_dmma<TA, TB, NT, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    FPLS_CUDA(cudaFuncSetAttribute(gemm_f64_dmma<TA, TB, NT, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return true;
  }();
  (void)once;
  if (vec) gemm_f64_dmma<TA, TB, NT, 2><<<grid, kThreads, smem, st>>>(g);
  else gemm_f64_dmma<TA, TB, NT, 1><<<grid, kThreads, smem, st>>>(g);
}

#define FPLS_GEMM64_INSTANTIATE(TA, TB)                                              \
  namespace fpls {                                                                   \
  namespace gemm64 {                                                                 \
  template <>                                                                        \
  void launch<TA, TB>(const Args& g, int nt, bool vec, dim3 grid, cudaStream_t st) { \
    switch (nt) {                                                                    \
      case 1: launch_width<TA, TB, 1>(g, vec, grid, st); break;                      \
      case 2: launch_width<TA, TB, 2>(g, vec, grid, st); break;                      \
      case 4: launch_width<TA, TB, 4>(g, vec, grid, st); break;                      \
      case 5: launch_width<TA, TB, 5>(g, vec, grid, st); break;                      \
      case 7: launch_width<TA, TB, 7>(g, vec, grid, st); break;                      \
      case 8: launch_width<TA, TB, 8>(g, vec, grid, st); break;                      \
      case 10: launch_width<TA, TB, 10>(g, vec, grid, st); break;                    \
      default: launch_width<TA, TB, 13>(g, vec, grid, st); break;                    \
    }                                                                                \
    note_launch();                                                                   \
    FPLS_CHECK_LAUNCH();                                                             \
  }                                                                                  \
  }                                                                                  \
  }

}  // namespace gemm64
}  // namespace fpls
