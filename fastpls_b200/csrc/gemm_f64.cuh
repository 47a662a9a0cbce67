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
// A thread's copies lie a fixed number of rows (KC) or, where the tile's width divides
// the threads, of columns apart: one pointer moves on, instead of an address each (with
// 8-byte copies, odd leading dimensions, the addresses were a third of all
// instructions).
template <bool KC, int MN, int V>   // V doubles a copy
__device__ __forceinline__ void fill_tile(double* S, const double* __restrict__ P, int ld, int mn0, int k0, int limit,
                                          int kend) {
  constexpr int kChunks = MN * kBK / V;
  if constexpr (!KC && kThreads % (MN / V) == 0 && kChunks >= kThreads) {
    constexpr int kRow = MN / V, kStep = kThreads / kRow;
    const int mn = (threadIdx.x % kRow) * V, k = threadIdx.x / kRow, left = limit - (mn0 + mn);
    const int n = left < 0 ? 0 : left < V ? left : V;
    const double* src = n ? P + mn0 + mn + (size_t)(k0 + k) * ld : P;
    const size_t step = n ? (size_t)kStep * ld : 0;
    double* dst = S + Tile<KC, MN>::at(mn, k);
    if (k0 + kBK <= kend) {
#pragma unroll
      for (int u = 0; u < kBK / kStep; ++u, src += step) copy_async<8 * V>(dst + Tile<KC, MN>::at(0, u * kStep), src, 8 * n);
    } else {
#pragma unroll
      for (int u = 0; u < kBK / kStep; ++u, src += step) {
        const bool in = k0 + k + u * kStep < kend;
        copy_async<8 * V>(dst + Tile<KC, MN>::at(0, u * kStep), in ? src : P, in ? 8 * n : 0);
      }
    }
    return;
  }
  if (KC && mn0 + MN <= limit) {
    constexpr int kRow = kBK / V, kStep = kThreads / kRow;
    const int k = (threadIdx.x % kRow) * V, mn = threadIdx.x / kRow, left = kend - (k0 + k);
    const int n = left < 0 ? 0 : left < V ? left : V;
    const double* src = n ? P + (size_t)(mn0 + mn) * ld + k0 + k : P;
    const size_t step = n ? (size_t)kStep * ld : 0;
    double* dst = S + Tile<KC, MN>::at(mn, k);
#pragma unroll
    for (int u = 0; u < (MN + kStep - 1) / kStep; ++u, src += step)
      if (MN % kStep == 0 || mn + u * kStep < MN) copy_async<8 * V>(dst + Tile<KC, MN>::at(u * kStep, 0), src, 8 * n);
    return;
  }
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

// Entries (m, n) and (m, n + 1) of the result.
__device__ __forceinline__ void store_pair(const Args& g, int m, int n0, const double (&acc)[2]) {
  if (m >= g.M) return;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int n = n0 + e;
    if (n >= g.N) continue;
    // split-K: each K range stores its own partial (summed in range order
    // by splitk_reduce_kernel, so runs repeat bit for bit)
    double* cp = g.C + (size_t)blockIdx.z * g.split_stride + m + (size_t)n * g.ldc;
    double v = g.alpha * acc[e];
    if (!g.split_stride && g.beta != 0.0) v += g.beta * *cp;
    if (g.row_add) v += g.row_add[n];
    *cp = v;
  }
}

// op(A) (m,k): TA ? A[k + m*lda] : A[m + k*lda]   -> K-contiguous when TA
// op(B) (k,n): TB ? B[n + k*ldb] : B[k + n*ldb]   -> K-contiguous when !TB
template <int NT>
constexpr int kResident = NT <= 8 ? 4 : NT <= 10 ? 3 : 2;   // CTAs of an SM, by registers

template <bool TA, bool TB, int NT, int V>
__global__ void __launch_bounds__(kThreads, kResident<NT>) gemm_f64_dmma(Args g) {
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
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) store_pair(g, bm + wm + i * 8 + gid, bn + j * 8 + tig * 2, acc[i][j]);
}

// The same product on 64 x 64 tiles (warps of 32 x 32) whose loads are staged in
// registers: 8 bytes an instruction whatever the alignment.  Where
// 64 columns are no padding, above all where only 8-byte copies are allowed, it holds the
// pace that the asynchronous copies lose (50001 x 60 x 769, A as it is: 198 us against
// 258).  Sums in the same order.
template <bool KC>
__device__ __forceinline__ void staged_load(double (&r)[8], const double* __restrict__ P, int ld, int mn0, int k0, int limit,
                                            int kend) {
  const int t = threadIdx.x;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = k0 + (KC ? (t & 15) : (t >> 6) + 2 * i), mn = mn0 + (KC ? (t >> 4) + 8 * i : (t & 63));
    r[i] = mn < limit && k < kend ? __ldg(KC ? P + (size_t)mn * ld + k : P + mn + (size_t)k * ld) : 0.0;
  }
}

template <bool KC>
__device__ __forceinline__ void staged_store(double (*S)[kBM + 4], const double (&r)[8]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int i = 0; i < 8; ++i) S[KC ? (t & 15) : (t >> 6) + 2 * i][KC ? (t >> 4) + 8 * i : (t & 63)] = r[i];
}

template <bool TA, bool TB>
__global__ void __launch_bounds__(kThreads) gemm_f64_staged(Args g) {
  __shared__ double As[2][kBK][kBM + 4], Bs[2][kBK][kBM + 4];
  const int bm = blockIdx.x * kBM, bn = blockIdx.y * kBM;
  if (g.upper && bm >= bn + kBM) return;
  const int kbeg = blockIdx.z * g.k_per_split, kend = min(g.K, kbeg + g.k_per_split);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  double ra[8], rb[8];
  if (kbeg < kend) {
    staged_load<TA>(ra, g.A, g.lda, bm, kbeg, g.M, kend);
    staged_load<!TB>(rb, g.B, g.ldb, bn, kbeg, g.N, kend);
    staged_store<TA>(As[0], ra);
    staged_store<!TB>(Bs[0], rb);
  }
  __syncthreads();
  int buf = 0;
  for (int k0 = kbeg; k0 < kend; k0 += kBK, buf ^= 1) {
    const bool more = k0 + kBK < kend;
    if (more) {
      staged_load<TA>(ra, g.A, g.lda, bm, k0 + kBK, g.M, kend);
      staged_load<!TB>(rb, g.B, g.ldb, bn, k0 + kBK, g.N, kend);
    }
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      double a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[buf][kk + tig][wm + i * 8 + gid];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[buf][kk + tig][wn + j * 8 + gid];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
    if (more) {
      staged_store<TA>(As[buf ^ 1], ra);
      staged_store<!TB>(Bs[buf ^ 1], rb);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) store_pair(g, bm + wm + i * 8 + gid, bn + wn + j * 8 + tig * 2, acc[i][j]);
}

// Tile widths, in 8 columns (kStaged: gemm_f64_staged, 64 columns), and the share of
// the tensor pipe's rate, in per cent, that an SM reaches with 1, 2, 3 and 4 CTAs of
// each, by the operands' layouts: A B, A B^T, A^T B, A^T B^T, each with 16-byte and with
// 8-byte copies (a least-squares fit of 18400 timed products, 8 to 1000 columns, 60 to
// 400000 rows and contractions, up to 64 K ranges; half of them within 2.5 per cent).
constexpr int kStaged = 0;
constexpr int kWidths[] = {kStaged, 1, 2, 4, 5, 7, 8, 10, 13};
constexpr unsigned char kRate[8][9][4] = {
    {{47, 74, 84, 80}, {21, 37, 39, 80}, {31, 51, 56, 80}, {44, 78, 76, 80}, {48, 86, 89, 80}, {49, 85, 83, 87}, {56, 81, 81, 87}, {60, 89, 93, 80}, {55, 84, 80, 80}},
    {{47, 73, 84, 80}, {21, 33, 39, 80}, {29, 46, 49, 80}, {45, 71, 70, 73}, {51, 81, 85, 80}, {58, 87, 87, 93}, {53, 74, 73, 76}, {59, 87, 90, 80}, {63, 86, 80, 80}},
    {{57, 84, 85, 91}, {22, 35, 37, 80}, {33, 54, 58, 80}, {44, 81, 79, 82}, {47, 81, 80, 84}, {51, 84, 88, 90}, {57, 88, 86, 90}, {60, 88, 92, 80}, {55, 83, 80, 80}},
    {{57, 84, 85, 91}, {20, 32, 35, 80}, {30, 49, 51, 80}, {43, 77, 76, 77}, {50, 79, 81, 79}, {53, 81, 82, 88}, {56, 87, 83, 86}, {56, 82, 86, 80}, {60, 81, 80, 80}},
    {{43, 66, 74, 80}, {16, 28, 32, 80}, {30, 53, 53, 80}, {41, 71, 83, 80}, {48, 82, 76, 80}, {52, 87, 92, 80}, {52, 83, 91, 80}, {61, 86, 82, 80}, {55, 85, 80, 80}},
    {{43, 66, 74, 80}, {21, 24, 25, 80}, {33, 41, 41, 80}, {47, 80, 83, 80}, {47, 67, 66, 80}, {55, 85, 89, 80}, {58, 85, 88, 80}, {54, 72, 73, 80}, {63, 85, 80, 80}},
    {{52, 74, 78, 86}, {19, 31, 34, 80}, {27, 48, 51, 80}, {40, 70, 83, 80}, {42, 71, 85, 80}, {48, 80, 78, 82}, {59, 89, 83, 85}, {62, 89, 91, 80}, {58, 84, 80, 80}},
    {{52, 74, 78, 86}, {18, 26, 26, 80}, {31, 38, 40, 80}, {45, 80, 79, 80}, {49, 80, 83, 80}, {53, 80, 81, 87}, {54, 75, 73, 75}, {55, 82, 86, 80}, {59, 80, 80, 80}}};

// CTAs of a width that an SM holds (four at most count), by shared memory and registers.
inline int resident_ctas(bool ta, bool tb, int nt) {
  if (nt == kStaged) return tb ? 4 : 3;
  const int stages = nt <= 2 ? 6 : nt <= 5 ? 4 : 3;
  const int a = ta ? kBM * (kBK + 4) : kBK * (kBM + 4), b = tb ? kBK * (8 * nt + 4) : 8 * nt * (kBK + 4);
  const int by_smem = 228 * 1024 / (8 * stages * (a + b) + 1024), by_regs = nt >= 13 ? 2 : nt >= 10 ? 3 : 4;
  return by_smem < by_regs ? by_smem : by_regs;
}

// Launches the tile kernel of (TA, TB) for 8 nt columns a tile (one of kWidths, or kStaged).
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
      case kStaged: gemm_f64_staged<TA, TB><<<grid, kThreads, 0, st>>>(g); break;    \
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
