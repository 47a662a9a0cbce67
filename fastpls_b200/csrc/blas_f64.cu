#include "blas_f64.cuh"

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "context.cuh"
#include "gemm_f64.cuh"
#include "gemv_f64.cuh"

namespace fpls {
namespace {

__global__ void scale_matrix_kernel(double* C, int M, int N, int ldc, double beta) {
  const size_t total = (size_t)M * N;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int m = static_cast<int>(idx % M);
    const int n = static_cast<int>(idx / M);
    double* cp = C + m + (size_t)n * ldc;
    *cp = (beta == 0.0) ? 0.0 : beta * *cp;
  }
}

constexpr int kGemvAhead = 32;

// y[m] = alpha * sum_k A[m + k*lda] x[k] (+ beta y); grid.y splits K into partials.
__global__ void __launch_bounds__(kGemvRows) gemv_n_kernel(int M, int K, double alpha, const double* __restrict__ A, int lda,
                                                           const double* __restrict__ x, double* __restrict__ y,
                                                           int k_per_split, long long split_stride, double beta) {
  __shared__ double xs[256];
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const int kbeg = blockIdx.y * k_per_split;
  const int kend = min(K, kbeg + k_per_split);
  double acc = 0.0;
  for (int kc = kbeg; kc < kend; kc += 256) {
    const int kn = min(256, kend - kc);
    __syncthreads();
    if (threadIdx.x < kn) xs[threadIdx.x] = x[kc + threadIdx.x];
    __syncthreads();
    if (m < M) acc = gemv_row<kGemvAhead>(A + m + (size_t)kc * lda, lda, xs, kn, acc);
  }
  if (m < M) {
    if (split_stride) y[(size_t)blockIdx.y * split_stride + m] = alpha * acc;
    else y[m] = (beta == 0.0) ? alpha * acc : alpha * acc + beta * y[m];
  }
}

// C (M x N, ldc) = beta C + sum_{z < splits} W_z, W_z = W + z stride (ld ldw):
// the split-K partials added in K-range order.
__global__ void splitk_reduce_kernel(const double* __restrict__ W, int splits, long long stride, int M, int N,
                                     int ldw, double beta, double* __restrict__ C, int ldc,
                                     const double* __restrict__ row_add) {
  const size_t total = (size_t)M * N;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const int m = static_cast<int>(t % M), n = static_cast<int>(t / M);
    double acc = 0.0;
    for (int z = 0; z < splits; ++z) acc += W[(size_t)z * stride + m + (size_t)n * ldw];
    double* cp = C + m + (size_t)n * ldc;
    double v = (beta == 0.0) ? acc : acc + beta * *cp;
    if (row_add) v += row_add[n];
    *cp = v;
  }
}

// y[n] = alpha * sum_k A[k + n*lda] x[k] + beta y[n]; one warp per column and
// range of kps rows (blockIdx.y; its result at y + range * stride).
__global__ void __launch_bounds__(128) gemv_t_kernel(int K, int N, double alpha, const double* __restrict__ A, int lda,
                                                     const double* __restrict__ x, double beta, double* __restrict__ y,
                                                     int kps, long long stride) {
  const int n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (n >= N) return;
  const int k0 = blockIdx.y * kps;
  const int rows = min(kps, K - k0);
  const double* col = A + (size_t)n * lda + k0;
  const double acc = rows <= 32 * 2   ? gemv_column<2>(col, x + k0, rows)
                     : rows <= 32 * 8 ? gemv_column<8>(col, x + k0, rows)
                                      : gemv_column<kGemvAhead>(col, x + k0, rows);
  y += blockIdx.y * stride;
  if ((threadIdx.x & 31) == 0) y[n] = (beta == 0.0) ? alpha * acc : alpha * acc + beta * y[n];
}

// Per-column sums over rows: one warp a column, lane l adds the rows l, l + 32, ...
// in order, then a shuffle tree (so results do not depend on how far the loads
// run ahead).  48 loads go out before they are added: a column is one chain of
// loads, and 768 of them one at a time left 50000 rows at 2.1 TB/s (143 us; 100
// columns 142 us, the latency of 1563 loads in a row; 16 ahead: 110 us).
constexpr int kColWarps = 4;   // 768 columns fill the SMs in blocks of four
constexpr int kColAhead = 48;

template <int AHEAD, typename T, typename F>
__device__ __forceinline__ double lane_sum_ahead(const T* __restrict__ x, int n, F term) {
  double s = 0.0;
  int i = threadIdx.x & 31;
  for (; i < n; i += 32 * AHEAD) {
    T v[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (i + 32 * u < n) v[u] = __ldg(x + i + 32 * u);
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (i + 32 * u < n) s += term(static_cast<double>(v[u]));
  }
  return warp_sum(s);
}

// A short column would pass 48 bounds for its one to eight loads.
template <typename T, typename F>
__device__ __forceinline__ double lane_column_sum(const T* __restrict__ x, int n, F term) {
  return n <= 32 * 8 ? lane_sum_ahead<8>(x, n, term) : lane_sum_ahead<kColAhead>(x, n, term);
}

__device__ __forceinline__ int warp_column() { return blockIdx.x * kColWarps + (threadIdx.x >> 5); }

// FP64 column means; single-precision input is summed in FP64 in the same
// order, so its means equal those of the widened FP64 copy bit for bit.
template <typename T>
__global__ void __launch_bounds__(32 * kColWarps) col_mean_kernel(const T* __restrict__ X, int n, int p, int ldx,
                                                                  double* __restrict__ out) {
  const int j = warp_column();
  if (j >= p) return;
  const double s = lane_column_sum(X + (size_t)j * ldx, n, [](double v) { return v; });
  if ((threadIdx.x & 31) == 0) out[j] = s / static_cast<double>(n);
}

__global__ void __launch_bounds__(32 * kColWarps) col_sd_kernel(const double* __restrict__ X, int n, int p, int ldx,
                                                                double* __restrict__ out) {
  const int j = warp_column();
  if (j >= p) return;
  const double* xp = X + (size_t)j * ldx;
  // Two-pass (mean of the centred column, then squares) matches Welford to rounding.
  const double mu = lane_column_sum(xp, n, [](double v) { return v; }) / static_cast<double>(n);
  const double q = lane_column_sum(xp, n, [mu](double v) { const double d = v - mu; return d * d; });
  if ((threadIdx.x & 31) == 0) out[j] = sqrt(q / static_cast<double>(n - 1));
}

// Column sums (the loop and warp reduction of col_mean_kernel, without the
// division): the partial sums of a row-sharded fit.
__global__ void __launch_bounds__(32 * kColWarps) col_sum_kernel(const double* __restrict__ X, int n, int p, int ldx,
                                                                 double* __restrict__ out) {
  const int j = warp_column();
  if (j >= p) return;
  const double s = lane_column_sum(X + (size_t)j * ldx, n, [](double v) { return v; });
  if ((threadIdx.x & 31) == 0) out[j] = s;
}

// Sums of squared deviations from mu (the second pass of col_sd_kernel).
__global__ void __launch_bounds__(32 * kColWarps) col_sqdev_kernel(const double* __restrict__ X, int n, int p, int ldx,
                                                                   const double* __restrict__ mu,
                                                                   double* __restrict__ out) {
  const int j = warp_column();
  if (j >= p) return;
  const double m = mu[j];
  const double q = lane_column_sum(X + (size_t)j * ldx, n, [m](double v) { const double d = v - m; return d * d; });
  if ((threadIdx.x & 31) == 0) out[j] = q;
}

// out = in / d, or sqrt(in / d) when root is set.
__global__ void div_vec_kernel(const double* __restrict__ in, size_t count, double d, int root,
                               double* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
    out[i] = root ? sqrt(in[i] / d) : in[i] / d;
}

// dst[:, j] = (src[:, j] - mean[j]) / scale[j] (mean or scale may be null), both
// n x p with ld n, src FP32 or FP64 and possibly dst itself.  A thread takes eight
// rows (RowTiles) of a column, its loads in flight together, no index divisions:
// 20000 x 5000 from FP32 in one pass instead of a copy, a widening and a centring one.
template <typename T, int LOG>   // LOG: the tiles' log_rows, or -1
__global__ void __launch_bounds__(256) center_scale_kernel(const T* src, double* dst, int n, int p, RowTiles tiles,
                                                           const double* __restrict__ mean,
                                                           const double* __restrict__ scale) {
  const int log_rows = LOG < 0 ? tiles.log_rows : LOG, tx = 1 << log_rows, cols = 256 >> log_rows;
  const int i0 = blockIdx.x * 8 * tx + (threadIdx.x & (tx - 1));
  for (int j = blockIdx.y * cols + (threadIdx.x >> log_rows); j < p; j += gridDim.y * cols) {
    const T* x = src + (size_t)j * n;
    double* y = dst + (size_t)j * n;
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i0 + tx * u < n) v[u] = x[i0 + tx * u];
    const double m = mean ? mean[j] : 0.0, sc = scale ? scale[j] : 1.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (i0 + tx * u < n) {
        double w = static_cast<double>(v[u]);
        if (mean) w -= m;
        if (scale) w /= sc;
        y[i0 + tx * u] = w;
      }
    }
  }
}

__global__ void copy_matrix_kernel(double* dst, int ldd, const double* src, int lds, int n, int p) {
  const size_t total = (size_t)n * p;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int i = static_cast<int>(idx % n);
    const int j = static_cast<int>(idx / n);
    dst[i + (size_t)j * ldd] = src[i + (size_t)j * lds];
  }
}

__global__ void add_row_vector_kernel(double* X, int n, int p, int ldx, const double* v) {
  const size_t total = (size_t)n * p;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int i = static_cast<int>(idx % n);
    const int j = static_cast<int>(idx / n);
    X[i + (size_t)j * ldx] += v[j];
  }
}

// Column sums of Y in the order rq_sums_kernel takes them (one block).
__global__ void rq_col_sums_kernel(const double* __restrict__ Y, int n, int m, double* __restrict__ out) {
  __shared__ double scratch[32];
  for (int j = 0; j < m; ++j) {
    const double* yc = Y + (size_t)j * n;
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += yc[i];
    s = block_sum(s, scratch);
    if (threadIdx.x == 0) out[j] = s;
  }
}

// PRESS and TSS of Y against Yp; the TSS about the column means of these rows,
// or about mus (the means over all ranks' rows of a row-sharded fit).
__global__ void rq_sums_kernel(const double* __restrict__ Y, const double* __restrict__ Yp,
                               int n, int m, double* out2, const double* __restrict__ mus) {
  __shared__ double scratch[32];
  double press = 0.0, tss = 0.0;
  for (int j = 0; j < m; ++j) {
    const double* yc = Y + (size_t)j * n;
    double mu;
    if (mus) {
      mu = mus[j];
    } else {
      double s = 0.0;
      for (int i = threadIdx.x; i < n; i += blockDim.x) s += yc[i];
      s = block_sum(s, scratch);
      mu = s / static_cast<double>(n);
    }
    const double* pc = Yp + (size_t)j * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double d = yc[i] - pc[i];
      const double e = yc[i] - mu;
      press += d * d;
      tss += e * e;
    }
  }
  press = block_sum(press, scratch);
  tss = block_sum(tss, scratch);
  if (threadIdx.x == 0) {
    out2[0] = press;
    out2[1] = tss;
  }
}

__global__ void fill_kernel(double* x, size_t n, double v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    x[i] = v;
}

__global__ void scale_vec_kernel(double* x, size_t n, double a) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    x[i] *= a;
}

int grid_for(size_t total, int threads) {
  size_t g = (total + threads - 1) / threads;
  const size_t cap = (size_t)kSMCount * 16;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return static_cast<int>(g);
}

}  // namespace

namespace {

using gemm64::kBK;
using gemm64::kBM;

// K ranges of a product of `tiles` 64 x 64 output tiles: enough for two tiles an
// SM, at least 128 terms each.  The ranges set the order of the sum, so this rule
// does not look at the tile width.
int split_count(int tiles, int K, int sm_count) {
  const int target = 2 * sm_count;
  if (tiles >= target || K < 4 * kBK) return 1;
  return std::max(1, std::min(ceil_div(target, tiles), ceil_div(K, 8 * kBK)));
}

struct GemmPlan { int nt, splits, kps; };

// 16-byte copies need both operands' columns on 16-byte boundaries
bool wide_copies(const double* A, int lda, const double* B, int ldb) {
  auto aligned = [](const double* p, int ld) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 2 == 0; };
  return aligned(A, lda) && aligned(B, ldb);
}

// Tile width and K ranges by modelled time: the time of the SM with the most tiles.  A
// tile takes 8 nt cycles of the FP64 tensor pipe a contraction step; the tiles' operands
// come from L2 at some 3000 bytes a clock (all SMs); partials are written, read and summed
// once more.  Two estimates.  The plain one lets the pipe run at 95 per cent under
// several CTAs and at 85 under one; the other takes the rates that CTAs of each width
// and layout were measured to reach together (gemm64::kRate; one alone reaches half), in
// rounds of the CTAs that an SM holds.  The plain choice stands unless the measured
// rates put another one 7 per cent ahead: what they cannot tell apart, they rank by
// their own error (208 products: 6 per cent faster on average than the plain choice, 4
// of them more than 3 per cent slower; by the rates alone, 29).
// Products below 2^28 multiply-adds keep the ranges of split_count (only their width is
// chosen): they are over in tens of microseconds, and iterations that feed the split
// precisions need their last bits unchanged.  50000 x 768 x 100 (S = X^T Y): 551 us
// on 64 x 64 tiles in 13 ranges (312 tiles on 148 SMs), 361 us now; 20001 x 100 over
// 1001, A transposed: 238 us on those tiles, 288 by the plain choice, 179 now.
GemmPlan plan_gemm(bool ta, bool tb, bool wide, int M, int N, int K, int sm_count) {
  const bool large = static_cast<double>(M) * N * K >= 268435456.0;
  const int base = split_count(ceil_div(M, kBM) * ceil_div(N, 64), K, sm_count);
  const int smax = large ? std::max(1, std::min(64, K / (8 * kBK))) : base;
  GemmPlan plain{8, base, 0}, best{8, base, 0};
  double plain_cost = 1e300, plain_measured = 0.0, best_measured = 1e300;
  for (int i = 0; i < 9; ++i) {
    const int nt = gemm64::kWidths[i], columns = nt == gemm64::kStaged ? 64 : 8 * nt;
    if (ceil_div(N, columns) > 65535) continue;
    const unsigned char* rate = gemm64::kRate[4 * ta + 2 * tb + !wide][i];
    const double tiles = static_cast<double>(ceil_div(M, kBM)) * ceil_div(N, columns);
    const int resident = gemm64::resident_ctas(ta, tb, nt);
    for (int want = large ? 1 : base; want <= smax; ++want) {
      const GemmPlan plan{nt, 0, ceil_div(ceil_div(K, want), kBK) * kBK};
      const int splits = ceil_div(K, plan.kps);
      const double units = tiles * splits, waves = std::ceil(units / sm_count), work = static_cast<double>(plan.kps) * columns;
      const double bytes = units * plan.kps * (kBM + columns) * 8.0, sums = (2.0 * splits + 1.0) * M * N * 8.0;
      const int together = static_cast<int>(std::min<double>(waves, resident));
      const double rounds = std::floor(waves / together);
      const int rest = static_cast<int>(waves - rounds * together);
      // 400 cycles a tile before its first products (the staged kernel has none to fill)
      double measured = 100.0 * work * (rounds * together / rate[together - 1] + (rest ? static_cast<double>(rest) / rate[rest - 1] : 0.0));
      measured = std::max(measured + (nt == gemm64::kStaged ? 0.0 : 400.0 * waves), bytes / 3800.0);
      if (splits > 1) measured += 4500.0 + sums / 3600.0;
      if (measured < best_measured) {
        best_measured = measured;
        best = GemmPlan{nt, splits, plan.kps};
      }
      if (nt == gemm64::kStaged) continue;
      const double alone = work / 0.85 + 4000.0, held = std::min(waves, nt >= 13 ? 2.0 : nt >= 8 ? 3.0 : 4.0);
      double cost = std::max(waves * std::max(work / 0.95, alone / held), bytes / 2900.0);
      if (splits > 1) cost += 3000.0 + sums / 2900.0;
      if (cost < plain_cost) {
        plain_cost = cost;
        plain_measured = measured;
        plain = GemmPlan{nt, splits, plan.kps};
      }
    }
  }
  return best_measured < 0.93 * plain_measured ? best : plain;
}

void gemm_run(bool transA, bool transB, int nt, const gemm64::Args& g, int splits, cudaStream_t st) {
  const dim3 grid(ceil_div(g.M, kBM), ceil_div(g.N, nt == gemm64::kStaged ? 64 : 8 * nt), splits);
  const bool vec = wide_copies(g.A, g.lda, g.B, g.ldb);
  if (!transA && !transB) gemm64::launch<false, false>(g, nt, vec, grid, st);
  else if (transA && !transB) gemm64::launch<true, false>(g, nt, vec, grid, st);
  else if (!transA) gemm64::launch<false, true>(g, nt, vec, grid, st);
  else gemm64::launch<true, true>(g, nt, vec, grid, st);
}

}  // namespace

namespace {

// The tiles of a product: into C (beta, row_add applied) or, with several K
// ranges, into partials that the caller adds.
Partials gemm_tiles(bool transA, bool transB, int M, int N, int K, double alpha, const double* A, int lda,
                    const double* B, int ldb, double beta, double* C, int ldc, const double* row_add) {
  Context& ctx = Context::get();
  cudaStream_t st = ctx.stream;
  const GemmPlan plan = plan_gemm(transA, transB, wide_copies(A, lda, B, ldb), M, N, K, ctx.sm_count);
  gemm64::Args g{M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, plan.kps, 0, 0, row_add};
  if (plan.splits > 1) {
    g.split_stride = (long long)M * N;
    g.C = ctx.splitk_workspace(st, (size_t)plan.splits * M * N);
    g.ldc = M;
    g.beta = 0.0;
    g.row_add = nullptr;
  }
  const int slot = ctx.prof_begin("gemm_f64_dmma", st);
  gemm_run(transA, transB, plan.nt, g, plan.splits, st);
  // algorithmic work: 2MNK flops; each operand and the result once
  ctx.prof_end(slot, st, 8.0 * ((double)M * K + (double)K * N + (double)M * N), 2.0 * (double)M * N * K);
  return Partials{g.C, plan.splits, (size_t)M * N};
}

}  // namespace

Partials gemm_partials(bool transA, bool transB, int M, int N, int K, const double* A, int lda, const double* B,
                       int ldb, double* C) {
  if (M <= 0 || N <= 0 || K <= 0) {
    gemm(transA, transB, M, N, K, 1.0, A, lda, B, ldb, 0.0, C, M);
    return Partials{C, 1, 0};
  }
  return gemm_tiles(transA, transB, M, N, K, 1.0, A, lda, B, ldb, 0.0, C, M, nullptr);
}

void gemm(bool transA, bool transB, int M, int N, int K, double alpha, const double* A, int lda,
          const double* B, int ldb, double beta, double* C, int ldc, const double* row_add) {
  if (M <= 0 || N <= 0) return;
  cudaStream_t st = Context::get().stream;
  if (K <= 0) {
    scale_matrix_kernel<<<grid_for((size_t)M * N, 256), 256, 0, st>>>(C, M, N, ldc, beta); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    if (row_add) add_row_vector(C, M, N, ldc, row_add);
    return;
  }
  const Partials p = gemm_tiles(transA, transB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, row_add);
  // split-K partials are summed in order
  if (p.splits > 1) {
    splitk_reduce_kernel<<<grid_for((size_t)M * N, 256), 256, 0, st>>>(p.w, p.splits, p.stride, M, N, M, beta, C, ldc,
                                                                      row_add);
    ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
  }
}

__global__ void mirror_upper_f64_kernel(double* K, int n, int ldk) {
  const size_t total = (size_t)n * n;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const int i = static_cast<int>(t % n), j = static_cast<int>(t / n);
    if (i > j) K[i + (size_t)j * ldk] = K[j + (size_t)i * ldk];
  }
}

namespace {
// Upper tiles of op(X) op(X)^T (n x n) with n = rows of op(X) and p its
// columns, split-K partials summed in range order, then the lower triangle
// mirrored.  TX: X is stored p x n (op(X) = X^T).
template <bool TX>
void gram_tiles_f64(const double* X, int n, int p, int ldx, double* K, int ldk) {
  if (n <= 0) return;
  Context& ctx = Context::get();
  cudaStream_t st = ctx.stream;
  const int g = ceil_div(n, kBM);
  int splits = split_count(g * (g + 1) / 2, p, ctx.sm_count);
  const int kps = ceil_div(ceil_div(p, splits), kBK) * kBK;
  splits = ceil_div(p, kps);
  if (p <= 0) {
    scale_matrix_kernel<<<grid_for((size_t)n * n, 256), 256, 0, st>>>(K, n, n, ldk, 0.0); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
  }
  if (p > 0) {
    gemm64::Args a{n, n, p, 1.0, X, ldx, X, ldx, 0.0, K, ldk, kps, 0, 1, nullptr};
    if (splits > 1) {  // partials of the K ranges, summed in order (lower tiles stay unused)
      a.split_stride = (long long)n * n;
      a.C = ctx.splitk_workspace(st, (size_t)splits * n * n);
      a.ldc = n;
    }
    const int slot = ctx.prof_begin("gemm_f64_dmma", st);
    gemm_run(TX, !TX, 8, a, splits, st);   // square tiles, as the diagonal cuts them
    // algorithmic work: the upper tiles' share of 2 n^2 p flops
    ctx.prof_end(slot, st, 8.0 * ((double)n * p + (double)n * n), (double)n * (n + kBM) * p);
    if (splits > 1) {
      splitk_reduce_kernel<<<grid_for((size_t)n * n, 256), 256, 0, st>>>(a.C, splits, a.split_stride, n, n, n, 0.0, K,
                                                                        ldk, nullptr);
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
    }
  }
  mirror_upper_f64_kernel<<<grid_for((size_t)n * n, 256), 256, 0, st>>>(K, n, ldk); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}
}  // namespace

void gram_f64(const double* X, int n, int p, int ldx, double* K, int ldk) {
  gram_tiles_f64<false>(X, n, p, ldx, K, ldk);
}

namespace {
// B (cols x rows, ld ldb) = A^T for A (rows x cols, ld lda), column-major both,
// through 32 x 32 shared-memory tiles (column reads and column writes).
__global__ void __launch_bounds__(256) transpose_f64_kernel(const double* __restrict__ A, int rows, int cols,
                                                            int lda, double* __restrict__ B, int ldb) {
  __shared__ double t[32][33];
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const int x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
  for (int y = y0; y < 32; y += 8) {
    const int r = r0 + x, c = c0 + y;
    if (r < rows && c < cols) t[y][x] = A[r + static_cast<size_t>(c) * lda];
  }
  __syncthreads();
  for (int y = y0; y < 32; y += 8) {
    const int c = c0 + x, r = r0 + y;   // B(c, r) = A(r, c)
    if (r < rows && c < cols) B[c + static_cast<size_t>(r) * ldb] = t[x][y];
  }
}
}  // namespace

// G = S^T S through a transposed copy of S (q x p), so that the Gram's DMMA
// tiles read both operands in the layout of the row Gram X X^T (A along M,
// B along N) instead of reading S^T in place, for one extra pass over S.
void gram_t_f64(const double* S, int p, int q, int lds, double* G, int ldg) {
  if (q <= 0) return;
  if (p <= 0) {
    gram_tiles_f64<true>(S, q, p, lds, G, ldg);
    return;
  }
  Context& ctx = Context::get();
  double* St = ctx.arena.alloc_n<double>(static_cast<size_t>(q) * p);
  transpose_f64_kernel<<<dim3(ceil_div(p, 32), ceil_div(q, 32)), 256, 0, ctx.stream>>>(S, p, q, lds, St, q);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  gram_tiles_f64<false>(St, q, p, q, G, ldg);
}

Partials gemv_partials(int rows, int cols, const double* A, int lda, const double* x, double* y) {
  Context& ctx = Context::get();
  const GemvRanges gr = gemv_ranges(rows, std::max(cols, 1), ctx.sm_count);
  if (rows <= 0 || cols <= 0 || gr.splits == 1) {
    gemv(false, rows, cols, 1.0, A, lda, x, 0.0, y);
    return Partials{y, 1, 0};
  }
  cudaStream_t st = ctx.stream;
  const int slot = ctx.prof_begin("gemv_f64", st);
  double* ws = ctx.splitk_workspace(st, (size_t)gr.splits * rows);
  gemv_n_kernel<<<dim3(gr.row_blocks, gr.splits), kGemvRows, 0, st>>>(rows, cols, 1.0, A, lda, x, ws, gr.kps,
                                                                      (long long)rows, 0.0);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  ctx.prof_end(slot, st, 8.0 * ((double)rows * cols + rows + cols), 2.0 * (double)rows * cols);
  return Partials{ws, gr.splits, (size_t)rows};
}

Partials gemv_t_partials(int rows, int cols, const double* A, int lda, const double* x, double* y) {
  Context& ctx = Context::get();
  const GemvRanges gr = gemv_t_ranges(rows, std::max(cols, 1), ctx.sm_count);
  if (rows <= 0 || cols <= 0 || gr.splits == 1) {
    gemv(true, rows, cols, 1.0, A, lda, x, 0.0, y);
    return Partials{y, 1, 0};
  }
  cudaStream_t st = ctx.stream;
  const int slot = ctx.prof_begin("gemv_f64", st);
  double* ws = ctx.splitk_workspace(st, (size_t)gr.splits * cols);
  gemv_t_kernel<<<dim3(ceil_div(cols, 4), gr.splits), 128, 0, st>>>(rows, cols, 1.0, A, lda, x, 0.0, ws, gr.kps,
                                                                    (long long)cols);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  ctx.prof_end(slot, st, 8.0 * ((double)rows * cols + rows + cols), 2.0 * (double)rows * cols);
  return Partials{ws, gr.splits, (size_t)cols};
}

void gemv_t_ranged(int rows, int cols, const double* A, int lda, const double* x, double* y) {
  const Partials p = gemv_t_partials(rows, cols, A, lda, x, y);
  if (p.splits == 1) return;
  splitk_reduce_kernel<<<grid_for(cols, 256), 256, 0, Context::get().stream>>>(p.w, p.splits, (long long)p.stride, cols, 1,
                                                                              cols, 0.0, y, cols, nullptr);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void gemv(bool trans, int rows, int cols, double alpha, const double* A, int lda, const double* x,
          double beta, double* y) {
  Context& ctx = Context::get();
  cudaStream_t st = ctx.stream;
  const int slot = rows > 0 && cols > 0 ? ctx.prof_begin("gemv_f64", st) : -1;
  if (!trans) {
    if (rows <= 0) return;
    if (cols <= 0) {
      scale_matrix_kernel<<<grid_for(rows, 256), 256, 0, st>>>(y, rows, 1, rows, beta); ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      return;
    }
    const GemvRanges gr = gemv_ranges(rows, cols, ctx.sm_count);
    const int gx = gr.row_blocks, splits = gr.splits, kps = gr.kps;
    if (splits > 1) {
      // partials of the column ranges, summed in order (runs repeat bit for bit)
      double* ws = ctx.splitk_workspace(st, (size_t)splits * rows);
      gemv_n_kernel<<<dim3(gx, splits), 256, 0, st>>>(rows, cols, alpha, A, lda, x, ws, kps, (long long)rows, 0.0);
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      splitk_reduce_kernel<<<grid_for(rows, 256), 256, 0, st>>>(ws, splits, rows, rows, 1, rows, beta, y, rows,
                                                               nullptr);
    } else {
      gemv_n_kernel<<<dim3(gx, splits), 256, 0, st>>>(rows, cols, alpha, A, lda, x, y, kps, 0ll, beta);
    }
    ::fpls::note_launch();
  } else {
    if (cols <= 0) return;
    gemv_t_kernel<<<ceil_div(cols, 4), 128, 0, st>>>(rows, cols, alpha, A, lda, x, beta, y, rows, 0ll);
    ::fpls::note_launch();
  }
  FPLS_CHECK_LAUNCH();
  // algorithmic bytes: the matrix once plus both vectors
  ctx.prof_end(slot, st, 8.0 * ((double)rows * cols + rows + cols), 2.0 * (double)rows * cols);
}

void col_mean(const double* X, int n, int p, int ldx, double* out) {
  if (p <= 0) return;
  col_mean_kernel<double><<<ceil_div(p, kColWarps), 32 * kColWarps, 0, Context::get().stream>>>(X, n, p, ldx, out); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void col_mean(const float* X, int n, int p, int ldx, double* out) {
  if (p <= 0) return;
  col_mean_kernel<float><<<ceil_div(p, kColWarps), 32 * kColWarps, 0, Context::get().stream>>>(X, n, p, ldx, out); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void col_sd_centered(const double* X, int n, int p, int ldx, double* out) {
  if (p <= 0) return;
  col_sd_kernel<<<ceil_div(p, kColWarps), 32 * kColWarps, 0, Context::get().stream>>>(X, n, p, ldx, out); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void col_sum(const double* X, int n, int p, int ldx, double* out) {
  if (p <= 0) return;
  col_sum_kernel<<<ceil_div(p, kColWarps), 32 * kColWarps, 0, Context::get().stream>>>(X, n, p, ldx, out); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void col_sqdev(const double* X, int n, int p, int ldx, const double* mu, double* out) {
  if (p <= 0) return;
  col_sqdev_kernel<<<ceil_div(p, kColWarps), 32 * kColWarps, 0, Context::get().stream>>>(X, n, p, ldx, mu, out); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void div_vec(const double* in, size_t count, double d, bool root, double* out) {
  if (count == 0) return;
  div_vec_kernel<<<grid_for(count, 256), 256, 0, Context::get().stream>>>(in, count, d, root ? 1 : 0, out); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

namespace {
template <typename T>
void center_scale_run(const T* src, double* dst, int n, int p, const double* mean, const double* scale) {
  if ((size_t)n * p == 0) return;
  const RowTiles t(n);
  auto kernel = t.log_rows == 8 ? center_scale_kernel<T, 8> : center_scale_kernel<T, -1>;
  kernel<<<t.grid(n, p), 256, 0, Context::get().stream>>>(src, dst, n, p, t, mean, scale); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}
}  // namespace

void center_scale(const double* src, double* dst, int n, int p, const double* mean, const double* scale) {
  center_scale_run(src, dst, n, p, mean, scale);
}

void center_scale(const float* src, double* dst, int n, int p, const double* mean, const double* scale) {
  center_scale_run(src, dst, n, p, mean, scale);
}

void copy_matrix(double* dst, int ldd, const double* src, int lds, int n, int p) {
  if ((size_t)n * p == 0) return;
  copy_matrix_kernel<<<grid_for((size_t)n * p, 256), 256, 0, Context::get().stream>>>(dst, ldd, src, lds, n, p); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void add_row_vector(double* X, int n, int p, int ldx, const double* v) {
  if ((size_t)n * p == 0) return;
  add_row_vector_kernel<<<grid_for((size_t)n * p, 256), 256, 0, Context::get().stream>>>(X, n, p, ldx, v); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void rq_sums(const double* Y, const double* Yp, int n, int m, double* out2, const double* mus) {
  rq_sums_kernel<<<1, 512, 0, Context::get().stream>>>(Y, Yp, n, m, out2, mus); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

const double* shard_rq_means(const double* Y, int n, int m) {
  if (!sharded()) return nullptr;
  Context& ctx = Context::get();
  double* mu = ctx.arena.alloc_n<double>(m);
  rq_col_sums_kernel<<<1, 512, 0, ctx.stream>>>(Y, n, m, mu); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  shard_sum(mu, m);
  div_vec(mu, m, static_cast<double>(shard_rows(n)), false, mu);
  return mu;
}

void fill(double* x, size_t n, double v) {
  if (n == 0) return;
  fill_kernel<<<grid_for(n, 256), 256, 0, Context::get().stream>>>(x, n, v); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void scale_vec(double* x, size_t n, double a) {
  if (n == 0) return;
  scale_vec_kernel<<<grid_for(n, 256), 256, 0, Context::get().stream>>>(x, n, a); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

}  // namespace fpls
