// FP64 dense kernels on B200: DMMA (mma.sync m8n8k4 f64) tiled GEMM and
// bandwidth-bound GEMV / column statistics.  All matrices are column-major
// (R / Armadillo layout); pointers are device pointers; work is issued on the
// context stream.  tcgen05 has no f64 kind, so FP64 contractions run on the
// FP64 tensor path (DMMA) or on DFMA.
#pragma once

#include "common.cuh"

namespace fpls {

// Blocks of 256 threads over an n x p column-major matrix, eight rows a thread:
// 2048 rows of a column a block, several columns where n is smaller (a column a
// block is 20000 blocks for a prediction of one row of 20000 predictors: 22 us a
// pass instead of 3).
struct RowTiles {
  int log_rows = 0;   // 2^log_rows threads take a column
  explicit RowTiles(int n) {
    while (log_rows < 8 && (1 << log_rows) < (n < 32 ? n : n < 256 ? 32 : (n + 7) / 8)) ++log_rows;
  }
  dim3 grid(int n, int p) const {
    const int blocks = ceil_div(p, 256 >> log_rows);
    return dim3(ceil_div(n, 8 << log_rows), blocks < 65535 ? blocks : 65535);
  }
};

// C = alpha * op(A) * op(B) + beta * C, op(A): M x K, op(B): K x N; row_add
// (N values, or null) is then added to every row.
void gemm(bool transA, bool transB, int M, int N, int K, double alpha,
          const double* A, int lda, const double* B, int ldb, double beta,
          double* C, int ldc, const double* row_add = nullptr);

// A product left as partial sums: entry t is w[t] + w[t + stride] + ... (splits
// terms, in that order; one: the product itself).  Valid until the next product
// on the same stream.
struct Partials {
  const double* w;
  int splits;
  size_t stride;
};
// gemm (alpha 1, beta 0, ldc = M) whose K ranges the reader adds up.
Partials gemm_partials(bool transA, bool transB, int M, int N, int K, const double* A, int lda, const double* B,
                       int ldb, double* C);
// gemv (no transpose, alpha 1, beta 0) whose column ranges the reader adds up.
Partials gemv_partials(int rows, int cols, const double* A, int lda, const double* x, double* y);
// y = A^T x by gemv_t_ranges' row ranges, which the reader adds up (gemv_t_ranged: added here).
Partials gemv_t_partials(int rows, int cols, const double* A, int lda, const double* x, double* y);
void gemv_t_ranged(int rows, int cols, const double* A, int lda, const double* x, double* y);

// K (n x n) = X X^T for X n x p: the upper-triangle tiles by FP64 tensor-core
// MMA, the lower triangle mirrored (K exactly symmetric).
void gram_f64(const double* X, int n, int p, int ldx, double* K, int ldk);

// G (q x q) = S^T S for S p x q (lds): the same upper-tile product, mirrored.
void gram_t_f64(const double* S, int p, int q, int lds, double* G, int ldg);

// y = alpha * op(A) * x + beta * y.  A is rows x cols (lda).
void gemv(bool trans, int rows, int cols, double alpha, const double* A, int lda,
          const double* x, double beta, double* y);

// Column means of X (n x p).  out[p].
void col_mean(const double* X, int n, int p, int ldx, double* out);
void col_mean(const float* X, int n, int p, int ldx, double* out);
// Column standard deviation (n-1) of an already centred X.
void col_sd_centered(const double* X, int n, int p, int ldx, double* out);
// Column sums; sums of squared deviations from mu; out = in / d (sqrt(in / d)
// with root).  The pieces of col_mean / col_sd_centered for row-sharded fits.
void col_sum(const double* X, int n, int p, int ldx, double* out);
void col_sqdev(const double* X, int n, int p, int ldx, const double* mu, double* out);
void div_vec(const double* in, size_t count, double d, bool root, double* out);
// dst[:, j] = (src[:, j] - mean[j]) / scale[j] (mean or scale may be null); n x p,
// ld n, dst may be src.
void center_scale(const double* src, double* dst, int n, int p, const double* mean, const double* scale);
void center_scale(const float* src, double* dst, int n, int p, const double* mean, const double* scale);
// dst (n x p, ldd) = src (n x p, lds)
void copy_matrix(double* dst, int ldd, const double* src, int lds, int n, int p);
// X[i, j] += v[j] for all i (row broadcast)
void add_row_vector(double* X, int n, int p, int ldx, const double* v);
// Frobenius-type sums for R2: out[0] = sum((Y - Yp)^2), out[1] = sum((Y - colmean(Y))^2)
void rq_sums(const double* Y, const double* Yp, int n, int m, double* out2, const double* mus = nullptr);
// Row-sharded fits: the column means of Y over all ranks' rows, the TSS
// centre of rq_sums (null when the fit is not sharded).
const double* shard_rq_means(const double* Y, int n, int m);
void fill(double* x, size_t n, double v);
void scale_vec(double* x, size_t n, double a);

}  // namespace fpls
