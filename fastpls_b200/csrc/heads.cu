#include "xop_split.cuh"
#include "blas_f64.cuh"
#include "context.cuh"
#include "heads.cuh"
#include "linalg_small.cuh"
#include "row_topk.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

namespace fpls {
namespace {

// A thread a row: the loads of a warp are coalesced, those of the SM's other warps
// hide their latency, and one maximum is little to carry.  Bound by reading S
// (1,000,000 x 12: 15 us).
__global__ void __launch_bounds__(256) argmax_kernel(const double* __restrict__ S, int w, int C,
                                                     const double* __restrict__ bias, int* __restrict__ labels) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= w) return;
  int best = 0;
  double bv = S[i] + (bias ? bias[0] : 0.0);
  for (int c = 1; c < C; ++c) {
    const double v = S[i + (size_t)c * w] + (bias ? bias[c] : 0.0);
    if (v > bv) {
      bv = v;
      best = c;
    }
  }
  labels[i] = best + 1;
}

// Class sums of the score columns (T n x kmax into sums C x kmax) in a fixed
// order: warp w takes (class c, column j) = (w % C, w / C) and walks that
// class's rows in class-sorted order perm[off[c] .. off[c+1]) lane-strided,
// then a fixed shuffle tree -- the same rounding on every run (no atomics).
__global__ void class_sums_sorted_kernel(const double* __restrict__ T, int n, int kmax,
                                         const int* __restrict__ perm, const int* __restrict__ off, int C,
                                         double* __restrict__ sums) {
  const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (long long)C * kmax) return;  // whole warps leave together
  const int c = static_cast<int>(w % C), j = static_cast<int>(w / C);
  const double* tc = T + (size_t)j * n;
  double acc = 0.0;
  for (int i = off[c] + lane; i < off[c + 1]; i += 32) acc += tc[perm[i]];
  acc = warp_sum(acc);
  if (lane == 0) sums[c + (size_t)j * C] = acc;
}

__global__ void means_from_sums_kernel(double* M, int C, int k, const double* counts,
                                       double* Mw) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= C * k) return;
  const int c = t % C;
  const double m = M[t] / counts[c];
  M[t] = m;
  Mw[t] = m * counts[c];
}

// pooled = symmatu(P) / df   (upper triangle mirrored)
__global__ void symm_upper_scale_kernel(double* P, int k, double inv_df) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= k * k) return;
  const int i = t % k, j = t / k;
  if (i <= j) {
    const double v = P[i + (size_t)j * k] * inv_df;
    P[i + (size_t)j * k] = v;
    if (i != j) P[j + (size_t)i * k] = v;
  }
}

// One component count's system: out = leading kk x kk block of P plus lambda I
// with lambda = ridge * trace / kk (reference ridge rule), and Mt (kk x C) = the
// transposed leading columns of the means.  Every block forms the trace itself.
__global__ void __launch_bounds__(256)
lda_system_kernel(const double* __restrict__ P, int kmax, int kk, double ridge, const double* __restrict__ M, int C,
                  double* __restrict__ out, double* __restrict__ Mt, double* lambda_out) {
  __shared__ double scratch[32];
  __shared__ double lam;
  double tr = 0.0;
  for (int i = threadIdx.x; i < kk; i += blockDim.x) tr += P[i + (size_t)i * kmax];
  tr = block_sum(tr, scratch);
  if (threadIdx.x == 0) {
    double scale = tr / static_cast<double>(kk > 0 ? kk : 1);
    if (!isfinite(scale) || scale <= 0.0) scale = 1.0;
    double l = ridge;
    if (!isfinite(l) || l < 0.0) l = 1e-8;
    lam = l * scale;
    if (blockIdx.x == 0) *lambda_out = lam;
  }
  __syncthreads();
  const int first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (int t = first; t < kk * kk; t += step) {
    const int i = t % kk, j = t / kk;
    out[t] = P[i + (size_t)j * kmax] + (i == j ? lam : 0.0);
  }
  for (int t = first; t < kk * C; t += step) {
    const int c = t % C, j = t / C;
    Mt[j + (size_t)c * kk] = M[t];
  }
}

// One component count's model, a thread a class: the means' and the solution's
// (Xs, kk x C) leading columns into means and linear (C x kmax, zero past kk),
// constants[c] = -0.5 means_c . linear_c + log(max(prior_c, DBL_MIN)) and, with
// an offset, adjusted[c] = constants[c] - linear_c . offset.  With the system
// above this is two launches a component count beside the solve, where copies,
// clears, transposes and the two sums of a class had been eight.
__global__ void __launch_bounds__(32)
lda_model_kernel(const double* __restrict__ M, const double* __restrict__ Xs, int C, int kk, int kmax,
                 const double* __restrict__ counts, int n, const double* __restrict__ offset,
                 double* __restrict__ means, double* __restrict__ linear, double* __restrict__ constants,
                 double* __restrict__ adjusted, double* __restrict__ priors) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  double d = 0.0, off = 0.0;
#pragma unroll 8
  for (int j = 0; j < kk; ++j) {
    const double mean = M[c + (size_t)j * C], x = Xs[j + (size_t)c * kk];
    means[c + (size_t)j * C] = mean;
    linear[c + (size_t)j * C] = x;
    d += mean * x;
    if (offset) off = fma(x, offset[j], off);
  }
  for (int j = kk; j < kmax; ++j) {
    means[c + (size_t)j * C] = 0.0;
    linear[c + (size_t)j * C] = 0.0;
  }
  const double prior = counts[c] / static_cast<double>(n);
  const double constant = -0.5 * d + log(fmax(prior, DBL_MIN));
  constants[c] = constant;
  if (offset) adjusted[c] = constant - off;
  if (priors) priors[c] = prior;
}

}  // namespace

void lowrank_predict(const double* Xs, int w, int p, const double* R, int kmax, const double* W,
                     int m, const int* ncomp_host, int L, const double* mY, double* T,
                     double* Ypred) {
  xgemm(false, w, kmax, p, Xs, w, R, p, T, w);
  for (int a = 0; a < L; ++a) {
    const int mc = ncomp_host[a];
    double* Ya = Ypred + (size_t)a * w * m;
    gemm(false, false, w, m, mc, 1.0, T, w, W + (size_t)a * kmax * m, kmax, 0.0, Ya, w, mY);
  }
}

void row_argmax(const double* S, int w, int C, const double* bias, int* labels) {
  if (w <= 0) return;
  // Rows enough to fill the GPU: a thread a row (1,000,000 x 3: 6.5 us against 42 in
  // lists; 100000 x 100: 10.7 against 12.1).  Else several warps share a row's classes
  // (125 x 22: 2.9 us against 4.6, 20000 x 100: 6.6 against 8.5, 3000 x 1000: 8.6
  // against 53).
  if (w >= 65536 ? C <= 128 : w >= 16384 ? C <= 48 : C <= 4) {
    argmax_kernel<<<ceil_div(w, 256), 256, 0, Context::get().stream>>>(S, w, C, bias, labels); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    return;
  }
  // first maximum; a NaN first score, or no finite one, leaves class 1
  row_topk_launch(S, w, C, bias, 1, 1, true, labels, nullptr);
}

void row_topk(const double* S, int w, int C, const double* bias, int top_k, int* idx,
              double* score) {
  FPLS_REQUIRE(top_k >= 1 && top_k <= kRowTopkMax, "top-k supports 1..32 classes per row");
  if (w <= 0) return;
  row_topk_launch(S, w, C, bias, top_k, 0, false, idx, score);
}

void lda_train_prefix(const double* T, int n, int kmax, const int* y_host, int C,
                      const int* ncomp_host, int L, double ridge, LdaModelsDev out) {
  Context& ctx = Context::get();
  FPLS_REQUIRE(n > 0 && kmax > 0, "lda_train_prefix requires a non-empty score matrix");
  FPLS_REQUIRE(C >= 2, "lda_train_prefix requires at least two classes");
  // class counts and a stable class-sorted row order (host, O(n))
  std::vector<int> off(C + 1, 0), perm(n);
  for (int i = 0; i < n; ++i) {
    const int cls = y_host[i] - 1;
    if (cls < 0 || cls >= C) throw Error(kErrArgument, "lda_train_prefix labels must be encoded as 1..n_classes");
    ++off[cls + 1];
  }
  std::vector<double> hc(C);
  for (int c = 0; c < C; ++c) {
    if (off[c + 1] <= 0) throw Error(kErrArgument, "lda_train_prefix received an empty class");
    hc[c] = off[c + 1];
    off[c + 1] += off[c];
  }
  {
    std::vector<int> cur(off.begin(), off.end() - 1);
    for (int i = 0; i < n; ++i) perm[cur[y_host[i] - 1]++] = i;
  }
  double* M = ctx.arena.alloc_n<double>((size_t)C * kmax);
  double* Mw = ctx.arena.alloc_n<double>((size_t)C * kmax);
  double* counts = ctx.arena.alloc_n<double>(C);
  int* d_perm = ctx.arena.alloc_n<int>(n);
  int* d_off = ctx.arena.alloc_n<int>(C + 1);
  h2d(counts, hc.data(), C * sizeof(double));
  h2d(d_perm, perm.data(), n * sizeof(int));
  h2d(d_off, off.data(), (C + 1) * sizeof(int));
  const long long warps = (long long)C * kmax;
  class_sums_sorted_kernel<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, ctx.stream>>>(T, n, kmax, d_perm,
                                                                                        d_off, C, M);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  means_from_sums_kernel<<<ceil_div(C * kmax, 256), 256, 0, ctx.stream>>>(M, C, kmax, counts, Mw); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  double* P = ctx.arena.alloc_n<double>((size_t)kmax * kmax);
  gemm(true, false, kmax, kmax, n, 1.0, T, n, T, n, 0.0, P, kmax);
  gemm(true, false, kmax, kmax, C, -1.0, M, C, Mw, C, 1.0, P, kmax);
  const double df = std::max(1.0, static_cast<double>(n) - static_cast<double>(C));
  symm_upper_scale_kernel<<<ceil_div(kmax * kmax, 256), 256, 0, ctx.stream>>>(P, kmax, 1.0 / df); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  double* Pk = ctx.arena.alloc_n<double>((size_t)kmax * kmax);
  double* Mt = ctx.arena.alloc_n<double>((size_t)kmax * C);
  double* Xs = ctx.arena.alloc_n<double>((size_t)kmax * C);
  double* lam = ctx.arena.alloc_n<double>(L);
  for (int a = 0; a < L; ++a) {
    const int kk = ncomp_host[a];
    const int blocks = std::max(1, std::min(ctx.sm_count, ceil_div(kk * std::max(kk, C), 1024)));
    lda_system_kernel<<<blocks, 256, 0, ctx.stream>>>(P, kmax, kk, ridge, M, C, Pk, Mt, lam + a); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    spd_solve(kk, Pk, kk, C, Mt, kk, Xs, kk, ctx.d_status + 5);
    lda_model_kernel<<<ceil_div(C, 32), 32, 0, ctx.stream>>>(
        M, Xs, C, kk, kmax, counts, n, out.offset, out.means + (size_t)a * C * kmax, out.linear + (size_t)a * C * kmax,
        out.constants + (size_t)a * C, out.offset ? out.adjusted + (size_t)a * C : nullptr,
        a == 0 ? out.priors : nullptr);
    ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
  }
  std::vector<double> hl(L);
  d2h(hl.data(), lam, L * sizeof(double));
  int singular = 0;
  d2h(&singular, ctx.d_status + 5, sizeof(int));
  ctx.sync();
  if (singular) throw Error(kErrNumerical, "LDA pooled covariance is singular");
  for (int a = 0; a < L; ++a) out.lambda[a] = hl[a];
}

}  // namespace fpls
