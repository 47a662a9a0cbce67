#include "blas_f64.cuh"
#include "context.cuh"
#include "linalg_small.cuh"
#include "null_columns.cuh"

#include <algorithm>
#include <type_traits>
#include <vector>

namespace fpls {
namespace {

constexpr double kEps = 2.220446049250313e-16;

// ---------------------------------------------------------------- Cholesky ---
// In-place lower Cholesky of A (k x k, lda) in global scratch; returns false via
// *ok = 0 when a pivot is not positive.
__device__ void chol_lower_inplace(double* A, int k, int lda, int* ok) {
  for (int j = 0; j < k; ++j) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const double d = A[j + (size_t)j * lda];
      if (!(d > 0.0) || !isfinite(d)) *ok = 0;
      else A[j + (size_t)j * lda] = sqrt(d);
    }
    __syncthreads();
    if (!*ok) return;
    const double ljj = A[j + (size_t)j * lda];
    for (int i = j + 1 + threadIdx.x; i < k; i += blockDim.x) A[i + (size_t)j * lda] /= ljj;
    __syncthreads();
    const int rem = k - j - 1;
    const long long tot = (long long)rem * rem;
    for (long long t = threadIdx.x; t < tot; t += blockDim.x) {
      const int ii = j + 1 + static_cast<int>(t % rem);
      const int ll = j + 1 + static_cast<int>(t / rem);
      if (ll <= ii) A[ii + (size_t)ll * lda] -= A[ii + (size_t)j * lda] * A[ll + (size_t)j * lda];
    }
  }
  __syncthreads();
}

// X = G^{-1} B by LU with partial pivoting on [G | B] (k x (k + nrhs)) in the
// global workspace W, for one CTA; raises *d_flag when G is singular.
__device__ void lu_solve(int k, const double* __restrict__ G, int ldg, double ridge, int nrhs,
                         const double* __restrict__ B, int ldb, double* __restrict__ X, int ldx, double* W,
                         int* d_flag) {
  __shared__ int piv, ok;
  if (threadIdx.x == 0) ok = 1;
  __syncthreads();
  const int ncol = k + nrhs;
  for (long long t = threadIdx.x; t < (long long)k * ncol; t += blockDim.x) {
    const int i = static_cast<int>(t % k), j = static_cast<int>(t / k);
    W[i + (size_t)j * k] = (j < k) ? G[i + (size_t)j * ldg] + (i == j ? ridge : 0.0)
                                   : B[i + (size_t)(j - k) * ldb];
  }
  for (int j = 0; j < k; ++j) {
    __syncthreads();
    if (threadIdx.x == 0) {
      int best = j;
      double bv = fabs(W[j + (size_t)j * k]);
      for (int i = j + 1; i < k; ++i) {
        const double v = fabs(W[i + (size_t)j * k]);
        if (v > bv) { bv = v; best = i; }
      }
      piv = best;
      if (!(bv > 0.0)) { ok = -1; }
    }
    __syncthreads();
    if (ok == -1) break;
    if (piv != j) {
      for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
        const double a = W[j + (size_t)c * k];
        W[j + (size_t)c * k] = W[piv + (size_t)c * k];
        W[piv + (size_t)c * k] = a;
      }
    }
    __syncthreads();
    const double pv = W[j + (size_t)j * k];
    const int rem = k - j - 1;
    const int cols = ncol - j - 1;
    for (long long t = threadIdx.x; t < (long long)rem * cols; t += blockDim.x) {
      const int i = j + 1 + static_cast<int>(t % rem);
      const int c = j + 1 + static_cast<int>(t / rem);
      W[i + (size_t)c * k] -= (W[i + (size_t)j * k] / pv) * W[j + (size_t)c * k];
    }
  }
  __syncthreads();
  if (ok == -1) {
    if (threadIdx.x == 0) atomicExch(d_flag, 1);
    return;
  }
  for (int c = threadIdx.x; c < nrhs; c += blockDim.x) {
    double* x = X + (size_t)c * ldx;
    for (int i = k - 1; i >= 0; --i) {
      double s = W[i + (size_t)(k + c) * k];
      for (int l = i + 1; l < k; ++l) s -= W[i + (size_t)l * k] * x[l];
      x[i] = s / W[i + (size_t)i * k];
    }
  }
}

// ridge_rel mean(diag G) (ridge_rel itself when that is not a positive number).
__device__ double ridge_of(int k, const double* __restrict__ G, int ldg, double ridge_rel) {
  __shared__ double scratch[32];
  if (!(ridge_rel > 0.0)) return 0.0;
  double dsum = 0.0;
  for (int i = threadIdx.x; i < k; i += blockDim.x) dsum += G[i + (size_t)i * ldg];
  dsum = block_sum(dsum, scratch);
  const double r = ridge_rel * dsum / static_cast<double>(k);
  return (!isfinite(r) || r <= 0.0) ? ridge_rel : r;
}

// Systems too large for shared memory: one CTA, the factor in global memory.
__global__ void spd_solve_large_kernel(int k, const double* __restrict__ G, int ldg, int nrhs,
                                       const double* __restrict__ B, int ldb, double* __restrict__ X,
                                       int ldx, double* W, int* d_flag, double ridge_rel) {
  __shared__ int ok;
  if (threadIdx.x == 0) ok = 1;
  const double ridge = ridge_of(k, G, ldg, ridge_rel);
  for (long long t = threadIdx.x; t < (long long)k * k; t += blockDim.x) {
    const int i = static_cast<int>(t % k), j = static_cast<int>(t / k);
    W[i + (size_t)j * k] = G[i + (size_t)j * ldg] + (i == j ? ridge : 0.0);
  }
  __syncthreads();
  chol_lower_inplace(W, k, k, &ok);
  if (!ok) {
    __syncthreads();
    lu_solve(k, G, ldg, ridge, nrhs, B, ldb, X, ldx, W, d_flag);
    return;
  }
  // Forward and back substitution, one thread per right-hand side.
  for (int c = threadIdx.x; c < nrhs; c += blockDim.x) {
    double* x = X + (size_t)c * ldx;
    const double* b = B + (size_t)c * ldb;
    for (int i = 0; i < k; ++i) {
      double s = b[i];
      for (int l = 0; l < i; ++l) s -= W[i + (size_t)l * k] * x[l];
      x[i] = s / W[i + (size_t)i * k];
    }
    for (int i = k - 1; i >= 0; --i) {
      double s = x[i];
      for (int l = i + 1; l < k; ++l) s -= W[l + (size_t)i * k] * x[l];
      x[i] = s / W[i + (size_t)i * k];
    }
  }
}

// ---- Cholesky factor and triangular solves in shared memory (k <= kCholMax) ---
// The factor is held column-major with an odd leading dimension of at least
// 8 NR (zero rows below k); eight lanes share one right-hand side, lane g with
// its entries g, g + 8, ... in NR registers, so a solved entry reaches the
// others by one shuffle and the update needs no barrier.  Every CTA factors
// its own copy (a few us, bound by the chain of k pivots) and then takes 64
// right-hand sides at a time: one launch instead of a factor launch and a solve
// launch, and no CTA waits for another.
constexpr int kCholMax = 160;
constexpr int kCholThreads = 512;
constexpr int kCholGroups = kCholThreads / 8;
constexpr int chol_ld(int nr) { return 8 * nr + 1; }
constexpr size_t chol_smem(int nr) { return (size_t)(8 * nr) * (chol_ld(nr) + 1) * sizeof(double); }

// Up to 16 columns (NR = 2) the factor takes roots and divisions in the order
// of the plain right-looking loop, as it always did: the OPLS filter's
// subspace iteration runs on eight columns, and the split-precision products
// behind it turn a different last bit into 1e-5 of the trailing components.
// Larger ones multiply by reciprocal roots.
template <int NR>
constexpr bool kCholDivides = NR <= 2;
template <int NR>
__device__ __forceinline__ double over_diag(double v, double d) { return kCholDivides<NR> ? v / d : v * d; }

// Factors G (+ ridge) into L; diag[j] = L[j][j], or its reciprocal where the
// solves multiply.  False (in every thread) when a pivot is not positive.  The
// trailing matrix stays in registers (lane = rows lane, lane + 32, ..., warp =
// columns warp, warp + 16, ...); a column reaches shared memory, scaled by its
// owning warp, just before it is used, so a column costs one barrier and its
// chain is barrier, load, multiply-add, shuffle, root.
template <int NR>
__device__ bool chol_factor(int k, const double* __restrict__ G, int ldg, double ridge, double* L, double* diag) {
  constexpr int ld = chol_ld(NR), kWarps = kCholThreads / 32;
  constexpr int U = (8 * NR + 31) / 32, M = (8 * NR + kWarps - 1) / kWarps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double a[U][M];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int i = lane + 32 * u, c = warp + kWarps * m;
      a[u][m] = (i < k && c <= i) ? G[i + (size_t)c * ldg] + (i == c ? ridge : 0.0) : 0.0;
    }
  for (int j = 0; j < k; ++j) {
    if (warp == j % kWarps) {
      const int mj = j / kWarps, uj = j / 32;
      double v[U], pivot = 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        v[u] = 0.0;
#pragma unroll
        for (int m = 0; m < M; ++m) v[u] = m == mj ? a[u][m] : v[u];
        pivot = u == uj ? v[u] : pivot;
      }
      pivot = __shfl_sync(0xffffffffu, pivot, j & 31);
      const bool good = pivot > 0.0 && isfinite(pivot);
      const double d = !good ? -1.0 : kCholDivides<NR> ? sqrt(pivot) : rsqrt(pivot);
      if (lane == 0) diag[j] = d;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = lane + 32 * u;
        if (i < 8 * NR) L[i + j * ld] = i > j ? over_diag<NR>(v[u], d) : 0.0;
      }
    }
    __syncthreads();
    if (diag[j] < 0.0) return false;
    double f[M];
#pragma unroll
    for (int m = 0; m < M; ++m) f[m] = warp + kWarps * m < 8 * NR ? L[warp + kWarps * m + j * ld] : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double li = lane + 32 * u < 8 * NR ? L[lane + 32 * u + j * ld] : 0.0;
#pragma unroll
      for (int m = 0; m < M; ++m) a[u][m] -= li * f[m];
    }
  }
  return true;
}

// y <- L^{-1} y for the group's right-hand side.
template <int NR>
__device__ __forceinline__ void solve_lower(double (&y)[NR], int k, int g, const double* L, const double* diag) {
  constexpr int ld = chol_ld(NR);
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    if (8 * r >= k) break;
#pragma unroll 2
    for (int jl = 0; jl < 8; ++jl) {
      const int j = 8 * r + jl;
      if (j >= k) break;
      const double q = __shfl_sync(0xffffffffu, over_diag<NR>(y[r], diag[j]), jl, 8);
      const double* col = L + g + j * ld;
      y[r] = g == jl ? q : g > jl ? y[r] - col[8 * r] * q : y[r];
#pragma unroll
      for (int u = r + 1; u < NR; ++u) y[u] -= col[8 * u] * q;
    }
  }
}

// y <- L^{-T} y.
template <int NR>
__device__ __forceinline__ void solve_lower_t(double (&y)[NR], int k, int g, const double* L, const double* diag) {
  constexpr int ld = chol_ld(NR);
#pragma unroll
  for (int r = NR - 1; r >= 0; --r) {
    if (8 * r >= k) continue;
#pragma unroll 2
    for (int jl = 7; jl >= 0; --jl) {
      const int j = 8 * r + jl;
      if (j >= k) continue;
      const double q = __shfl_sync(0xffffffffu, over_diag<NR>(y[r], diag[j]), jl, 8);
      const double* row = L + j + g * ld;
      y[r] = g == jl ? q : g < jl ? y[r] - row[8 * r * ld] * q : y[r];
#pragma unroll
      for (int u = 0; u < r; ++u) y[u] -= row[8 * u * ld] * q;
    }
  }
}

template <int NR>
__global__ void __launch_bounds__(kCholThreads)
spd_solve_kernel(int k, const double* __restrict__ G, int ldg, int nrhs, const double* __restrict__ B, int ldb,
                 double* __restrict__ X, int ldx, double* W, int* d_flag, double ridge_rel) {
  extern __shared__ double L[];
  double* diag = L + 8 * NR * chol_ld(NR);
  const double ridge = ridge_of(k, G, ldg, ridge_rel);
  if (!chol_factor<NR>(k, G, ldg, ridge, L, diag)) {
    if (blockIdx.x == 0) lu_solve(k, G, ldg, ridge, nrhs, B, ldb, X, ldx, W, d_flag);
    return;
  }
  const int g = threadIdx.x & 7, group = threadIdx.x >> 3;
  for (int c0 = blockIdx.x * kCholGroups; c0 < nrhs; c0 += gridDim.x * kCholGroups) {
    const int c = c0 + group;
    double y[NR];
#pragma unroll
    for (int u = 0; u < NR; ++u) y[u] = (c < nrhs && g + 8 * u < k) ? B[g + 8 * u + (size_t)c * ldb] : 0.0;
    solve_lower<NR>(y, k, g, L, diag);
    solve_lower_t<NR>(y, k, g, L, diag);
#pragma unroll
    for (int u = 0; u < NR; ++u)
      if (c < nrhs && g + 8 * u < k) X[g + 8 * u + (size_t)c * ldx] = y[u];
  }
}

// One CholeskyQR pass: Q = Y R^{-1} with G = Y^T Y = R^T R (each row of Q solves
// R^T q = y).  Raises *d_flag when G is not positive definite.
template <int NR>
__global__ void __launch_bounds__(kCholThreads)
chol_qr_kernel(int k, const double* __restrict__ G, int rows, const double* Y, int ldy, double* Q, int ldq,
               int* d_flag) {
  extern __shared__ double L[];
  double* diag = L + 8 * NR * chol_ld(NR);
  if (!chol_factor<NR>(k, G, k, 0.0, L, diag)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicExch(d_flag, 1);
    return;
  }
  const int g = threadIdx.x & 7, group = threadIdx.x >> 3;
  for (int i0 = blockIdx.x * kCholGroups; i0 < rows; i0 += gridDim.x * kCholGroups) {
    const int i = i0 + group;
    double y[NR];
#pragma unroll
    for (int u = 0; u < NR; ++u) y[u] = (i < rows && g + 8 * u < k) ? Y[i + (size_t)(g + 8 * u) * ldy] : 0.0;
    solve_lower<NR>(y, k, g, L, diag);
#pragma unroll
    for (int u = 0; u < NR; ++u)
      if (i < rows && g + 8 * u < k) Q[i + (size_t)(g + 8 * u) * ldq] = y[u];
  }
}

// The register count of a size: f(std::integral_constant<int, NR>).
template <typename F>
void with_chol_size(int k, F&& f) {
  if (k <= 16) f(std::integral_constant<int, 2>{});
  else if (k <= 32) f(std::integral_constant<int, 4>{});
  else if (k <= 64) f(std::integral_constant<int, 8>{});
  else if (k <= 104) f(std::integral_constant<int, 13>{});
  else if (k <= 128) f(std::integral_constant<int, 16>{});
  else f(std::integral_constant<int, 20>{});
}

template <typename K>
void allow_smem(K kernel, size_t bytes) {
  FPLS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
}

// ------------------------------------------------- Gram-Schmidt fallback ---
__global__ void normalize_col_kernel(double* q, int rows, const double* nrm2) {
  const double nr = sqrt(*nrm2);
  const double inv = (nr > 0.0 && isfinite(nr)) ? 1.0 / nr : 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x)
    q[i] *= inv;
}

__global__ void dot_self_kernel(const double* x, int n, double* out) {
  __shared__ double scratch[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += x[i] * x[i];
  s = block_sum(s, scratch);
  if (threadIdx.x == 0) *out = s;
}

// ------------------------------------------------------------- Jacobi eigen ---
// Up to kEigTiny the rotations are applied in place, rows then columns, V along
// with W.  The OPLS filter takes its leading vectors through 8 x 8 cores of
// this size; the split-precision products behind it turn a different last bit
// here into 1e-5 of the trailing components, so this arithmetic stays.
constexpr int kEigTiny = 16;
__global__ void jacobi_eig_tiny_kernel(int l, const double* __restrict__ G, int ldg, double* evals_out,
                                       double* V_out, int ldv, const int max_sweeps) {
  extern __shared__ double sm[];
  const int npair = (l + 1) / 2;
  const int le = 2 * npair;
  double* cs = sm;              // [npair] cos
  double* sn = sm + npair;      // [npair] sin
  int* arr = reinterpret_cast<int*>(sm + 2 * npair);   // [le]
  int* pp = arr + le;           // [npair]
  int* qq = pp + npair;         // [npair]
  __shared__ double scratch[32];
  __shared__ int sweep_done;
  double* W = sm + 4 * npair;
  double* V = W + (size_t)l * l;
  for (int t = threadIdx.x; t < l * l; t += blockDim.x) W[t] = G[t % l + (size_t)(t / l) * ldg];
  for (int t = threadIdx.x; t < l * l; t += blockDim.x) V[t] = (t % l == t / l) ? 1.0 : 0.0;
  __shared__ int rotated;
  __syncthreads();
  // Frobenius norm for the convergence test.
  double fro = 0.0;
  for (int t = threadIdx.x; t < l * l; t += blockDim.x) fro += W[t] * W[t];
  fro = block_sum(fro, scratch);
  const double thresh = kEps * kEps * fro;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    double off = 0.0;
    for (int t = threadIdx.x; t < l * l; t += blockDim.x) {
      const int i = t % l, j = t / l;
      if (i != j) off += W[t] * W[t];
    }
    off = block_sum(off, scratch);
    if (threadIdx.x == 0) {
      sweep_done = (off <= thresh) ? 1 : 0;
      rotated = 0;
    }
    __syncthreads();
    if (sweep_done) break;
    for (int r = 0; r < le - 1; ++r) {
      // round-robin pairing of round r: position 0 stays, positions 1..le-1
      // have turned r places (position i holds 1 + (i - 1 - r) mod (le - 1))
      for (int k = threadIdx.x; k < npair; k += blockDim.x) {
        const int ik = le - 1 - k;
        int p = k == 0 ? 0 : 1 + ((k - 1 - r) % (le - 1) + (le - 1)) % (le - 1);
        int q = 1 + ((ik - 1 - r) % (le - 1) + (le - 1)) % (le - 1);
        if (p > q) { const int t = p; p = q; q = t; }
        pp[k] = p; qq[k] = q;
        double c = 1.0, s = 0.0;
        if (q < l) {
          const double apq = W[p + (size_t)q * l];
          const double app = W[p + (size_t)p * l];
          const double aqq = W[q + (size_t)q * l];
          // a rotation is skipped once the pair is decoupled to rounding
          if (apq != 0.0 && fabs(apq) > 1e-300 && fabs(apq) > kEps * sqrt(fabs(app * aqq))) {
            const double tau = (aqq - app) / (2.0 * apq);
            const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
            c = 1.0 / sqrt(1.0 + t * t);
            s = t * c;
            rotated = 1;
          }
        }
        cs[k] = c; sn[k] = s;
      }
      __syncthreads();
      {
        // lane = pair, warps stride over the rows / columns (no index division)
        const int k = threadIdx.x & 31, w0 = threadIdx.x >> 5, nw = blockDim.x >> 5;
        const bool act = k < npair && qq[k] < l && sn[k] != 0.0;
        const int p = act ? pp[k] : 0, q = act ? qq[k] : 0;
        const double c = act ? cs[k] : 1.0, sv = act ? sn[k] : 0.0;
        // rows: W <- J^T W
        if (act)
          for (int j = w0; j < l; j += nw) {
            const double wp = W[p + j * l], wq = W[q + j * l];
            W[p + j * l] = c * wp - sv * wq;
            W[q + j * l] = sv * wp + c * wq;
          }
        __syncthreads();
        // columns: W <- W J, V <- V J
        if (act)
          for (int i = w0; i < l; i += nw) {
            const double wp = W[i + p * l], wq = W[i + q * l];
            W[i + p * l] = c * wp - sv * wq;
            W[i + q * l] = sv * wp + c * wq;
            const double vp = V[i + p * l], vq = V[i + q * l];
            V[i + p * l] = c * vp - sv * vq;
            V[i + q * l] = sv * vp + c * vq;
          }
        __syncthreads();
      }
    }
    if (!rotated) break;   // a whole sweep without a rotation: converged
  }
  // Sort eigenvalues descending (selection order kept in arr).
  if (threadIdx.x == 0) {
    for (int i = 0; i < l; ++i) arr[i] = i;
    for (int i = 0; i < l; ++i) {
      int best = i;
      for (int j = i + 1; j < l; ++j)
        if (W[arr[j] + (size_t)arr[j] * l] > W[arr[best] + (size_t)arr[best] * l]) best = j;
      const int t = arr[i]; arr[i] = arr[best]; arr[best] = t;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < l; i += blockDim.x) evals_out[i] = W[arr[i] + (size_t)arr[i] * l];
  for (long long t = threadIdx.x; t < (long long)l * l; t += blockDim.x) {
    const int i = static_cast<int>(t % l), j = static_cast<int>(t / l);
    V_out[i + (size_t)j * ldv] = V[i + (size_t)arr[j] * l];
  }
}

// Cyclic two-sided Jacobi on one CTA, for l <= kEigMax.  What bounds it is the
// chain of rounds (le - 1 a sweep, six to nine sweeps), so a round is one
// barrier long:
//  * W is held by round-robin position, not by index (upper triangle), twice in
//    shared memory: a round reads one copy and writes the other with every
//    position moved on by one, so each thread's addresses are the same in
//    every round and no barrier stands between the two halves of a rotation;
//    one thread takes the 2 x 2 block of two pairs through both;
//  * meanwhile one warp (two above 64) works out the next round's angles from
//    the old blocks that its pairs come from, on a scheduler that the update
//    warps leave to it: its chain of dependent FP64 operations is as long as
//    the whole update;
//  * V takes no part: the angles go to a log in global memory, and
//    jacobi_apply_log_kernel runs V's rows through it, one warp a row, all
//    rows at once over the GPU.
// Measured: 0.66 us a round at 60 x 60 (the angles alone 0.47 us, the update
// alone 0.37 us), 302 us + 50 us for V against 1600 us when W and V were updated
// in place with three barriers a round; 110 x 110: 0.8 + 0.15 ms against 4.1 ms
// of the whole-GPU one-sided Jacobi with its grid barrier a round.
constexpr int kEigMax = 112;         // two copies of W in 227 KB of shared memory
constexpr int kEigWarps = 32;
constexpr int kEigSweeps = 60;
constexpr int eig_blocks(int npair) { return npair * (npair / 2 + 1); }
constexpr int kEigUpdate = 32 * (kEigWarps / 4) * 3;   // update threads, at most: schedulers 1 to 3
constexpr int kEigBlocks = (eig_blocks(kEigMax / 2) + kEigUpdate - 1) / kEigUpdate;

__device__ __forceinline__ int upper_at(int i, int j, int ld) { return i < j ? i + j * ld : j + i * ld; }

struct Rot { double c, s; };   // top' = c top - s bot, bot' = s top + c bot

// Whether the pair (p, q) is still coupled: |apq| above rounding of its diagonal.
__device__ __forceinline__ bool coupled(double app, double apq, double aqq) {
  return fabs(apq) > 1e-300 && fabs(apq) > kEps * sqrt(fabs(app * aqq));
}

// The rotation that decouples the pair (top, bot); a pair decoupled to rounding
// is left alone.  tan solves wtb t^2 + (wbb - wtt) t - wtb = 0: its first value
// comes from single precision (of numbers scaled by the larger one's power of
// two) and one Newton step on that equation takes it to about 1e-13, which is
// far below what the next sweep removes; the cosine is full double precision,
// so the rotation is orthogonal to rounding whatever the angle.  `swap`: the
// top index is the larger one (equal diagonals turn by +45 degrees from the
// smaller index).
__device__ __forceinline__ Rot decouple(bool swap, double wtt, double wtb, double wbb) {
  const double d = wbb - wtt;
  const int hid = __double2hiint(d) & 0x7ff00000, hiw = __double2hiint(wtb) & 0x7ff00000;
  const int ex = max(hid, hiw);                      // exponent bits of the larger one
  const bool plain = ex < 0x5d000000 && ex > 0x2b500000;   // about 1e-100 .. 1e140
  const double scale = __hiloint2double(0x7fe00000 - (plain ? ex : 0x3ff00000), 0);   // 2^-exponent
  const double ds = d * scale, es = wtb * scale;
  const float df = static_cast<float>(ds), ef = static_cast<float>(es);
  const float sq = fmaf(df, df, 4.0f * ef * ef);     // >= 1 (plain)
  const float root = sq * rsqrtf(sq);
  const float tf = __fdividef(2.0f * ef, df >= 0.0f ? df + root : df - root);
  double t = static_cast<double>(tf);
  t -= fma(es, fma(t, t, -1.0), ds * t) * static_cast<double>(__fdividef(1.0f, fmaf(2.0f * ef, tf, df)));
  bool go = wtb * wtb > (kEps * kEps) * fabs(wtt * wbb) && hiw > 0x20b00000;   // above 1e-150
  if (!plain) {
    go = coupled(wtt, wtb, wbb);
    const double tau = go ? d / (2.0 * wtb) : 0.0;
    t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
  } else if (fabsf(tf) < 1e-18f) {
    t = go ? wtb / d : 0.0;   // the small-angle limit
  }
  if (d == 0.0) t = swap ? -1.0 : 1.0;
  t = go ? t : 0.0;
  Rot r;
  r.c = rsqrt(fma(t, t, 1.0));
  r.s = t * r.c;
  return r;
}

// Element (x, y) of the rotated block w of two pairs: x is the first pair's
// top or bottom, y the second's.
__device__ __forceinline__ double rotated_at(const double (&w)[4], Rot ra, bool x_top, Rot rb, bool y_top) {
  const double u0 = x_top ? ra.c : ra.s, u1 = x_top ? -ra.s : ra.c;
  const double v0 = y_top ? rb.c : rb.s, v1 = y_top ? -rb.s : rb.c;
  return fma(v0, fma(u0, w[0], u1 * w[2]), v1 * fma(u0, w[1], u1 * w[3]));
}

// Round-robin: position 0 keeps its index, the others move on by one a round;
// pair k is the positions k (top) and le - 1 - k (bottom).
__device__ __forceinline__ int next_position(int i, int le) { return i == 0 ? 0 : i == le - 1 ? 1 : i + 1; }
__device__ __forceinline__ int ring_prev(int i, int le) { return i == 1 ? le - 1 : i - 1; }

// Offsets of the block of pairs a and b in W (from), and of where its elements
// go (to).
__device__ __forceinline__ void block_offsets(int a, int b, int le, int ld, int (&from)[4], int (&to)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int i = e & 2 ? le - 1 - a : a, j = e & 1 ? le - 1 - b : b;
    from[e] = upper_at(i, j, ld);
    to[e] = upper_at(next_position(i, le), next_position(j, le), ld);
  }
}

template <int NB>   // blocks of the pair grid per update thread
__global__ void __launch_bounds__(32 * kEigWarps)
jacobi_eig_kernel(int l, const double* __restrict__ G, int ldg, double* __restrict__ evals, int* __restrict__ rank_of,
                  double2* __restrict__ log, int* __restrict__ rounds_out, int max_sweeps) {
  extern __shared__ double sm[];
  // Along a warp the two positions of a block move by one each, so an even
  // leading dimension makes every step odd: no bank conflicts.
  const int le = l + (l & 1), npair = le / 2, ld = le, half = le * ld;
  Rot* rots = reinterpret_cast<Rot*>(sm + 2 * half);   // [2][npair]
  __shared__ double scratch[32];
  __shared__ int open;
  const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31;
  for (int t = tid; t < le * le; t += nt) {
    const int i = t % le, j = t / le;
    sm[i + j * ld] = (i < l && j < l) ? G[i + (size_t)j * ldg] : 0.0;
  }
  __syncthreads();
  double fro = 0.0;
  for (int t = tid; t < l * l; t += nt) {
    const double w = sm[t % l + (t / l) * ld];
    fro += w * w;
  }
  const double thresh = kEps * kEps * block_sum(fro, scratch);
  // Warps 0 and 4 work out the angles (pair k); the warps of schedulers 1 to 3
  // update, each thread the block of a pair a (fastest) with pair a + delta
  // around the ring, delta up to half of it: one thread for each couple of pairs.
  const int k = warp == 0 ? lane : lane + 32;
  const bool angles = (warp == 0 || warp == 4) && k < npair;
  const int update = 32 * 3 * (nt / 128), uid = 32 * (3 * (warp >> 2) + (warp & 3) - 1) + lane;
  int pa[NB], pb[NB], from[NB][4], to[NB][4];
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    pa[u] = -1;
    const int t = uid + u * update, a = t % npair, delta = t / npair;
    if ((warp & 3) == 0 || 2 * delta > npair || (2 * delta == npair && a >= npair / 2)) continue;
    pa[u] = a;
    pb[u] = a + delta < npair ? a + delta : a + delta - npair;
    block_offsets(pa[u], pb[u], le, ld, from[u], to[u]);
  }
  // the current pairs whose indices pair k has next: its top is the top of
  // k - 1 (the bottom of 0 for k = 1), its bottom the bottom of k + 1 (the top
  // of the last pair for the last)
  const int A = k == 0 ? 0 : k - 1, B = min(k + 1, npair - 1);
  const bool a_top = k != 1, b_top = k == npair - 1 && npair > 1;
  int faa[4], fab[4], fbb[4], unused[4];
  int top = k, bot = le - 1 - k;   // pair k's indices
  if (angles) {
    block_offsets(A, A, le, ld, faa, unused);
    block_offsets(A, B, le, ld, fab, unused);
    block_offsets(B, B, le, ld, fbb, unused);
    rots[k] = decouple(top > bot, sm[top + top * ld], sm[upper_at(top, bot, ld)], sm[bot + bot * ld]);
  }
  int cur = 0, round = 0;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    // converged when the off-diagonal part is at rounding of the whole, or no
    // pair is coupled any more (which a sweep without a rotation would show)
    if (tid == 0) open = 0;
    const double* Wc = sm + cur * half;
    double off = 0.0;
    bool mine = false;
    __syncthreads();
    for (int t = tid; t < l * l; t += nt) {
      const int i = t % l, j = t / l;
      if (i < j) {
        const double w = Wc[i + j * ld];
        off += 2.0 * w * w;
        mine = mine || coupled(Wc[i + i * ld], w, Wc[j + j * ld]);
      }
    }
    if (mine) open = 1;
    off = block_sum(off, scratch);
    if (off <= thresh || !open) break;
    for (int r = 0; r < le - 1; ++r, ++round) {
      const double* W = sm + cur * half;
      double* Wn = sm + (cur ^ 1) * half;
      const Rot* rc = rots + cur * npair;
      if (angles) {
        const Rot rA = rc[A], rB = rc[B];
        double waa[4], wab[4], wbb[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          waa[e] = W[faa[e]];
          wab[e] = W[fab[e]];
          wbb[e] = W[fbb[e]];
        }
        if (k != 0) top = ring_prev(top, le);
        bot = ring_prev(bot, le);
        rots[(cur ^ 1) * npair + k] = decouple(top > bot, rotated_at(waa, rA, a_top, rA, a_top),
                                               rotated_at(wab, rA, a_top, rB, b_top),
                                               rotated_at(wbb, rB, b_top, rB, b_top));
        log[(size_t)round * npair + k] = make_double2(rc[k].c, rc[k].s);
      }
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        if (pa[u] < 0) continue;
        const Rot ra = rc[pa[u]], rb = rc[pb[u]];
        const double w00 = W[from[u][0]], w01 = W[from[u][1]], w10 = W[from[u][2]], w11 = W[from[u][3]];
        const double r00 = ra.c * w00 - ra.s * w10, r01 = ra.c * w01 - ra.s * w11;
        const double r10 = ra.s * w00 + ra.c * w10, r11 = ra.s * w01 + ra.c * w11;
        Wn[to[u][0]] = rb.c * r00 - rb.s * r01;
        Wn[to[u][1]] = rb.s * r00 + rb.c * r01;
        if (pa[u] != pb[u]) Wn[to[u][2]] = rb.c * r10 - rb.s * r11;
        Wn[to[u][3]] = rb.s * r10 + rb.c * r11;
      }
      cur ^= 1;
      __syncthreads();
    }
  }
  // a whole number of sweeps: every position holds its own index again
  if (tid == 0) *rounds_out = round;
  const double* Wc = sm + cur * half;
  for (int i = tid; i < l; i += nt) {
    const double ev = Wc[i + i * ld], v = isnan(ev) ? -INFINITY : ev;
    int rank = 0;
    for (int j = 0; j < l; ++j) {
      const double wj = Wc[j + j * ld], w = isnan(wj) ? -INFINITY : wj;
      rank += (w > v) || (w == v && j < i);
    }
    rank_of[i] = rank;
    evals[rank] = ev;
  }
}

// Row i of V = e_i through the logged rotations, written in the eigenvalues'
// order.  One warp a row (lane = pair, and pair + 32), the row in shared
// memory, kStage rounds of angles loaded ahead: bound by the latency of one
// round's shared-memory update, for all rows at once.
constexpr int kApplyWarps = 4;
template <int PP>   // pairs per lane
__global__ void __launch_bounds__(32 * kApplyWarps)
jacobi_apply_log_kernel(int l, const double2* __restrict__ log, const int* __restrict__ rounds,
                        const int* __restrict__ rank_of, double* __restrict__ V, int ldv) {
  __shared__ double rows[kApplyWarps][kEigMax + 2];
  constexpr int kStage = 16 / PP;
  const int le = l + (l & 1), npair = le / 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * kApplyWarps + warp;
  if (i >= l) return;   // whole warps; no block-wide barrier below
  double* row = rows[warp];
  for (int j = lane; j < le; j += 32) row[j] = j == i ? 1.0 : 0.0;
  __syncwarp();
  int top[PP], bot[PP];
#pragma unroll
  for (int u = 0; u < PP; ++u) {
    const int k = lane + 32 * u;
    top[u] = k;
    bot[u] = le - 1 - k;
  }
  const int R = *rounds;
  double2 now[kStage][PP], next[kStage][PP];
  auto fetch = [&](int r0, double2 (&d)[kStage][PP]) {
#pragma unroll
    for (int g = 0; g < kStage; ++g)
#pragma unroll
      for (int u = 0; u < PP; ++u) {
        const int k = lane + 32 * u;
        d[g][u] = (r0 + g < R && k < npair) ? __ldg(log + (size_t)(r0 + g) * npair + k) : make_double2(1.0, 0.0);
      }
  };
  fetch(0, now);
  for (int r0 = 0; r0 < R; r0 += kStage) {
    fetch(r0 + kStage, next);
#pragma unroll
    for (int g = 0; g < kStage; ++g) {
      if (r0 + g < R) {
#pragma unroll
        for (int u = 0; u < PP; ++u) {
          if (lane + 32 * u < npair) {
            const double c = now[g][u].x, s = now[g][u].y;
            const double x = row[top[u]], y = row[bot[u]];
            row[top[u]] = c * x - s * y;
            row[bot[u]] = s * x + c * y;
            if (lane + 32 * u != 0) top[u] = ring_prev(top[u], le);
            bot[u] = ring_prev(bot[u], le);
          }
        }
        __syncwarp();
      }
    }
#pragma unroll
    for (int g = 0; g < kStage; ++g)
#pragma unroll
      for (int u = 0; u < PP; ++u) now[g][u] = next[g][u];
  }
  for (int j = lane; j < l; j += 32) V[i + (size_t)rank_of[j] * ldv] = row[j];
}

// ---------------------------------------------------------- one-sided Jacobi ---
// ---- Thin SVD of up to kThinMax columns: QR first, one-sided Jacobi on R ----
// The rotations of one-sided Jacobi depend on the columns' inner products only,
// and those of A = Q R are those of R; so A is reduced to its c x c triangle by
// Householder QR over row blocks (one CTA a block, the blocks' triangles stacked
// and reduced again) and the sweeps run on R.  A sweep over A itself moves its
// columns three times through shared (or global) memory: 375 x 22 took 340 us
// that way, 5000 x 22 several ms.  U = Q (R V / s): the rotated columns R V are
// orthogonal to rounding whatever their lengths, and the reflectors keep them so.
// (U = A V / s, one product, loses orthogonality as 1 / s, and a NaN of A reaches
// every column.)
constexpr int kThinMax = 96;

// R (c x c, upper) of rows [b rb, b rb + rb) of A into rows [b c, b c + c) of
// out.  Every warp works out the reflector of a column for itself and applies it
// to its own columns, so a column costs one barrier.  The reflectors I - tau v v^T
// stay in F (rows x c, v from the diagonal down) and tau (c a block).
__global__ void __launch_bounds__(512) qr_block_kernel(const double* __restrict__ A, int rows, int c, int lda, int rb,
                                                       double* __restrict__ out, int ldo, double* __restrict__ F,
                                                       double* __restrict__ tau) {
  extern __shared__ double sm[];
  double* X = sm;                       // [rb][c], column-major
  double* diag = sm + (size_t)rb * c;   // [c]
  double* heads = diag + c;             // [c]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int r0 = blockIdx.x * rb, nr = min(rb, rows - r0), steps = min(c, nr);
  for (int j = warp; j < c; j += nw)
    for (int i = lane; i < nr; i += 32) X[i + j * rb] = A[r0 + i + (size_t)j * lda];
  __syncthreads();
  for (int j = 0; j < steps; ++j) {
    const double* x = X + j * rb;
    double sigma = 0.0;
    for (int i = j + 1 + lane; i < nr; i += 32) sigma += x[i] * x[i];
    sigma = warp_sum(sigma);
    const double alpha = x[j], norm = sqrt(alpha * alpha + sigma);
    const double beta = alpha >= 0.0 ? -norm : norm, head = alpha - beta;
    const double inv = norm > 0.0 ? 1.0 / (norm * (norm + fabs(alpha))) : 0.0;   // 2 / v.v, v = (head, x below)
    if (threadIdx.x == 0) {
      diag[j] = beta;
      heads[j] = head;
      tau[blockIdx.x * c + j] = inv;
    }
    if (norm > 0.0) {
      for (int col = j + 1 + warp; col < c; col += nw) {
        double* y = X + col * rb;
        double d = 0.0;
        for (int i = j + 1 + lane; i < nr; i += 32) d += x[i] * y[i];
        const double yj = y[j], w = (warp_sum(d) + head * yj) * inv;
        for (int i = j + 1 + lane; i < nr; i += 32) y[i] -= w * x[i];
        __syncwarp();
        if (lane == 0) y[j] = yj - w * head;
      }
    }
    __syncthreads();
  }
  for (int j = warp; j < c; j += nw) {
    for (int i = lane; i < c; i += 32) {
      const double v = i < j ? (i < nr ? X[i + j * rb] : 0.0) : i == j && j < steps ? diag[j] : 0.0;
      out[blockIdx.x * c + i + (size_t)j * ldo] = v;
    }
    if (j < steps)
      for (int i = j + lane; i < nr; i += 32) F[r0 + i + (size_t)j * rows] = i == j ? heads[j] : X[i + j * rb];
  }
}

// Rows [b rb, b rb + rb) of Z (rows x need) = the block's reflectors applied to rows
// [b c, b c + c) of Y, zero below.  The reflectors come into shared memory once; one
// warp a column then, its rows in registers, without barriers: a reflector is a shuffle
// tree and two passes over the registers (375 x 22: 13 us with each reflector fetched
// from L2 ahead of its turn).
constexpr int kApplyCols = 8;   // columns (warps) a CTA
template <int NE>               // 32 NE rows at least
__global__ void __launch_bounds__(32 * kApplyCols)
qr_apply_kernel(const double* __restrict__ F, const double* __restrict__ tau, int rows, int c, int rb,
                const double* __restrict__ Y, int ldy, int need, double* __restrict__ Z, int ldz) {
  extern __shared__ double sm[];   // [rb][c] reflectors, [c] tau
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col = blockIdx.y * kApplyCols + warp;
  const int b = blockIdx.x, r0 = b * rb, nr = min(rb, rows - r0), steps = min(c, nr);
  double* taus = sm + (size_t)rb * c;
  for (int j = warp; j < steps; j += kApplyCols) {
#pragma unroll 8
    for (int i = lane; i < nr; i += 32) sm[i + j * rb] = i >= j ? F[r0 + i + (size_t)j * rows] : 0.0;
    if (lane == 0) taus[j] = tau[(size_t)b * c + j];
  }
  double z[NE];
#pragma unroll
  for (int e = 0; e < NE; ++e)
    z[e] = lane + 32 * e < steps && col < need ? Y[(size_t)b * c + lane + 32 * e + (size_t)col * ldy] : 0.0;
  __syncthreads();
  if (col >= need) return;
  for (int j = steps - 1; j >= 0; --j) {
    const double t = taus[j];
    double v[NE], part[2] = {0.0, 0.0};   // two chains: a multiply-add waits 16 cycles for the one before
#pragma unroll
    for (int e = 0; e < NE; ++e) v[e] = lane + 32 * e < nr ? sm[lane + 32 * e + j * rb] : 0.0;
#pragma unroll
    for (int e = 0; e < NE; ++e) part[e & 1] = fma(v[e], z[e], part[e & 1]);
    const double d = warp_sum(part[0] + part[1]) * t;
    if (t == 0.0) continue;   // a column without a reflector (zero, or not a number)
#pragma unroll
    for (int e = 0; e < NE; ++e) z[e] -= d * v[e];
  }
#pragma unroll
  for (int e = 0; e < NE; ++e)
    if (lane + 32 * e < nr) Z[r0 + lane + 32 * e + (size_t)col * ldz] = z[e];
}

// A column whose norm is below 4 eps c of the columns' root mean square may be a null
// direction: its angle to the others is rounding, which no rotation removes, so a
// rank-deficient matrix (every centred class response) would only stop when the column
// has underflowed.  Such a column is rotated, which resolves a small singular value and
// takes a null direction down by eps a sweep, but asks for no further sweep, and is left
// alone below the square of this share.
__device__ inline double null_share(int c) { return 4.0 * kEps * c; }

// One-sided Jacobi on R (c x c, column-major), one CTA, one warp a column pair,
// the pairs turning as in the symmetric solver: singular values, and of V and of
// R V / s the first `need` columns, descending (R V / s: c x need; zero where s is
// at most tol_rel of the largest).  A column of R and the one of V below it sit in
// NE registers a lane each while their rotation is worked out.
template <int NE>
__global__ void __launch_bounds__(1024)
jacobi_core_kernel(const double* __restrict__ R, int c, int max_sweeps, double tol_rel, int need, double* __restrict__ s_out,
                   double* __restrict__ V_out, int ldv, double* __restrict__ RV_out) {
  extern __shared__ double sm[];
  double* W = sm;                       // [c][c]
  double* V = W + c * c;
  double* norms = V + c * c;
  __shared__ double scratch[32];
  __shared__ int rotated;
  const int npair = (c + 1) / 2, ce = 2 * npair;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  double fro = 0.0;
  for (int t = threadIdx.x; t < c * c; t += blockDim.x) {
    const double w = R[t];
    W[t] = w;
    V[t] = t % c == t / c ? 1.0 : 0.0;
    fro += w * w;
  }
  const double weak2 = block_sum(fro, scratch) / c * null_share(c) * null_share(c);
  const double null2 = weak2 * null_share(c) * null_share(c);
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x == 0) rotated = 0;
    __syncthreads();
    for (int rr = 0; rr < ce - 1; ++rr) {
      for (int k = warp; k < npair; k += nw) {
        const int u = k - 1 - rr, v = ce - 2 - k - rr;   // positions k and ce - 1 - k, turned rr places
        int p = k == 0 ? 0 : 1 + (u < 0 ? u + ce - 1 : u), q = 1 + (v < 0 ? v + ce - 1 : v);
        if (p > q) { const int t = p; p = q; q = t; }
        if (q >= c) continue;
        double x[NE], y[NE], vx[NE], vy[NE];
        double a = 0.0, b = 0.0, g = 0.0;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
          const int i = lane + 32 * e;
          const bool in = i < c;
          x[e] = in ? W[i + p * c] : 0.0;
          y[e] = in ? W[i + q * c] : 0.0;
          vx[e] = in ? V[i + p * c] : 0.0;
          vy[e] = in ? V[i + q * c] : 0.0;
          a += x[e] * x[e];
          b += y[e] * y[e];
          g += x[e] * y[e];
        }
        a = warp_sum(a); b = warp_sum(b); g = warp_sum(g);
        if (fmin(a, b) <= null2) continue;
        const Rot t = decouple(false, a, g, b);
        if (t.s == 0.0) continue;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
          const int i = lane + 32 * e;
          if (i < c) {
            W[i + p * c] = t.c * x[e] - t.s * y[e];
            W[i + q * c] = t.s * x[e] + t.c * y[e];
            V[i + p * c] = t.c * vx[e] - t.s * vy[e];
            V[i + q * c] = t.s * vx[e] + t.c * vy[e];
          }
        }
        if (lane == 0 && !(fmin(a, b) <= weak2)) rotated = 1;
      }
      __syncthreads();
    }
    if (!rotated) break;
    __syncthreads();   // every thread has read the flag before it is cleared
  }
  for (int k = warp; k < c; k += nw) {
    double a = 0.0;
    for (int i = lane; i < c; i += 32) a += W[i + k * c] * W[i + k * c];
    a = warp_sum(a);
    if (lane == 0) norms[k] = sqrt(a);
  }
  __syncthreads();
  for (int k = warp; k < c; k += nw) {   // rank of column k, then its place in the outputs
    const double sk = norms[k], v = isnan(sk) ? -INFINITY : sk;
    int rank = 0;
    double top = -INFINITY;
    for (int j = lane; j < c; j += 32) {
      const double w = isnan(norms[j]) ? -INFINITY : norms[j];
      rank += (w > v) || (w == v && j < k);
      top = fmax(top, w);
    }
    rank = __reduce_add_sync(0xffffffffu, rank);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (lane == 0) s_out[rank] = sk;
    if (rank >= need) continue;
    const bool ok = sk > tol_rel * top && sk > 0.0;
    for (int i = lane; i < c; i += 32) {
      V_out[i + (size_t)rank * ldv] = V[i + k * c];
      RV_out[i + rank * c] = ok ? W[i + k * c] / sk : 0.0;
    }
  }
}

// More columns than kThinMax, or so few that the launches of the reduction are the
// time (kDirect below): W (r x c, r >= c) is overwritten in global memory, V (c x c)
// accumulates the rotations; one CTA, one warp a pair.
__global__ void __launch_bounds__(1024) jacobi_svd_kernel(int r, int c, double* W, double* V, int max_sweeps,
                                  double* U_out, int ldu, double* s_out, double* V_out, int ldv,
                                  int transpose_out) {
  extern __shared__ double sm[];
  const int npair = (c + 1) / 2;
  const int ce = 2 * npair;
  double* norms = sm;
  int* order = reinterpret_cast<int*>(sm + c);
  __shared__ int rotated;
  __shared__ double scratch0[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int t = threadIdx.x; t < c * c; t += blockDim.x) V[t] = (t % c == t / c) ? 1.0 : 0.0;
  __syncthreads();
  double weak2 = -1.0, null2 = -1.0;   // as in jacobi_core_kernel; four columns underflow in a few sweeps
  if (c > 4) {
    double fro = 0.0;
    for (int j = warp; j < c; j += nwarps)
      for (int i = lane; i < r; i += 32) fro += W[i + (size_t)j * r] * W[i + (size_t)j * r];
    weak2 = block_sum(fro, scratch0) / c * null_share(c) * null_share(c);
    null2 = weak2 * null_share(c) * null_share(c);
  }
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x == 0) rotated = 0;
    __syncthreads();
    for (int rr = 0; rr < ce - 1; ++rr) {
      for (int k = warp; k < npair; k += nwarps) {
        const int u = k - 1 - rr, v = ce - 2 - k - rr;
        int p = k == 0 ? 0 : 1 + (u < 0 ? u + ce - 1 : u), q = 1 + (v < 0 ? v + ce - 1 : v);
        if (p > q) { const int t = p; p = q; q = t; }
        if (q >= c) continue;
        double* wp = W + (size_t)p * r;
        double* wq = W + (size_t)q * r;
        double a = 0.0, b = 0.0, g = 0.0;
        for (int i = lane; i < r; i += 32) {
          const double x = wp[i], y = wq[i];
          a += x * x; b += y * y; g += x * y;
        }
        a = warp_sum(a); b = warp_sum(b); g = warp_sum(g);
        if (fmin(a, b) <= null2) continue;
        const Rot t = decouple(false, a, g, b);
        if (t.s != 0.0) {
          for (int i = lane; i < r; i += 32) {
            const double x = wp[i], y = wq[i];
            wp[i] = t.c * x - t.s * y;
            wq[i] = t.s * x + t.c * y;
          }
          for (int i = lane; i < c; i += 32) {
            const double x = V[i + (size_t)p * c], y = V[i + (size_t)q * c];
            V[i + (size_t)p * c] = t.c * x - t.s * y;
            V[i + (size_t)q * c] = t.s * x + t.c * y;
          }
          if (lane == 0 && !(fmin(a, b) <= weak2)) rotated = 1;
        }
      }
      __syncthreads();
    }
    if (!rotated) break;
    __syncthreads();
  }
  // Column norms and descending order.
  for (int k = warp; k < c; k += nwarps) {
    double a = 0.0;
    for (int i = lane; i < r; i += 32) a += W[i + (size_t)k * r] * W[i + (size_t)k * r];
    a = warp_sum(a);
    if (lane == 0) norms[k] = sqrt(a);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < c; i += blockDim.x) {
    const double v = isnan(norms[i]) ? -INFINITY : norms[i];
    int rank = 0;
    for (int j = 0; j < c; ++j) {
      const double w = isnan(norms[j]) ? -INFINITY : norms[j];
      rank += (w > v) || (w == v && j < i);
    }
    order[rank] = i;
  }
  __syncthreads();
  const double smax = norms[order[0]];
  const double tol = kEps * static_cast<double>(r > c ? r : c) * smax;
  // Output: U columns = W columns / s (completed when s is negligible).
  for (int j = 0; j < c; ++j) {
    const int src = order[j];
    const double sj = norms[src];
    double* uj = transpose_out ? V_out + (size_t)j * ldv : U_out + (size_t)j * ldu;
    double* vj = transpose_out ? U_out + (size_t)j * ldu : V_out + (size_t)j * ldv;
    if (threadIdx.x == 0) s_out[j] = sj;
    if (sj > tol && sj > 0.0) {
      for (int i = threadIdx.x; i < r; i += blockDim.x) uj[i] = W[i + (size_t)src * r] / sj;
      __syncthreads();
    } else {
      complete_null_column(r, j, transpose_out ? V_out : U_out, transpose_out ? ldv : ldu, scratch0);
    }
    for (int i = threadIdx.x; i < c; i += blockDim.x) vj[i] = V[i + (size_t)src * c];
    __syncthreads();
  }
}

__global__ void transpose_kernel(const double* __restrict__ A, int rows, int cols, int lda,
                                 double* __restrict__ B) {
  const size_t total = (size_t)rows * cols;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    const int i = static_cast<int>(t % rows), j = static_cast<int>(t / rows);
    B[j + (size_t)i * cols] = A[i + (size_t)j * lda];
  }
}

}  // namespace

void spd_solve(int k, const double* G, int ldg, int nrhs, const double* B, int ldb, double* X,
               int ldx, int* d_flag, double ridge_rel) {
  if (k <= 0 || nrhs <= 0) return;
  Context& ctx = Context::get();
  double* W = ctx.arena.alloc_n<double>((size_t)k * (k + nrhs));   // the factor, or the LU fallback's
  int* flag = d_flag ? d_flag : ctx.d_status + 1;
  if (k > kCholMax) {
    spd_solve_large_kernel<<<1, 512, 0, ctx.stream>>>(k, G, ldg, nrhs, B, ldb, X, ldx, W, flag, ridge_rel);
  } else {
    const int grid = std::min(ceil_div(nrhs, kCholGroups), 2 * ctx.sm_count);
    with_chol_size(k, [&](auto nr) {
      constexpr int NR = decltype(nr)::value;
      static const bool once = (allow_smem(spd_solve_kernel<NR>, chol_smem(NR)), true);
      (void)once;
      spd_solve_kernel<NR><<<grid, kCholThreads, chol_smem(NR), ctx.stream>>>(k, G, ldg, nrhs, B, ldb, X, ldx, W,
                                                                              flag, ridge_rel);
    });
  }
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

static void cgs2_orthonormalize(int rows, int cols, const double* Y, int ldy, double* Q, int ldq) {
  Context& ctx = Context::get();
  double* w = ctx.arena.alloc_n<double>(cols > 0 ? cols : 1);
  double* nrm = ctx.arena.alloc_n<double>(1);
  for (int j = 0; j < cols; ++j) {
    double* q = Q + (size_t)j * ldq;
    copy_matrix(q, rows, Y + (size_t)j * ldy, rows, rows, 1);
    for (int pass = 0; pass < 2 && j > 0; ++pass) {
      gemv(true, rows, j, 1.0, Q, ldq, q, 0.0, w);
      gemv(false, rows, j, -1.0, Q, ldq, w, 1.0, q);
    }
    dot_self_kernel<<<1, 512, 0, ctx.stream>>>(q, rows, nrm); ::fpls::note_launch();
    normalize_col_kernel<<<ceil_div(rows, 256), 256, 0, ctx.stream>>>(q, rows, nrm); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
  }
}

void qr_orthonormalize(int rows, int cols, const double* Y, int ldy, double* Q, int ldq) {
  if (cols <= 0 || rows <= 0) return;
  Context& ctx = Context::get();
  double* G = ctx.arena.alloc_n<double>((size_t)cols * cols);
  int* flag = ctx.d_status + 8;
  dzero(flag, sizeof(int));
  const double* src = Y;
  int lds = ldy;
  if (cols <= kCholMax) {
    for (int pass = 0; pass < 2; ++pass) {
      gemm(true, false, cols, cols, rows, 1.0, src, lds, src, lds, 0.0, G, cols);
      const int grid = std::min(ceil_div(rows, kCholGroups), 2 * ctx.sm_count);
      with_chol_size(cols, [&](auto nr) {
        constexpr int NR = decltype(nr)::value;
        static const bool once = (allow_smem(chol_qr_kernel<NR>, chol_smem(NR)), true);
        (void)once;
        chol_qr_kernel<NR><<<grid, kCholThreads, chol_smem(NR), ctx.stream>>>(cols, G, rows, src, lds, Q, ldq, flag);
      });
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      src = Q;
      lds = ldq;
    }
    int h = 0;
    FPLS_CUDA(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, ctx.stream));
    FPLS_CUDA(cudaStreamSynchronize(ctx.stream));
    if (h == 0) return;
  }
  cgs2_orthonormalize(rows, cols, Y, ldy, Q, ldq);
}

bool eig_sym_fits(int l) { return l <= kEigMax; }

void eig_sym_desc(int l, const double* G, int ldg, double* evals, double* V, int ldv) {
  if (l <= 0) return;
  FPLS_REQUIRE(eig_sym_fits(l), "eig_sym_desc: the matrix does not fit in shared memory");
  Context& ctx = Context::get();
  if (l <= kEigTiny) {
    const size_t smem = (2 * (size_t)l * l + 4 * (size_t)((l + 1) / 2)) * sizeof(double);
    jacobi_eig_tiny_kernel<<<1, 64, smem, ctx.stream>>>(l, G, ldg, evals, V, ldv, kEigSweeps);
    ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    return;
  }
  const int le = l + (l & 1), npair = le / 2;
  const size_t smem = 2 * (size_t)le * le * sizeof(double) + 2 * (size_t)npair * sizeof(Rot);
  // whole groups of four warps (one of each scheduler); the warp pair 0 and 4
  // is there from 65 on
  const int groups = std::min(kEigWarps / 4, std::max(npair > 32 ? 2 : 1, ceil_div(eig_blocks(npair), 96)));
  const int blocks = ceil_div(eig_blocks(npair), 96 * groups);
  auto kernel = blocks == 1 ? jacobi_eig_kernel<1> : blocks == 2 ? jacobi_eig_kernel<2> : jacobi_eig_kernel<kEigBlocks>;
  static bool attr_set = false;
  if (!attr_set) {
    FPLS_CUDA(cudaFuncSetAttribute(jacobi_eig_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    FPLS_CUDA(cudaFuncSetAttribute(jacobi_eig_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    FPLS_CUDA(cudaFuncSetAttribute(jacobi_eig_kernel<kEigBlocks>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    attr_set = true;
  }
  double2* log = ctx.arena.alloc_n<double2>((size_t)kEigSweeps * (le - 1) * npair);
  int* rank_of = ctx.arena.alloc_n<int>(l + 1);
  int* rounds = rank_of + l;
  kernel<<<1, 128 * groups, smem, ctx.stream>>>(l, G, ldg, evals, rank_of, log, rounds, kEigSweeps);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  const int grid = ceil_div(l, kApplyWarps);
  if (npair <= 32)
    jacobi_apply_log_kernel<1><<<grid, 32 * kApplyWarps, 0, ctx.stream>>>(l, log, rounds, rank_of, V, ldv);
  else
    jacobi_apply_log_kernel<2><<<grid, 32 * kApplyWarps, 0, ctx.stream>>>(l, log, rounds, rank_of, V, ldv);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

namespace {

// One level of the reduction: the reflectors of nb blocks of rb rows.
struct QrLevel {
  double *F, *tau;
  int rows, rb, nb;
};

// R of A (rows x c, lda) by blocks of rows until one block holds it all.
const double* reduce_to_triangle(const double* A, int rows, int c, int lda, std::vector<QrLevel>& levels) {
  Context& ctx = Context::get();
  const int rb_max = std::min(512, static_cast<int>((200 * 1024 / sizeof(double) - 2 * c) / c));
  static const bool once = (allow_smem(qr_block_kernel, 200 * 1024), true);
  (void)once;
  while (true) {
    // blocks of 256 rows (three times the columns, at least) keep the first pass on many SMs
    const int rb = rows <= rb_max ? rows : std::min(rb_max, std::max(256, 3 * c));
    const int nb = ceil_div(rows, rb);
    double* out = ctx.arena.alloc_n<double>((size_t)nb * c * c);
    const QrLevel level{ctx.arena.alloc_n<double>((size_t)rows * c), ctx.arena.alloc_n<double>((size_t)nb * c), rows, rb, nb};
    const size_t smem = ((size_t)rb * c + 2 * c) * sizeof(double);
    qr_block_kernel<<<nb, 512, smem, ctx.stream>>>(A, rows, c, lda, rb, out, nb * c, level.F, level.tau); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    levels.push_back(level);
    if (nb == 1) return out;
    A = out;
    rows = nb * c;
    lda = rows;
  }
}

// Z (rows x need, ldz) = Q Y for the Q of the levels, Y c x need.
void apply_reflectors(const std::vector<QrLevel>& levels, int c, const double* Y, int need, double* Z, int ldz) {
  Context& ctx = Context::get();
  static const bool once = (allow_smem(qr_apply_kernel<2>, 200 * 1024), allow_smem(qr_apply_kernel<8>, 200 * 1024),
                            allow_smem(qr_apply_kernel<16>, 200 * 1024), true);
  (void)once;
  int ldy = c;
  for (size_t l = levels.size(); l-- > 0;) {
    const QrLevel& q = levels[l];
    double* out = l == 0 ? Z : ctx.arena.alloc_n<double>((size_t)q.rows * need);
    const int ldo = l == 0 ? ldz : q.rows;
    const dim3 grid(q.nb, ceil_div(need, kApplyCols));
    auto kernel = q.rb <= 64 ? qr_apply_kernel<2> : q.rb <= 256 ? qr_apply_kernel<8> : qr_apply_kernel<16>;
    kernel<<<grid, 32 * kApplyCols, ((size_t)q.rb * c + c) * sizeof(double), ctx.stream>>>(q.F, q.tau, q.rows, c, q.rb, Y, ldy, need, out, ldo); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    Y = out;
    ldy = ldo;
  }
}

}  // namespace

void svd_thin(int rows, int cols, const double* A, int lda, double* U, int ldu, double* s,
              double* V, int ldv, int need) {
  if (rows <= 0 || cols <= 0) return;
  Context& ctx = Context::get();
  const bool tall = rows >= cols;
  const int r = tall ? rows : cols;
  const int c = tall ? cols : rows;
  const double* M = A;   // the tall form, r x c
  int ldm = lda;
  // up to four columns of little work a sweep in one launch, against four or six:
  // 2000 x 1: 10 against 25 us, 2000 x 2: 24 against 30, 4000 x 2: 37 against 30,
  // 512 x 4: 35 against 35
  constexpr int kDirect = 8192;
  const bool direct = c > kThinMax || (c <= 4 && (long long)r * c * c <= kDirect);
  double* W = nullptr;
  if (!tall || direct) {
    W = ctx.arena.alloc_n<double>((size_t)r * c);
    if (tall) {
      copy_matrix(W, r, A, lda, rows, cols);
    } else {
      transpose_kernel<<<256, 256, 0, ctx.stream>>>(A, rows, cols, lda, W); ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
    }
    M = W;
    ldm = r;
  }
  // tall: U (rows x c) is M's side, V (cols x c) the rotations.
  // wide: A^T = U' S V'^T, so U (rows x c) <- V', V (cols x c) <- U'.
  if (direct) {
    double* Vw = ctx.arena.alloc_n<double>((size_t)c * c);
    const size_t lists = (size_t)(c + (c + 1) / 2) * sizeof(double);
    jacobi_svd_kernel<<<1, 1024, lists, ctx.stream>>>(r, c, W, Vw, 60, U, ldu, s, V, ldv, tall ? 0 : 1);
    ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    return;
  }
  std::vector<QrLevel> levels;
  const double* R = reduce_to_triangle(M, r, c, ldm, levels);
  double* RV = ctx.arena.alloc_n<double>((size_t)c * need);
  double* left = tall ? U : V;    // M's side
  const int ldl = tall ? ldu : ldv;
  const size_t smem = (2 * (size_t)c * c + c) * sizeof(double);
  const int threads = 32 * std::min(32, std::max(4, (c + 1) / 2));
  auto core = c <= 32 ? jacobi_core_kernel<1> : c <= 64 ? jacobi_core_kernel<2> : jacobi_core_kernel<3>;
  static const bool once = (allow_smem(jacobi_core_kernel<1>, 160 * 1024), allow_smem(jacobi_core_kernel<2>, 160 * 1024),
                            allow_smem(jacobi_core_kernel<3>, 160 * 1024), true);
  (void)once;
  core<<<1, threads, smem, ctx.stream>>>(R, c, 60, kEps * static_cast<double>(r), need, s, tall ? V : U, tall ? ldv : ldu, RV);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  apply_reflectors(levels, c, RV, need, left, ldl);
  complete_null_columns(r, need, s, left, ldl);
}

}  // namespace fpls
