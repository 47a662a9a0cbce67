#include "blas_f64.cuh"
#include "context.cuh"
#include "gemv_f64.cuh"
#include "simpls_engine.cuh"

#include <algorithm>
#include <array>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>
#include <string>
#include <typeinfo>
#include <vector>

namespace fpls {
namespace {

// Threads a block.  The order of every sum is that of kSumThreads lanes (and
// kSumThreads / 32 warps), whatever the block: larger blocks only bring more
// loads in flight and more columns at a time.
constexpr int kMaxThreads = 1024;
constexpr int kSumThreads = 256;
constexpr int kSumWarps = kSumThreads / 32;
constexpr int kAhead = 16;    // loads of one thread that go out before they are used

struct Eng {
  int n, p, m, F, K, cp, cn, szp, szn;
  const double* Yg;
  const int* labels;
  const double* mY_all;
  const uint8_t* mask;
  const double* delta;
  const double* colsum;
  const double* colscale;
  const double* dY;
  double* S;
  const double* omega;
  int m1_mode;
  int iters;
  double* R;
  double* Q;
  double* V;
  double* tnorm;
  double* Tkeep;
  int* ncomp_done;
  int* status;
  // workspace
  double* y;       // F x p
  double* zA;      // F x cp x m
  double* zB;      // F x cp x m
  double* npart;   // F x cp
  double* r;       // F x p (unit r before the t normalisation)
  double* Rhat;    // p x F
  double* cpart;   // F x cp
  double* U;       // n x F
  double* T;       // n x F
  double* tpart;   // F x cn x 2
  double* qpart;   // F x cn x m
  double* P;       // p x F
  double* pv;      // F x p
  double* wpart;   // F x cp x K
  double* v;       // F x p
  double* vpart;   // F x cp
  double* vSpart;  // F x cp x m
  // U and P as partial sums of the products' ranges (Partials), added in order
  // where they are read: the separate reductions were 8 % of a grid's component
  double* upart;
  const double* ppart;
  int usplits, psplits;   // up to 1: U, P hold the sums
};

__device__ __forceinline__ void chunk_range(int chunk, int sz, int total, int& b, int& e) {
  b = chunk * sz;
  e = min(total, b + sz);
}

// parts[0] + parts[stride] + ... in order, kAhead loads at a time (each kernel of
// the loop starts with such a sum, and its loads one after another were a third
// of the launch).
__device__ __forceinline__ double sum_parts(const double* parts, int count, size_t stride) {
  double s = 0.0;
  for (int c0 = 0; c0 < count; c0 += kAhead) {
    double v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) v[u] = c0 + u < count ? parts[(c0 + u) * stride] : 0.0;
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (c0 + u < count) s += v[u];
  }
  return s;
}

// Block-wide sum of term(r) over r < rows, in kSumThreads lanes and warp order;
// all threads.
template <typename F>
__device__ __forceinline__ double chunk_sum(int rows, double* scratch, F term) {
  double s = 0.0;
  if (threadIdx.x < kSumThreads) {
    for (int r = threadIdx.x; r < rows; r += kSumThreads) s = term(r, s);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = s;
  }
  __syncthreads();
  double r = 0.0;
#pragma unroll
  for (int i = 0; i < kSumWarps; ++i) r += scratch[i];
  __syncthreads();
  return r;
}

constexpr int kMaxChunk = 4096;  // rows of a chunk staged in shared memory

// out[j * out_stride] = sum_{r < rows} M[r + j*ld] * xs[r] for j < ncols, with xs
// (the chunk's vector) in shared memory.  Warps take columns; when there are
// fewer columns than kSumWarps, several warps split the rows of one column.  Each
// lane streams consecutive rows, so every column read is coalesced, and takes
// the eight rows of a 256-row stretch at once: a column is one wait for memory,
// not one for each 64 rows (8000 x 100 in chunks of 250 rows: 19 us of a 45 us
// launch went there).
__device__ void chunk_dots(const double* M, size_t ld, int ncols,
                           const double* xs, int rows, double* out, int out_stride) {
  __shared__ double red[kSumWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (ncols >= kSumWarps) {
#pragma unroll 2
    for (int j = warp; j < ncols; j += blockDim.x >> 5) {
      const double* col = M + (size_t)j * ld;
      double a0 = 0.0, a1 = 0.0;
      for (int r0 = lane; r0 < rows; r0 += 256) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = r0 + 32 * u < rows ? col[r0 + 32 * u] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
          const int r = r0 + 32 * u;
          if (r + 32 < rows) {
            a0 += v[u] * xs[r];
            a1 += v[u + 1] * xs[r + 32];
          } else if (r < rows) {
            a0 += v[u] * xs[r];
          }
        }
      }
      const double acc = warp_sum(a0 + a1);
      if (lane == 0) out[(size_t)j * out_stride] = acc;
    }
    return;
  }
  const int g = kSumWarps / max(ncols, 1);   // warps per column
  const int j = warp / g, sub = warp % g;
  double acc = 0.0;
  if (warp < kSumWarps && j < ncols) {
    const double* col = M + (size_t)j * ld;
    for (int r0 = sub * 32 + lane; r0 < rows; r0 += 256 * g) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = r0 + 32 * g * u < rows ? col[r0 + 32 * g * u] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (r0 + 32 * g * u < rows) acc += v[u] * xs[r0 + 32 * g * u];
    }
  }
  acc = warp_sum(acc);
  if (lane == 0 && warp < kSumWarps) red[warp] = acc;
  __syncthreads();
  if (threadIdx.x < ncols) {
    double t = 0.0;
    for (int u = 0; u < g; ++u) t += red[threadIdx.x * g + u];
    out[(size_t)threadIdx.x * out_stride] = t;
  }
  __syncthreads();
}

// Partials of S_f^T y over the chunk (y staged in ys), or the chunk's ||y||^2.
__device__ __forceinline__ void chunk_StY(const Eng& e, int f, int chunk, const double* Sf,
                                          const double* ys, int b, int en, double* zout,
                                          bool norm_only) {
  if (norm_only) {
    __shared__ double scratch[32];
    const double s2 = chunk_sum(en - b, scratch, [&](int r, double s) { return s + ys[r] * ys[r]; });
    if (threadIdx.x == 0) e.npart[(size_t)f * e.cp + chunk] = s2;
    return;
  }
  chunk_dots(Sf + b, e.p, e.m, ys, en - b, zout + ((size_t)f * e.cp + chunk) * e.m, 1);
}

// First component's refresh start: y = Omega (or the single column of S).
__device__ __forceinline__ void refresh_start_chunk(const Eng& e, int f, int chunk, double* ys) {
  int b, en;
  chunk_range(chunk, e.szp, e.p, b, en);
  const double* Sf = e.S + (size_t)f * e.p * e.m;
  const double* y0 = e.m1_mode ? Sf : e.omega + (size_t)f * e.p;
  double* yf = e.y + (size_t)f * e.p;
  for (int i = b + threadIdx.x; i < en; i += blockDim.x) {
    yf[i] = y0[i];
    ys[i - b] = y0[i];
  }
  __syncthreads();
  chunk_StY(e, f, chunk, Sf, ys, b, en, e.zA, e.iters == 0);
}

__global__ void __launch_bounds__(kMaxThreads) k_refresh_start(Eng e) {
  __shared__ double vec[kMaxChunk];
  if (e.status[blockIdx.y]) return;
  refresh_start_chunk(e, blockIdx.y, blockIdx.x, vec);
}

// y <- S z with z = sum of the partials of S^T y; then the next partials (or ||y||^2).
__device__ __forceinline__ void refresh_apply_chunk(const Eng& e, const double* zin, double* zout, int last, int f, int chunk, double* zs, double* ys) {
  int b, en;
  chunk_range(chunk, e.szp, e.p, b, en);
  const double* Sf = e.S + (size_t)f * e.p * e.m;
  double* yf = e.y + (size_t)f * e.p;
  // the first columns of this thread's row are on their way while z is summed
  double v[kAhead];
  {
    const int i = b + threadIdx.x;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) v[u] = i < en && u < e.m ? Sf[i + (size_t)u * e.p] : 0.0;
  }
  for (int j = threadIdx.x; j < e.m; j += blockDim.x)
    zs[j] = sum_parts(zin + (size_t)f * e.cp * e.m + j, e.cp, e.m);
  __syncthreads();
  for (int i = b + threadIdx.x; i < en; i += blockDim.x) {
    double acc = 0.0;
    for (int j0 = 0; j0 < e.m; j0 += kAhead) {
      if (j0 > 0 || i >= b + (int)blockDim.x) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) v[u] = j0 + u < e.m ? Sf[i + (size_t)(j0 + u) * e.p] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (j0 + u < e.m) acc += v[u] * zs[j0 + u];
    }
    yf[i] = acc;
    ys[i - b] = acc;
  }
  __syncthreads();
  chunk_StY(e, f, chunk, Sf, ys, b, en, zout, last != 0);
}

__global__ void __launch_bounds__(kMaxThreads) k_refresh_apply(Eng e, const double* zin, double* zout, int last) {
  extern __shared__ double coef[];
  __shared__ double vec[kMaxChunk];
  if (e.status[blockIdx.y]) return;
  refresh_apply_chunk(e, zin, zout, last, blockIdx.y, blockIdx.x, coef, vec);
}

// r = -sign(y0) y / ||y|| (Householder QR of a single column; the 1 x m core
// SVD from gesvd keeps U = 1).  Rhat = colscale * r; cpart = delta . Rhat.
__device__ __forceinline__ void refresh_finish_chunk(const Eng& e, int f, int chunk, double* rhs, double* scratch) {
  int b, en;
  chunk_range(chunk, e.szp, e.p, b, en);
  const double nrm = sqrt(sum_parts(e.npart + (size_t)f * e.cp, e.cp, 1));
  if (!(nrm > 0.0) || !isfinite(nrm)) {
    // Degenerate refresh: the reference's refresh returns false and the loop stops.
    if (chunk == 0 && threadIdx.x == 0) e.status[f] = 1;
    return;
  }
  const double* yf = e.y + (size_t)f * e.p;
  const double sgn = (yf[0] >= 0.0) ? -1.0 : 1.0;
  const double* sc = e.colscale ? e.colscale + (size_t)f * e.p : nullptr;
  const double* dl = e.delta ? e.delta + (size_t)f * e.p : nullptr;
  for (int i = b + threadIdx.x; i < en; i += blockDim.x) {
    const double ri = sgn * yf[i] / nrm;
    e.r[(size_t)f * e.p + i] = ri;
    const double rh = sc ? ri * sc[i] : ri;
    e.Rhat[(size_t)f * e.p + i] = rh;
    rhs[i - b] = rh;
  }
  if (dl) {
    __syncthreads();
    const double c = chunk_sum(en - b, scratch, [&](int r, double s) { return s + dl[b + r] * rhs[r]; });
    if (threadIdx.x == 0) e.cpart[(size_t)f * e.cp + chunk] = c;
  }
}

__global__ void __launch_bounds__(kMaxThreads) k_refresh_finish(Eng e) {
  __shared__ double vec[kMaxChunk];
  __shared__ double scratch[32];
  if (e.status[blockIdx.y]) return;
  refresh_finish_chunk(e, blockIdx.y, blockIdx.x, vec, scratch);
}

// t = mask * (U - delta.rhat); partial sums of t^2, t and q = Y^T t (LABELS: Y is
// the one-hot matrix of e.labels).
template <bool LABELS>
__device__ __forceinline__ void scores_chunk(const Eng& e, int a, int f, int chunk, double* qs, double* ts, double* scratch) {
  int b, en;
  chunk_range(chunk, e.szn, e.n, b, en);
  const double c = e.delta ? sum_parts(e.cpart + (size_t)f * e.cp, e.cp, 1) : 0.0;
  const uint8_t* mk = e.mask ? e.mask + (size_t)f * e.n : nullptr;
  const double* Uf = e.U + (size_t)f * e.n;
  double* Tf = e.T + (size_t)f * e.n;
  double* keep = e.Tkeep ? e.Tkeep + ((size_t)f * e.K + a) * e.n : nullptr;
  if (LABELS) {
    for (int j = threadIdx.x; j < e.m; j += blockDim.x) qs[j] = 0.0;
    __syncthreads();
  }
  for (int i = b + threadIdx.x; i < en; i += blockDim.x) {
    const double u = (e.usplits > 1 ? sum_parts(e.upart + (size_t)f * e.n + i, e.usplits, (size_t)e.n * e.F) : Uf[i]) - c;
    const double t = (mk && !mk[i]) ? 0.0 : u;
    Tf[i] = t;
    ts[i - b] = t;
    if (keep) keep[i] = u;
    if (LABELS && t != 0.0) atomicAdd(&qs[e.labels[i]], t);
  }
  __syncthreads();
  const double s2 = chunk_sum(en - b, scratch, [&](int r, double s) { return s + ts[r] * ts[r]; });
  const double s1 = chunk_sum(en - b, scratch, [&](int r, double s) { return s + ts[r]; });
  if (threadIdx.x == 0) {
    e.tpart[((size_t)f * e.cn + chunk) * 2 + 0] = s2;
    e.tpart[((size_t)f * e.cn + chunk) * 2 + 1] = s1;
  }
  double* qp = e.qpart + ((size_t)f * e.cn + chunk) * e.m;
  if (LABELS) {
    for (int j = threadIdx.x; j < e.m; j += blockDim.x) qp[j] = qs[j];
  } else {
    chunk_dots(e.Yg + b, e.n, e.m, ts, en - b, qp, 1);
  }
}

template <bool LABELS>
__global__ void __launch_bounds__(LABELS ? kSumThreads : kMaxThreads) k_scores(Eng e, int a) {
  extern __shared__ double coef[];
  __shared__ double vec[kMaxChunk];
  __shared__ double scratch[32];
  if (e.status[blockIdx.y]) return;
  scores_chunk<LABELS>(e, a, blockIdx.y, blockIdx.x, coef, vec, scratch);
}

__device__ __forceinline__ void t_stats(const Eng& e, int f, double& tn, double& st) {
  const double2* tp = reinterpret_cast<const double2*>(e.tpart) + (size_t)f * e.cn;
  double s2 = 0.0, s1 = 0.0;
  for (int c0 = 0; c0 < e.cn; c0 += kAhead / 2) {
    double2 v[kAhead / 2];
#pragma unroll
    for (int u = 0; u < kAhead / 2; ++u) v[u] = c0 + u < e.cn ? tp[c0 + u] : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < kAhead / 2; ++u) {
      if (c0 + u < e.cn) {
        s2 += v[u].x;
        s1 += v[u].y;
      }
    }
  }
  tn = sqrt(s2);
  st = s1;
}

// p = colscale * (P - delta * sum(t)) / ||t||; partial w = V^T p.
__device__ __forceinline__ void loading_chunk(const Eng& e, int a, int f, int chunk, double* ps) {
  int b, en;
  chunk_range(chunk, e.szp, e.p, b, en);
  const double* Pf = e.P + (size_t)f * e.p;
  auto p_at = [&](int i) {
    return e.psplits > 1 ? sum_parts(e.ppart + (size_t)f * e.p + i, e.psplits, (size_t)e.p * e.F) : Pf[i];
  };
  const double p0 = b + (int)threadIdx.x < en ? p_at(b + threadIdx.x) : 0.0;   // on its way during the sums
  double tn, st;
  t_stats(e, f, tn, st);
  if (!(tn > 0.0) || !isfinite(tn)) {
    if (chunk == 0 && threadIdx.x == 0) e.status[f] = 1;
    return;
  }
  const double* sc = e.colscale ? e.colscale + (size_t)f * e.p : nullptr;
  const double* dl = e.delta ? e.delta + (size_t)f * e.p : nullptr;
  double* pf = e.pv + (size_t)f * e.p;
  for (int i = b + threadIdx.x; i < en; i += blockDim.x) {
    double v = i < b + (int)blockDim.x ? p0 : p_at(i);
    if (dl) v -= dl[i] * st;
    if (sc) v *= sc[i];
    v /= tn;
    pf[i] = v;
    ps[i - b] = v;
  }
  __syncthreads();
  if (a > 0)
    chunk_dots(e.V + (size_t)f * e.p * e.K + b, e.p, a, ps, en - b,
               e.wpart + ((size_t)f * e.cp + chunk) * e.K, 1);
}

__global__ void __launch_bounds__(kMaxThreads) k_loading(Eng e, int a) {
  __shared__ double vec[kMaxChunk];
  if (e.status[blockIdx.y]) return;
  loading_chunk(e, a, blockIdx.y, blockIdx.x, vec);
}

// v = p - V (V^T p); partials of ||v||^2 and of S^T v.
__device__ __forceinline__ void orth_chunk(const Eng& e, int a, int f, int chunk, double* ws, double* vsh, double* scratch) {
  int b, en;
  chunk_range(chunk, e.szp, e.p, b, en);
  const double* Vf = e.V + (size_t)f * e.p * e.K;
  const double* pf = e.pv + (size_t)f * e.p;
  double* vf = e.v + (size_t)f * e.p;
  // this thread's row is on its way while w is summed
  double v[kAhead], x0 = 0.0;
  {
    const int i = b + threadIdx.x;
    if (i < en) x0 = pf[i];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) v[u] = i < en && u < a ? Vf[i + (size_t)u * e.p] : 0.0;
  }
  for (int l = threadIdx.x; l < a; l += blockDim.x)
    ws[l] = sum_parts(e.wpart + (size_t)f * e.cp * e.K + l, e.cp, e.K);
  __syncthreads();
  for (int i = b + threadIdx.x; i < en; i += blockDim.x) {
    const bool first = i < b + (int)blockDim.x;
    double x = first ? x0 : pf[i];
    for (int l0 = 0; l0 < a; l0 += kAhead) {
      if (l0 > 0 || !first) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) v[u] = l0 + u < a ? Vf[i + (size_t)(l0 + u) * e.p] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kAhead; u += 4) {
        const int l = l0 + u;
        const double v0 = v[u], v1 = v[u + 1], v2 = v[u + 2], v3 = v[u + 3];
        if (l + 4 <= a) {
          x -= v0 * ws[l] + v1 * ws[l + 1] + v2 * ws[l + 2] + v3 * ws[l + 3];
        } else {   // the last one to three columns one by one
          if (l < a) x -= v0 * ws[l];
          if (l + 1 < a) x -= v1 * ws[l + 1];
          if (l + 2 < a) x -= v2 * ws[l + 2];
        }
      }
    }
    vf[i] = x;
    vsh[i - b] = x;
  }
  __syncthreads();
  const double s2 = chunk_sum(en - b, scratch, [&](int r, double s) { return s + vsh[r] * vsh[r]; });
  if (threadIdx.x == 0) e.vpart[(size_t)f * e.cp + chunk] = s2;
  // S^T v (unnormalised) for the deflation.
  chunk_dots(e.S + (size_t)f * e.p * e.m + b, e.p, e.m, vsh, en - b,
             e.vSpart + ((size_t)f * e.cp + chunk) * e.m, 1);
}

__global__ void __launch_bounds__(kMaxThreads) k_orth(Eng e, int a) {
  extern __shared__ double coef[];
  __shared__ double vec[kMaxChunk];
  __shared__ double scratch[32];
  if (e.status[blockIdx.y]) return;
  orth_chunk(e, a, blockIdx.y, blockIdx.x, coef, vec, scratch);
}

// v /= ||v||; V[:, a] = v; S -= v (v^T S); R[:, a] = r / ||t||; Q[:, a] = q / ||t||;
// then the next component's refresh start (partials of S^T r_a over the
// deflated S, or ||S[:,0]||^2 when m == 1).
__device__ __forceinline__ void deflate_chunk(const Eng& e, int a, int next, int f, int chunk, double* vs, double* ysh) {
  int b, en;
  chunk_range(chunk, e.szp, e.p, b, en);
  double* Sf = e.S + (size_t)f * e.p * e.m;
  double* vf = e.v + (size_t)f * e.p;
  double* Vcol = e.V + ((size_t)f * e.K + a) * e.p;
  double* Rcol = e.R + ((size_t)f * e.K + a) * e.p;
  const double* rf = e.r + (size_t)f * e.p;
  double* yf = e.y + (size_t)f * e.p;
  // The rows' own values are on their way while the partials are summed: v and r
  // of row threadIdx.x, and the first eight columns of S that this thread updates
  // (one column group for each kSumThreads).
  const int group = threadIdx.x / kSumThreads, groups = blockDim.x / kSumThreads;
  const int i0 = b + threadIdx.x, s0 = b + threadIdx.x % kSumThreads;
  const double v0 = i0 < en ? vf[i0] : 0.0, r0 = i0 < en ? rf[i0] : 0.0;
  double x[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) x[u] = s0 < en && 8 * group + u < e.m ? Sf[s0 + (size_t)(8 * group + u) * e.p] : 0.0;
  for (int j = threadIdx.x; j < e.m; j += blockDim.x) vs[j] = sum_parts(e.vSpart + (size_t)f * e.cp * e.m + j, e.cp, e.m);
  double tn, st;
  t_stats(e, f, tn, st);
  const double vn = sqrt(sum_parts(e.vpart + (size_t)f * e.cp, e.cp, 1));
  if (!(vn > 0.0) || !isfinite(vn)) {
    if (chunk == 0 && threadIdx.x == 0) e.status[f] = 1;
    return;
  }
  for (int j = threadIdx.x; j < e.m; j += blockDim.x) vs[j] /= vn;
  for (int i = i0; i < en; i += blockDim.x) {
    const double vi = (i == i0 ? v0 : vf[i]) / vn;
    vf[i] = vi;
    Vcol[i] = vi;
    ysh[i - b] = vi;
  }
  __syncthreads();
  // the rank-1 update, elementwise, eight columns of a row loaded before any is stored
  for (int i = s0; i < en; i += kSumThreads) {
    const double vi = ysh[i - b];
    for (int j0 = 8 * group; j0 < e.m; j0 += 8 * groups) {
      if (i > s0 || j0 > 8 * group) {
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = j0 + u < e.m ? Sf[i + (size_t)(j0 + u) * e.p] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (j0 + u < e.m) Sf[i + (size_t)(j0 + u) * e.p] = x[u] - vi * vs[j0 + u];
    }
  }
  __syncthreads();
  for (int i = i0; i < en; i += blockDim.x) {
    const double ri = (i == i0 ? r0 : rf[i]) / tn;
    Rcol[i] = ri;
    if (next) {
      const double y0 = e.m1_mode ? Sf[i] : ri;
      yf[i] = y0;
      ysh[i - b] = y0;
    }
  }
  if (chunk == 0) {
    double* Qcol = e.Q + ((size_t)f * e.K + a) * e.m;
    for (int j = threadIdx.x; j < e.m; j += blockDim.x) {
      double q = sum_parts(e.qpart + (size_t)f * e.cn * e.m + j, e.cn, e.m);
      double off = 0.0;
      if (e.labels) off += e.mY_all[j];
      if (e.dY) off += e.dY[(size_t)f * e.m + j];
      q -= off * st;
      Qcol[j] = q / tn;
    }
    if (threadIdx.x == 0) {
      e.tnorm[(size_t)f * e.K + a] = tn;
      e.ncomp_done[f] = a + 1;
    }
  }
  if (next) {
    __syncthreads();
    chunk_StY(e, f, chunk, Sf, ysh, b, en, e.zA, e.iters == 0);
  }
}

__global__ void __launch_bounds__(kMaxThreads) k_deflate(Eng e, int a, int next) {
  extern __shared__ double coef[];
  __shared__ double vec[kMaxChunk];
  if (e.status[blockIdx.y]) return;
  deflate_chunk(e, a, next, blockIdx.y, blockIdx.x, coef, vec);
}

// ---- The same bodies on a chunk of S in shared memory ---------------------------
// The bodies above are bound by what they wait for in L2 and by their address
// arithmetic.  These take a chunk of at most kTile rows whose S lies in shared
// memory with that pitch, rows past the chunk zero: every offset is an immediate,
// no load needs a bound, and each sum keeps the order of the body above it (a
// zero row adds +0), so the results are the same bit for bit.  Sums of partials
// that every block needs are loaded by one warp together instead of by every
// thread in turn.
constexpr int kTile = 256;
constexpr int kTileStage = 1280;   // doubles staged at a time
struct __align__(16) TileShared {   // stage is read as double2 too
  double x[kTile];       // the phase's vector: p, v, y
  double pv[kTile], v[kTile];
  double stage[kTileStage];
  double red[32];
  double norm[kSumWarps];   // tile_norm's own: tile_dots follows it without a barrier
  double tn, st, nrm;
};

// s[0] + s[step] + ... (n of them) in order.
__device__ __forceinline__ double in_order(const double* s, int n, int step) {
  double t = 0.0;
  int i = 0;
  for (; i + 8 <= n; i += 8)
#pragma unroll
    for (int u = 0; u < 8; ++u) t += s[(i + u) * step];
  for (; i < n; ++i) t += s[i * step];
  return t;
}

// One warp: the sum of `count` values in order, in every lane.
__device__ __forceinline__ double warp_parts(const double* parts, int count, double* stage) {
  const int lane = threadIdx.x & 31;
  double t = 0.0;
  for (int c0 = 0; c0 < count; c0 += 512) {
    const int n = min(512, count - c0);
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = lane + 32 * u < n ? parts[c0 + lane + 32 * u] : 0.0;
#pragma unroll
    for (int u = 0; u < 16; ++u)
      if (lane + 32 * u < n) stage[lane + 32 * u] = v[u];
    __syncwarp();
    for (int i = 0; i < n; ++i) t += stage[i];
    __syncwarp();
  }
  return t;
}

// out[j] = parts[j] + parts[j + stride] + ... (`count` of them, in order) for
// j < ncols: groups of threads take kAhead partials of every column each, so that
// all loads are in flight at once, and add them in turn.  Ends with a barrier.
template <int NT>
__device__ __forceinline__ void column_sums(double* out, const double* parts, int ncols, int count, int stride) {
  int shift = 5;
  while ((1 << shift) < ncols && (1 << shift) < NT) ++shift;
  const int width = 1 << shift, groups = NT >> shift, g = threadIdx.x >> shift, j0 = threadIdx.x & (width - 1);
  for (int j = j0; j - j0 < ncols; j += width) {
    for (int c0 = 0; c0 < count; c0 += groups * kAhead) {
      const int c = c0 + g * kAhead;
      const double* src = parts + j + (size_t)c * stride;
      double v[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        v[u] = j < ncols && c + u < count ? *src : 0.0;
        src += stride;
      }
      const int turns = min(groups, (count - c0 + kAhead - 1) / kAhead);
      for (int t = 0; t < turns; ++t) {
        if (t == g && j < ncols) {
          double s = c > 0 ? out[j] : 0.0;
#pragma unroll
          for (int u = 0; u < kAhead; ++u)
            if (c + u < count) s += v[u];
          out[j] = s;
        }
        __syncthreads();
      }
    }
  }
}

// out[j] = sum_r M[r + j ld] x[r] in the order of chunk_dots, for j < ncols.  M in
// shared memory with zero rows (BOUND: in memory, rows read up to `rows` only).
template <int NT, bool BOUND>
__device__ __forceinline__ void tile_dots(const double* M, int ld, int ncols, TileShared& sh, int rows, double* out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (ncols >= kSumWarps) {
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = sh.x[lane + 32 * u];
#pragma unroll 2
    for (int j = warp; j < ncols; j += NT / 32) {
      const double* col = M + (size_t)j * ld + lane;
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = !BOUND || lane + 32 * u < rows ? col[32 * u] : 0.0;
      double a0 = 0.0, a1 = 0.0;
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        a0 += v[u] * x[u];
        a1 += v[u + 1] * x[u + 1];
      }
      const double acc = warp_sum(a0 + a1);
      if (lane == 0) out[j] = acc;
    }
    return;
  }
  const int g = kSumWarps / max(ncols, 1);   // warps per column
  const int j = warp / g, sub = warp - j * g;
  if (warp < kSumWarps && j < ncols) {
    const double* col = M + (size_t)j * ld;
    double acc = 0.0;
    for (int r = sub * 32 + lane; r < kTile; r += 32 * g) {
      const double v = !BOUND || r < rows ? col[r] : 0.0;
      acc += v * sh.x[r];
    }
    acc = warp_sum(acc);
    if (lane == 0) sh.red[warp] = acc;
  }
  __syncthreads();
  if (threadIdx.x < ncols) {
    double t = 0.0;
    for (int u = 0; u < g; ++u) t += sh.red[threadIdx.x * g + u];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

// Sum of x[r]^2 in chunk_sum's order, by the first kSumWarps warps; thread 0 stores
// it, after the last barrier: sh.norm may be written again behind a later one only.
__device__ __forceinline__ void tile_norm(TileShared& sh, double* out) {
  if (threadIdx.x < kTile) {
    const double x = sh.x[threadIdx.x];
    const double s = warp_sum(x * x);
    if ((threadIdx.x & 31) == 0) sh.norm[threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < kSumWarps; ++i) t += sh.norm[i];
    *out = t;
  }
}

// Where a chunk lies: its rows b .. b + rows of the p, its S and V.
struct TileView {
  int b, rows;
  double* S;          // shared, pitch kTile
  const double* V;    // row b of V: shared with pitch kTile, or memory with pitch p
  int ldv;
};

template <int NT, bool VMEM>
__device__ __forceinline__ void tile_loading(const Eng& e, const TileView& w, int a, int f, int chunk, TileShared& sh) {
  const int row = threadIdx.x & (kTile - 1), i = w.b + row;
  const bool mine = threadIdx.x < kTile && row < w.rows;
  double P = 0.0;
  if (threadIdx.x >= NT - 32) {   // the last warp: ||t|| and sum(t)
    const int lane = threadIdx.x & 31;
    const double2* tp = reinterpret_cast<const double2*>(e.tpart) + (size_t)f * e.cn;
    double2* st = reinterpret_cast<double2*>(sh.stage);
    double s2 = 0.0, s1 = 0.0;
    for (int c0 = 0; c0 < e.cn; c0 += 256) {
      const int n = min(256, e.cn - c0);
      double2 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = lane + 32 * u < n ? tp[c0 + lane + 32 * u] : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (lane + 32 * u < n) st[lane + 32 * u] = v[u];
      __syncwarp();
#pragma unroll 4
      for (int c = 0; c < n; ++c) {
        s2 += st[c].x;
        s1 += st[c].y;
      }
      __syncwarp();
    }
    if (lane == 0) {
      sh.tn = sqrt(s2);
      sh.st = s1;
    }
  }
  if (mine)
    P = e.psplits > 1 ? sum_parts(e.ppart + (size_t)f * e.p + i, e.psplits, (size_t)e.p * e.F) : e.P[(size_t)f * e.p + i];
  __syncthreads();
  const double tn = sh.tn, st = sh.st;
  if (!(tn > 0.0) || !isfinite(tn)) {
    if (chunk == 0 && threadIdx.x == 0) e.status[f] = 1;
    return;
  }
  if (threadIdx.x < kTile) {
    double v = 0.0;
    if (mine) {
      v = P;
      if (e.delta) v -= e.delta[(size_t)f * e.p + i] * st;
      if (e.colscale) v *= e.colscale[(size_t)f * e.p + i];
      v /= tn;
    }
    sh.pv[row] = v;
    sh.x[row] = v;
  }
  __syncthreads();
  if (a > 0) tile_dots<NT, VMEM>(w.V, VMEM ? w.ldv : kTile, a, sh, w.rows, e.wpart + ((size_t)f * e.cp + chunk) * e.K);
}

template <int NT, bool VMEM>
__device__ __forceinline__ void tile_orth(const Eng& e, const TileView& w, int a, int f, int chunk, double* ws,
                                          TileShared& sh) {
  // Row r is thread r of every group of kTile threads: the groups take the columns
  // of V four at a time in turn (a quad's sum of products is formed where its
  // columns arrive) and the first group subtracts the quads' sums in order.
  constexpr int groups = NT / kTile;
  const int g = threadIdx.x / kTile, row = threadIdx.x % kTile;
  const int quads = a / 4;
  const int ld = VMEM ? w.ldv : kTile;
  const bool in = !VMEM || row < w.rows;
  const double* Vr = w.V + row;
  double x = g == 0 ? sh.pv[row] : 0.0;
  bool summed = false;
  for (int q0 = 0; q0 < quads || q0 == 0; q0 += 4 * groups) {
    double v[4][4];
    const double* col = Vr + (size_t)(4 * (q0 + g)) * ld;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool have = in && q0 + g + u * groups < quads;
#pragma unroll
      for (int c = 0; c < 4; ++c) v[u][c] = have ? col[(size_t)c * ld] : 0.0;
      col += (size_t)(4 * groups) * ld;
    }
    if (!summed) {   // w, while the first columns are on their way
      if (a > 0) column_sums<NT>(ws, e.wpart + (size_t)f * e.cp * e.K, a, e.cp, e.K);
      summed = true;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int qu = q0 + u * groups;   // group 0's quad of this turn
      if (qu >= quads) break;
      const int q = qu + g, l = 4 * q;
      double t = 0.0;
      if (q < quads) t = v[u][0] * ws[l] + v[u][1] * ws[l + 1] + v[u][2] * ws[l + 2] + v[u][3] * ws[l + 3];
      if (groups == 1) {
        x -= t;
      } else {
        sh.stage[threadIdx.x] = t;
        __syncthreads();
        if (g == 0) {
#pragma unroll
          for (int h = 0; h < groups; ++h)
            if (qu + h < quads) x -= sh.stage[h * kTile + row];
        }
        __syncthreads();
      }
    }
  }
  if (g == 0) {
    for (int l = 4 * quads; l < a; ++l)   // the last one to three columns
      if (in) x -= Vr[(size_t)l * ld] * ws[l];
    sh.v[row] = x;
    sh.x[row] = x;
  }
  __syncthreads();
  tile_norm(sh, e.vpart + (size_t)f * e.cp + chunk);
  // S^T v (unnormalised) for the deflation
  tile_dots<NT, false>(w.S, kTile, e.m, sh, w.rows, e.vSpart + ((size_t)f * e.cp + chunk) * e.m);
}

// Partials of S^T x, or ||x||^2 (x in sh.x).
template <int NT>
__device__ __forceinline__ void tile_StY(const Eng& e, const TileView& w, int f, int chunk, TileShared& sh, double* zout,
                                         bool norm_only) {
  if (norm_only) tile_norm(sh, e.npart + (size_t)f * e.cp + chunk);
  else tile_dots<NT, false>(w.S, kTile, e.m, sh, w.rows, zout + ((size_t)f * e.cp + chunk) * e.m);
}

// Vsh: V in shared memory (null: only memory's); Sg: memory's S, row b (null: not kept).
template <int NT>
__device__ __forceinline__ void tile_deflate(const Eng& e, const TileView& w, int a, int next, int f, int chunk, double* vs,
                                             TileShared& sh, double* Vsh, double* Sg) {
  constexpr int groups = NT / kTile;
  const int g = threadIdx.x / kTile, row = threadIdx.x % kTile, i = w.b + row;
  const bool in = row < w.rows;
  const double r0 = g == 0 && in ? e.r[(size_t)f * e.p + i] : 0.0;
  column_sums<NT>(vs, e.vSpart + (size_t)f * e.cp * e.m, e.m, e.cp, e.m);
  if (threadIdx.x >= NT - 32) {
    const double s = warp_parts(e.vpart + (size_t)f * e.cp, e.cp, sh.stage);
    if ((threadIdx.x & 31) == 0) sh.nrm = sqrt(s);
  }
  __syncthreads();
  const double vn = sh.nrm, tn = sh.tn, st = sh.st;
  if (!(vn > 0.0) || !isfinite(vn)) {
    if (chunk == 0 && threadIdx.x == 0) e.status[f] = 1;
    return;
  }
  for (int j = threadIdx.x; j < e.m; j += NT) vs[j] /= vn;
  if (g == 0) {
    const double vi = sh.v[row] / vn;   // 0 past the chunk
    sh.v[row] = vi;
    if (Vsh) Vsh[a * kTile + row] = vi;
    else if (in) e.V[((size_t)f * e.K + a) * e.p + i] = vi;
  }
  __syncthreads();
  {   // the rank-1 update, elementwise
    const double vi = sh.v[row];
    double* col = w.S + row + g * kTile;
    if (Sg) {
      double* mem = Sg + row + (size_t)g * e.p;
#pragma unroll 4
      for (int j = g; j < e.m; j += groups) {
        const double s = *col - vi * vs[j];
        *col = s;
        if (in) *mem = s;
        col += groups * kTile;
        mem += (size_t)groups * e.p;
      }
    } else {
#pragma unroll 4
      for (int j = g; j < e.m; j += groups) {
        *col = *col - vi * vs[j];
        col += groups * kTile;
      }
    }
  }
  __syncthreads();
  if (g == 0) {
    const double ri = r0 / tn;
    if (in) e.R[((size_t)f * e.K + a) * e.p + i] = ri;
    if (next) {
      const double y0 = e.m1_mode ? w.S[row] : ri;
      if (in) e.y[(size_t)f * e.p + i] = y0;
      sh.x[row] = in ? y0 : 0.0;
    }
  }
  // q: chunk c takes responses c, c + cp, ..., a thread a partial
  {
    double* Qcol = e.Q + ((size_t)f * e.K + a) * e.m;
    const int cols = e.m > chunk ? (e.m - chunk + e.cp - 1) / e.cp : 0;   // of this chunk
    const int fit = e.cn <= kTileStage ? kTileStage / e.cn : 0;           // columns staged at a time
    for (int c0 = 0; c0 < cols; c0 += max(fit, 1)) {
      const int nc = min(max(fit, 1), cols - c0);
      for (int t = threadIdx.x; fit > 0 && t < nc * e.cn; t += NT) {
        const int c = t / e.cn;
        sh.stage[t] = e.qpart[((size_t)f * e.cn + (t - c * e.cn)) * e.m + chunk + (c0 + c) * e.cp];
      }
      __syncthreads();
      for (int c = threadIdx.x; c < nc; c += NT) {
        const int j = chunk + (c0 + c) * e.cp;
        double q = fit > 0 ? in_order(sh.stage + c * e.cn, e.cn, 1)
                           : sum_parts(e.qpart + (size_t)f * e.cn * e.m + j, e.cn, e.m);
        double off = 0.0;
        if (e.labels) off += e.mY_all[j];
        if (e.dY) off += e.dY[(size_t)f * e.m + j];
        q -= off * st;
        Qcol[j] = q / tn;
      }
      __syncthreads();
    }
    if (chunk == 0 && threadIdx.x == 0) {
      e.tnorm[(size_t)f * e.K + a] = tn;
      e.ncomp_done[f] = a + 1;
    }
  }
  if (next) {
    __syncthreads();
    tile_StY<NT>(e, w, f, chunk, sh, e.zA, e.iters == 0);
  }
}

template <int NT>
__device__ __forceinline__ void tile_start(const Eng& e, const TileView& w, int f, int chunk, TileShared& sh) {
  if (threadIdx.x < kTile) {
    const int row = threadIdx.x, i = w.b + row;
    double y = 0.0;
    if (row < w.rows) {
      y = e.m1_mode ? w.S[row] : e.omega[(size_t)f * e.p + i];
      e.y[(size_t)f * e.p + i] = y;
    }
    sh.x[row] = y;
  }
  __syncthreads();
  tile_StY<NT>(e, w, f, chunk, sh, e.zA, e.iters == 0);
}

template <int NT>
__device__ __forceinline__ void tile_apply(const Eng& e, const TileView& w, const double* zin, double* zout, int last, int f,
                                           int chunk, double* zs, TileShared& sh) {
  column_sums<NT>(zs, zin + (size_t)f * e.cp * e.m, e.m, e.cp, e.m);
  if (threadIdx.x < kTile) {
    const int row = threadIdx.x;
    const double* s = w.S + row;
    double acc = 0.0;
    int j = 0;
    for (; j + 8 <= e.m; j += 8, s += 8 * kTile)
#pragma unroll
      for (int u = 0; u < 8; ++u) acc += s[u * kTile] * zs[j + u];
    for (; j < e.m; ++j, s += kTile) acc += *s * zs[j];
    if (row < w.rows) e.y[(size_t)f * e.p + w.b + row] = acc;
    sh.x[row] = acc;   // 0 past the chunk
  }
  __syncthreads();
  tile_StY<NT>(e, w, f, chunk, sh, zout, last != 0);
}

// The chunk's S into shared memory, asynchronously, rows past the chunk zero;
// tile_here() before it is read.
template <int NT>
__device__ __forceinline__ void tile_load(double* S, const double* src, size_t ld, int m, int rows) {
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(S));
  const int row = threadIdx.x % kTile;
  for (int j = threadIdx.x / kTile; j < m; j += NT / kTile) {
    if (row < rows)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8u * static_cast<uint32_t>(j * kTile + row)),
                   "l"(src + row + (size_t)j * ld)
                   : "memory");
    else S[j * kTile + row] = 0.0;
  }
}

__device__ __forceinline__ void tile_here() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// ---- The component loop of one small fit in one launch -----------------------
// A fit of a few hundred samples spends its time between kernels: eleven launches
// a component, 5.2 us each inside a graph, for phases that move a few hundred
// kilobytes of L2.  Here the phases are the bodies above (sums in the same
// order: the results are those of the launches bit for bit) with a grid barrier
// between them, eight a component: the split sums of X r and the normalisation of
// r are folded into the phases that read them, and a block keeps its chunk of S
// and V in shared memory.  400 x 2000, 5 responses: 57 us a component as a graph
// of launches, 36 us now (1.2 us a barrier, about 3 us a phase).
struct LoopArgs {
  Eng e;
  const double* X;    // n x p
  GemvRanges xr;      // ranges of X r
  int coef_len;       // doubles of dynamic shared memory before the vector
  int vec_len;        // and of the vector
  unsigned* barrier;  // zero at the start
  unsigned* stop;     // barrier after which a stopped fit leaves (all ones: none)
  int* fail;          // a barrier wait gave up
  int* host_fail;     // the same for the host (mapped)
};

// Threads of a block: a chunk has 250 rows or so, and more warps only add issue
// slots spent on predicated-off loads (1024 threads: 48 us a component).
constexpr int kLoopThreads = 256;
constexpr int kLoopWarps = kLoopThreads / 32;
constexpr size_t kLoopSmem = 208 * 1024;   // beside the static arrays
// Looks at a counter before a wait gives up: some seconds of a running grid.  Looks,
// not clock cycles: a grid whose GPU is lent to another process for a while goes on
// afterwards.
constexpr int kBarrierLooks = 1 << 23;

// `count` CTAs in all have arrived at *counter (CTAs of one cooperative launch);
// false when a wait ran out, in every thread of every CTA sooner or later.
__device__ bool counted_barrier(unsigned* counter, unsigned count, int* fail, int* host_fail) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(counter, 1u);
    ok = 1;
    for (int looks = 0;; ++looks) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
      if (seen >= count) break;
      if (*(volatile int*)fail || looks > kBarrierLooks) {
        atomicExch(fail, 1);
        *(volatile int*)host_fail = 1;
        ok = 0;
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

__global__ void __launch_bounds__(kLoopThreads) simpls_loop_kernel(LoopArgs g) {
  extern __shared__ double coef[];   // max(m, K), a score chunk's vector, the X tile, S, V
  __shared__ double scratch[32];
  __shared__ TileShared sh;
  double* vec = coef + g.coef_len;
  const Eng& e = g.e;
  unsigned arrived = 0;
  // The block's own chunk of S and V (a chunk a block) stays in shared memory for
  // the whole loop: what a phase waits for in L2 is other blocks' partials only.
  double* tile = vec + g.vec_len;              // [256][32]
  TileView w{0, 0, tile + 256 * 32, nullptr, kTile};
  double* Vsh = w.S + (size_t)e.m * kTile;
  w.V = Vsh;
  const int own = blockIdx.x;
  if (own < e.cp) {
    int en;
    chunk_range(own, e.szp, e.p, w.b, en);
    w.rows = en - w.b;
    tile_load<kLoopThreads>(w.S, e.S + w.b, e.p, e.m, w.rows);
    tile_here();
  }
  // A phase over `count` chunks; false: leave (a wait gave up, or the fit stopped).
  // Block 0 has chunk 0, which raises the status: it names the barrier that ends
  // this phase, so that a block still on its way from the one before does not
  // leave early.
  auto phase = [&](int count, auto body) {
    for (int c = blockIdx.x; c < count; c += gridDim.x) {
      body(c);
      __syncthreads();   // the next chunk reuses the shared arrays
    }
    ++arrived;
    if (blockIdx.x == 0 && threadIdx.x == 0 && e.status[0] != 0) *(volatile unsigned*)g.stop = arrived;
    if (!counted_barrier(g.barrier, arrived * gridDim.x, g.fail, g.host_fail)) return false;
    return *(volatile unsigned*)g.stop > arrived;
  };
  if (!phase(e.cp, [&](int c) { tile_start<kLoopThreads>(e, w, 0, c, sh); })) return;
  for (int a = 0; a < e.K; ++a) {
    double *zin = e.zA, *zout = e.zB;
    for (int it = 0; it < e.iters; ++it) {
      const int last = it == e.iters - 1 ? 1 : 0;
      if (!phase(e.cp, [&](int c) { tile_apply<kLoopThreads>(e, w, zin, zout, last, 0, c, coef, sh); })) return;
      double* t = zin;
      zin = zout;
      zout = t;
    }
    // r = +-y / ||y|| and X r: an item is 32 rows of one column range.  Its X tile
    // comes in by all threads at once (one wait for L2, 148 SMs sharing X); one
    // warp then takes the rows' chains, 256 dependent multiply-adds each at most.
    {
      const double nrm = sqrt(sum_parts(e.npart, e.cp, 1));
      if (!(nrm > 0.0) || !isfinite(nrm)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) e.status[0] = 1;
      } else {
        const double sgn = (e.y[0] >= 0.0) ? -1.0 : 1.0;
        const int row_groups = (e.n + 31) / 32, items = row_groups * g.xr.splits;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (int i = w.b + threadIdx.x; i < w.b + w.rows; i += blockDim.x) e.r[i] = sgn * e.y[i] / nrm;
        for (int item = blockIdx.x; item < items; item += gridDim.x) {
          const int rg = item % row_groups, z = item / row_groups, row = 32 * rg + lane;
          const int kbeg = z * g.xr.kps, kend = min(e.p, kbeg + g.xr.kps);
          double acc = 0.0;
          for (int kc = kbeg; kc < kend; kc += 256) {
            const int kn = min(256, kend - kc);
            double x[256 / kLoopWarps];
#pragma unroll
            for (int u = 0; u < 256 / kLoopWarps; ++u) {
              const int k = warp + kLoopWarps * u;
              x[u] = k < kn && row < e.n ? __ldg(g.X + row + (size_t)(kc + k) * e.n) : 0.0;
            }
            if (threadIdx.x < kn) {
              const double r = sgn * e.y[kc + threadIdx.x] / nrm;
              vec[threadIdx.x] = r;
            }
#pragma unroll
            for (int u = 0; u < 256 / kLoopWarps; ++u) tile[(warp + kLoopWarps * u) * 32 + lane] = x[u];
            __syncthreads();
            if (warp == 0) {
#pragma unroll 8
              for (int k = 0; k < kn; ++k) acc = fma(tile[k * 32 + lane], vec[k], acc);
            }
            __syncthreads();
          }
          if (warp == 0 && row < e.n) {
            if (e.usplits > 1) e.upart[(size_t)z * e.n + row] = acc;
            else e.U[row] = acc;
          }
        }
      }
    }
    if (!phase(0, [](int) {})) return;
    if (!phase(e.cn, [&](int c) { scores_chunk<false>(e, a, 0, c, coef, vec, scratch); })) return;
    for (int j = blockIdx.x * (kLoopThreads / 32) + (threadIdx.x >> 5); j < e.p; j += gridDim.x * (kLoopThreads / 32)) {
      const double acc = gemv_column<32>(g.X + (size_t)j * e.n, e.T, e.n);
      if ((threadIdx.x & 31) == 0) e.P[j] = acc;
    }
    if (!phase(0, [](int) {})) return;
    if (!phase(e.cp, [&](int c) { tile_loading<kLoopThreads, false>(e, w, a, 0, c, sh); })) return;
    if (!phase(e.cp, [&](int c) { tile_orth<kLoopThreads, false>(e, w, a, 0, c, coef, sh); })) return;
    if (!phase(e.cp, [&](int c) { tile_deflate<kLoopThreads>(e, w, a, a + 1 < e.K ? 1 : 0, 0, c, coef, sh, Vsh, nullptr); }))
      return;
  }
}

// ---- From X^T t to the next r in one launch ------------------------------------
// A larger fit, or a batch of fits, runs its two products as kernels of their
// own; the phases between them (loading, orthogonalisation, deflation, the next
// component's refresh) work on chunks of S that fit shared memory.  One launch
// takes all of them: block (chunk, fit) loads its chunk of S once, the phases are
// the chunk bodies above (sums in the same order: the results are those of the
// separate launches bit for bit), and S is written back as it is deflated.  The
// chunks of one fit meet between the phases: up to eight of them are a thread
// block cluster and meet at its barrier, whatever the number of fits; more of them
// need all blocks resident (a cooperative launch) and count arrivals in memory.
// Bound by the latency of the phases' chains of sums and, at a few microseconds a
// phase, by the instructions of a warp (a first form that called the bodies on
// memory's layout executed four times as many and took as long as the launches).
// A component's phases: 30 fits of 501 x 5, 2 chunks each: 50 -> 33 us; 8000 x
// 100, 32 chunks: 105 -> 54 us; 1000 x 100, 4 chunks: 114 -> 57 us.
constexpr int kClusterChunks = 8;
constexpr size_t kUpdateSmem = 208 * 1024;   // dynamic, beside the static arrays
struct UpdateArgs {
  int coef_len;       // doubles before the chunk of S
  unsigned arrived;   // barriers of the earlier launches of this fit
  unsigned* counter;  // arrivals, 32 apart by fit (counted form)
  // Where a stopped fit leaves, 32 apart (all ones: nowhere): 2 b at barrier b, 2 b + 1
  // at the end of the launch whose last barrier was b.  A launch begins on what earlier
  // launches wrote here, never on the status, which chunk 0 may set before another block
  // has started: that block would leave without arriving at the first barrier.
  unsigned* stop;
  int* fail;
  int* host_fail;
};

// a: the component whose X^T t is in P, or -1 for the first refresh; next: refresh follows.
template <int THREADS, bool CLUSTER>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 2 : 1) k_update(Eng e, UpdateArgs g, int a, int next) {
  extern __shared__ double coef[];   // max(m, K), then the chunk of S
  __shared__ TileShared sh;
  const int f = blockIdx.y, chunk = blockIdx.x;
  if (*(volatile unsigned*)(g.stop + 32 * f) <= 2 * g.arrived + 1) return;
  int b, en;
  chunk_range(chunk, e.szp, e.p, b, en);
  double* Sg = e.S + (size_t)f * e.p * e.m + b;
  const TileView w{b, en - b, coef + g.coef_len, e.V + (size_t)f * e.p * e.K + b, e.p};
  tile_load<THREADS>(w.S, Sg, e.p, e.m, w.rows);
  unsigned arrived = g.arrived;
  // all chunks of the fit have finished the phase; false: the fit stopped, or a wait
  // gave up.  Every thread of the fit decides alike, however late it reads: a value
  // from a later phase is larger.
  auto meet = [&]() {
    ++arrived;
    if (!CLUSTER) __syncthreads();
    if (chunk == 0 && threadIdx.x == 0 && e.status[f] != 0) *(volatile unsigned*)(g.stop + 32 * f) = 2 * arrived;
    if (CLUSTER) {
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else if (!counted_barrier(g.counter + 32 * f, arrived * gridDim.x, g.fail, g.host_fail)) {
      return false;
    }
    return *(volatile unsigned*)(g.stop + 32 * f) > 2 * arrived;
  };
  if (a >= 0) {
    tile_loading<THREADS, true>(e, w, a, f, chunk, sh);
    tile_here();
    if (!meet()) return;
    tile_orth<THREADS, true>(e, w, a, f, chunk, coef, sh);
    if (!meet()) return;
    tile_deflate<THREADS>(e, w, a, next, f, chunk, coef, sh, nullptr, Sg);
    if (!next) return;
  } else {
    tile_here();
    tile_start<THREADS>(e, w, f, chunk, sh);
  }
  if (!meet()) return;
  double *zin = e.zA, *zout = e.zB;
  for (int it = 0; it < e.iters; ++it) {
    tile_apply<THREADS>(e, w, zin, zout, it == e.iters - 1 ? 1 : 0, f, chunk, coef, sh);
    if (!meet()) return;
    double* t = zin;
    zin = zout;
    zout = t;
  }
  // r = -sign(y0) y / ||y||, Rhat and delta . Rhat as refresh_finish_chunk
  if (threadIdx.x >= THREADS - 32) {
    const double s = warp_parts(e.npart + (size_t)f * e.cp, e.cp, sh.stage);
    if ((threadIdx.x & 31) == 0) sh.nrm = sqrt(s);
  }
  const int row = threadIdx.x;
  const double* yf = e.y + (size_t)f * e.p;
  const bool mine = row < w.rows;
  const double y0 = yf[0], y = mine ? yf[b + row] : 0.0;
  __syncthreads();
  const double nrm = sh.nrm;
  if (!(nrm > 0.0) || !isfinite(nrm)) {
    if (chunk == 0 && threadIdx.x == 0) {
      e.status[f] = 1;
      *(volatile unsigned*)(g.stop + 32 * f) = 2 * arrived + 1;
    }
    return;
  }
  const double sgn = y0 >= 0.0 ? -1.0 : 1.0;
  const size_t at = (size_t)f * e.p + b + row;
  double rh = 0.0;
  if (mine) {
    const double ri = sgn * y / nrm;
    e.r[at] = ri;
    rh = e.colscale ? ri * e.colscale[at] : ri;
    e.Rhat[at] = rh;
  }
  if (e.delta) {
    double s = 0.0;
    if (mine) s = s + e.delta[at] * rh;
    s = warp_sum(s);
    if ((row & 31) == 0) sh.red[row >> 5] = s;
    __syncthreads();
    if (row == 0) {
      double t = 0.0;
#pragma unroll
      for (int i = 0; i < kSumWarps; ++i) t += sh.red[i];
      e.cpart[(size_t)f * e.cp + chunk] = t;
    }
  }
}

// What the driver may refuse: a grid that has to be resident, or a cluster (another
// process's share of the GPU, a partition of it).  FASTPLS_TEST_REFUSE_FROM=k (tests
// only): from the k-th such launch of a fit on, none is made.
bool launch_accepted(const cudaLaunchConfig_t& cfg, const void* kernel, void** args, int& made) {
  const char* from = std::getenv("FASTPLS_TEST_REFUSE_FROM");
  if (from && from[0] && made >= std::atoi(from)) return false;
  if (cudaLaunchKernelExC(&cfg, kernel, args) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  ++made;
  ::fpls::note_launch();
  return true;
}

// The launch of k_update for one engine: which kernel, and its shared memory.
struct UpdateLaunch {
  const void* kernel = nullptr;   // null: separate launches
  bool cluster = false;
  dim3 grid;
  int threads = 0;
  size_t smem = 0;
  UpdateArgs args{};
  int made = 0;

  // False, with nothing done, when the driver refuses it: separate launches from here
  // on (S, V, R and the vectors between the phases are theirs in memory).
  bool run(const Eng& e, int a, int next, cudaStream_t st) {
    if (!kernel) return false;
    args.arrived = a < 0 ? 0u : (unsigned)(1 + e.iters) + (unsigned)a * (3 + e.iters);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    if (cluster) {
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = grid.x;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
    } else {
      at[0].id = cudaLaunchAttributeCooperative;
      at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    Eng ec = e;
    void* argv[] = {&ec, &args, &a, &next};
    if (!launch_accepted(cfg, kernel, argv, made)) kernel = nullptr;
    return kernel != nullptr;
  }
};

template <int THREADS>
const void* update_kernel(bool cluster) {
  static const bool once = [] {
    FPLS_CUDA(cudaFuncSetAttribute(k_update<THREADS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kUpdateSmem));
    FPLS_CUDA(cudaFuncSetAttribute(k_update<THREADS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kUpdateSmem));
    return true;
  }();
  (void)once;
  return cluster ? (const void*)k_update<THREADS, true> : (const void*)k_update<THREADS, false>;
}

__global__ void k_masked_response(Eng e, double* M) {
  const size_t total = (size_t)e.n * e.F * e.m;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    const int i = static_cast<int>(t % e.n);
    const size_t col = t / e.n;
    const int f = static_cast<int>(col / e.m), j = static_cast<int>(col % e.m);
    const bool in = !e.mask || e.mask[(size_t)f * e.n + i];
    double v = 0.0;
    if (in) v = e.labels ? (e.labels[i] == j ? 1.0 : 0.0) : e.Yg[i + (size_t)j * e.n];
    M[t] = v;
  }
}

__global__ void k_crosscov_finish(Eng e, const double* P) {
  const size_t total = (size_t)e.F * e.p * e.m;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    const int i = static_cast<int>(t % e.p);
    const size_t col = t / e.p;
    const int f = static_cast<int>(col / e.m), j = static_cast<int>(col % e.m);
    double v = P[i + col * e.p];
    if (e.colsum) {
      double off = 0.0;
      if (e.labels) off += e.mY_all[j];
      if (e.dY) off += e.dY[(size_t)f * e.m + j];
      v -= e.colsum[(size_t)f * e.p + i] * off;
    }
    if (e.colscale) v *= e.colscale[(size_t)f * e.p + i];
    e.S[(size_t)f * e.p * e.m + i + (size_t)j * e.p] = v;
  }
}

// Row-sharded fits: after X^T T, the loading P (p x F), the score sums
// (t^T t, sum t: F x 2) and Y^T t (F x m) are rank-local partial sums.  Pack
// folds the row-chunk partials in chunk order into one buffer [P | t | q];
// after the all-reduce, unpack puts the totals in chunk 0 (the other chunks
// zero), so the kernels that follow read sums over all ranks' rows.
__global__ void k_shard_pack(Eng e, double* __restrict__ red) {
  const size_t np = (size_t)e.F * e.p, nt = (size_t)e.F * 2, nq = (size_t)e.F * e.m;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < np + nt + nq;
       i += (size_t)gridDim.x * blockDim.x) {
    if (i < np) {
      red[i] = e.P[i];
    } else if (i < np + nt) {
      const size_t k = i - np, f = k / 2, c2 = k % 2;
      double s = 0.0;
      for (int c = 0; c < e.cn; ++c) s += e.tpart[(f * e.cn + c) * 2 + c2];
      red[i] = s;
    } else {
      const size_t k = i - np - nt, f = k / e.m, j = k % e.m;
      double s = 0.0;
      for (int c = 0; c < e.cn; ++c) s += e.qpart[(f * e.cn + c) * e.m + j];
      red[i] = s;
    }
  }
}

__global__ void k_shard_unpack(Eng e, const double* __restrict__ red) {
  const size_t np = (size_t)e.F * e.p, nt = (size_t)e.F * e.cn * 2, nq = (size_t)e.F * e.cn * e.m;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < np + nt + nq;
       i += (size_t)gridDim.x * blockDim.x) {
    if (i < np) {
      e.P[i] = red[i];
    } else if (i < np + nt) {
      const size_t k = i - np, f = k / (2 * (size_t)e.cn), c = (k / 2) % e.cn, c2 = k % 2;
      e.tpart[k] = c == 0 ? red[np + f * 2 + c2] : 0.0;
    } else {
      const size_t k = i - np - nt, f = k / ((size_t)e.cn * e.m), c = (k / e.m) % e.cn, j = k % e.m;
      e.qpart[k] = c == 0 ? red[np + (size_t)e.F * 2 + f * e.m + j] : 0.0;
    }
  }
}

Eng make_eng(const SimplsBatch& b) {
  Eng e{};
  e.n = b.n; e.p = b.p; e.m = b.m; e.F = b.F; e.K = b.K;
  const int target = 4 * Context::get().sm_count;
  e.cp = std::max(1, std::min(ceil_div(target, b.F), ceil_div(b.p, 256)));
  e.cp = std::max(e.cp, ceil_div(b.p, kMaxChunk));
  e.szp = ceil_div(b.p, e.cp);
  e.cp = ceil_div(b.p, e.szp);
  e.cn = std::max(1, std::min(ceil_div(target, b.F), ceil_div(b.n, 256)));
  e.cn = std::max(e.cn, ceil_div(b.n, kMaxChunk));
  e.szn = ceil_div(b.n, e.cn);
  e.cn = ceil_div(b.n, e.szn);
  e.Yg = b.Yg; e.labels = b.labels; e.mY_all = b.mY_all; e.mask = b.mask; e.delta = b.delta;
  e.colsum = b.colsum;
  e.colscale = b.colscale; e.dY = b.dY; e.S = b.S; e.omega = b.omega; e.m1_mode = b.m1_mode;
  e.iters = b.m1_mode ? 0 : std::max(b.power_iters, 0);
  e.R = b.R; e.Q = b.Q; e.V = b.V; e.tnorm = b.tnorm; e.Tkeep = b.Tkeep;
  e.ncomp_done = b.ncomp_done; e.status = b.status;
  return e;
}

}  // namespace

void XOperatorF64::times(const double* Rhat, int F, double* U) {
  if (F == 1) gemv(false, n, p, 1.0, Xc, n, Rhat, 0.0, U);
  else gemm(false, false, n, F, p, 1.0, Xc, n, Rhat, p, 0.0, U, n);
}

void XOperatorF64::t_times(const double* T, int F, double* P) {
  if (F == 1) gemv_t_ranged(n, p, Xc, n, T, P);
  else gemm(true, false, p, F, n, 1.0, Xc, n, T, n, 0.0, P, p);
}

Partials XOperatorF64::times_partials(const double* Rhat, int F, double* U) {
  if (F == 1) return gemv_partials(n, p, Xc, n, Rhat, U);
  return gemm_partials(false, false, n, F, p, Xc, n, Rhat, p, U);
}

Partials XOperatorF64::t_times_partials(const double* T, int F, double* P) {
  if (F == 1) return gemv_t_partials(n, p, Xc, n, T, P);
  return gemm_partials(true, false, p, F, n, Xc, n, T, n, P);
}

void XOperatorF64::gram(double* K) { gram_f64(Xc, n, p, n, K, n); }

void simpls_batch_crosscov(const SimplsBatch& b, const double* /*Xc*/, const int* /*n_train*/) {
  Context& ctx = Context::get();
  Eng e = make_eng(b);
  double* M = ctx.arena.alloc_n<double>((size_t)b.n * b.F * b.m);
  double* P = ctx.arena.alloc_n<double>((size_t)b.p * b.F * b.m);
  k_masked_response<<<8 * ctx.sm_count, 256, 0, ctx.stream>>>(e, M); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  b.X->t_times(M, b.F * b.m, P);
  k_crosscov_finish<<<8 * ctx.sm_count, 256, 0, ctx.stream>>>(e, P); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

namespace {

// FASTPLS_LOOP_GRAPH=0 enqueues the component loop launch by launch.
bool simpls_graph_enabled() {
  static const int v = [] {
    const char* e = std::getenv("FASTPLS_LOOP_GRAPH");
    return e ? (e[0] != '0' ? 1 : 0) : 1;
  }();
  return v != 0;
}

// Shapes whose component loop has run once launch by launch: its GEMM plans,
// split-K workspace and arena blocks exist, so a later call of the shape enqueues
// launches only and can be captured.
std::set<std::array<long long, 9>>& simpls_seen() {
  static std::set<std::array<long long, 9>> seen;
  return seen;
}

// The executable graph of the last captured component loop; each call captures
// its loop and updates it in place when the topology matches, else
// instantiates a new one (launches already in flight are not affected).
cudaGraphExec_t g_simpls_exec = nullptr;

// Returns false, with nothing enqueued, when the loop could not be captured
// (a host step of the loop that a capture does not allow, such as the first
// allocation of a GEMM plan); the caller then runs the loop launch by launch.
template <typename Loop>
bool simpls_launch_as_graph(cudaStream_t st, Loop&& loop) {
  FPLS_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  cudaGraph_t graph = nullptr;
  try {
    loop();
  } catch (...) {
    cudaStreamEndCapture(st, &graph);
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    return false;
  }
  if (cudaStreamEndCapture(st, &graph) != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    return false;
  }
  bool updated = false;
  if (g_simpls_exec) {
    cudaGraphExecUpdateResultInfo info;
    updated = cudaGraphExecUpdate(g_simpls_exec, graph, &info) == cudaSuccess;
    if (!updated) {
      cudaGetLastError();
      cudaGraphExecDestroy(g_simpls_exec);
      g_simpls_exec = nullptr;
    }
  }
  cudaError_t e = cudaSuccess;
  if (!updated) e = cudaGraphInstantiate(&g_simpls_exec, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) {
    g_simpls_exec = nullptr;
    FPLS_CUDA(e);
  }
  FPLS_CUDA(cudaGraphLaunch(g_simpls_exec, st));
  return true;
}

}  // namespace

void simpls_release_graph() {
  if (g_simpls_exec) cudaGraphExecDestroy(g_simpls_exec);
  g_simpls_exec = nullptr;
  simpls_seen().clear();
}

void simpls_batch_run(const SimplsBatch& b) {
  Context& ctx = Context::get();
  Eng e = make_eng(b);
  Arena& ar = ctx.arena;
  const size_t F = b.F;
  e.y = ar.alloc_n<double>(F * b.p);
  e.zA = ar.alloc_n<double>(F * e.cp * b.m);
  e.zB = ar.alloc_n<double>(F * e.cp * b.m);
  e.npart = ar.alloc_n<double>(F * e.cp);
  e.r = ar.alloc_n<double>(F * b.p);
  e.Rhat = ar.alloc_n<double>(F * b.p);
  e.cpart = ar.alloc_n<double>(F * e.cp);
  e.U = ar.alloc_n<double>(F * b.n);
  e.T = ar.alloc_n<double>(F * b.n);
  e.tpart = ar.alloc_n<double>(F * e.cn * 2);
  e.qpart = ar.alloc_n<double>(F * e.cn * b.m);
  e.P = ar.alloc_n<double>(F * b.p);
  e.pv = ar.alloc_n<double>(F * b.p);
  e.wpart = ar.alloc_n<double>(F * e.cp * std::max(b.K, 1));
  e.v = ar.alloc_n<double>(F * b.p);
  e.vpart = ar.alloc_n<double>(F * e.cp);
  e.vSpart = ar.alloc_n<double>(F * e.cp * b.m);
  dzero(b.status, F * sizeof(int));
  dzero(b.ncomp_done, F * sizeof(int));
  dzero(b.R, F * b.p * b.K * sizeof(double));
  dzero(b.Q, F * b.m * b.K * sizeof(double));
  dzero(b.V, F * b.p * b.K * sizeof(double));
  dzero(b.tnorm, F * b.K * sizeof(double));
  const dim3 gp(e.cp, b.F), gn(e.cn, b.F);
  // Four warp columns at a time for every block of columns a kernel multiplies:
  // 256 threads up to 32 columns (60 fits of a grid fill the SMs with blocks as
  // it is, and 1024-thread ones took 35 us instead of 10 for their class scores),
  // then 512, then 1024.
  auto block = [](int cols) { return cols <= 32 ? 256 : cols <= 64 ? 512 : kMaxThreads; };
  const int tm = block(b.m), tq = b.labels ? kSumThreads : tm;
  constexpr int kThreads = 256;   // elementwise kernels
  // all-reduce buffer of a row-sharded fit: [P (F x p) | t^T t, sum t (F x 2) | Y^T t (F x m)]
  const size_t shard_count = sharded() ? F * ((size_t)b.p + 2 + b.m) : 0;
  double* shard_red = shard_count ? ar.alloc_n<double>(shard_count) : nullptr;
  const unsigned shard_grid =
      shard_count ? (unsigned)std::min<size_t>(ceil_div(F * ((size_t)b.p + e.cn * (2 + (size_t)b.m)), kThreads),
                                               (size_t)ctx.sm_count * 8)
                  : 1u;
  const size_t sm_m = std::max<size_t>(b.m, 1) * sizeof(double);
  const size_t sm_k = std::max<size_t>(b.K, 1) * sizeof(double);
  cudaStream_t st = ctx.stream;
  // Optional per-phase device timing (FASTPLS_TRACE=1), printed to stderr.
  const char* trace_env = std::getenv("FASTPLS_TRACE");
  const bool trace = trace_env && trace_env[0] == '1';
  std::vector<std::pair<const char*, cudaEvent_t>> marks;
  auto mark = [&](const char* name) {
    if (!trace) return;
    cudaEvent_t ev;
    FPLS_CUDA(cudaEventCreate(&ev));
    FPLS_CUDA(cudaEventRecord(ev, st));
    marks.emplace_back(name, ev);
  };
  mark("start");
  // One small fit on its own: the whole loop in one launch (not while a trace or
  // the profiler times the kernels, nor for row-sharded fits, whose all-reduce is
  // the caller's).  Above 4 M matrix elements the products are the time and have
  // more loads in flight as kernels of their own.
  auto* op64 = dynamic_cast<XOperatorF64*>(b.X);
  const int coef_len = std::max(std::max(b.m, 1), std::max(b.K, 1));
  const int vec_len = std::max(e.szn, kTile);
  const size_t loop_smem = (coef_len + vec_len + 256 * 32 + (size_t)kTile * (b.m + b.K)) * sizeof(double);
  if (simpls_graph_enabled() && !trace && !ctx.profile && !shard_red && op64 && b.F == 1 && !b.labels && !b.mask &&
      !b.delta && !b.colscale && !b.dY && (size_t)b.n * b.p <= ((size_t)1 << 22) && e.cp <= ctx.sm_count && e.szp <= kTile &&
      loop_smem <= kLoopSmem) {
    LoopArgs g;
    g.xr = gemv_ranges(b.n, b.p, ctx.sm_count);
    e.usplits = g.xr.splits;
    e.upart = e.usplits > 1 ? ar.alloc_n<double>((size_t)e.usplits * b.n) : nullptr;
    g.e = e;
    g.X = op64->Xc;
    unsigned* ctl = ar.alloc_n<unsigned>(128);   // each on a line of its own
    dzero(ctl, 64 * sizeof(unsigned));
    FPLS_CUDA(cudaMemsetAsync(ctl + 64, 0xff, sizeof(unsigned), st));
    g.barrier = ctl;
    g.fail = reinterpret_cast<int*>(ctl + 32);
    g.stop = ctl + 64;
    g.host_fail = ctx.host_fail;
    g.coef_len = coef_len;
    g.vec_len = vec_len;
    const int want = std::max({e.cp, e.cn, ceil_div(b.n, 32) * g.xr.splits, ceil_div(b.p, kLoopWarps)});
    static const bool once = [] {
      FPLS_CUDA(cudaFuncSetAttribute(simpls_loop_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLoopSmem));
      return true;
    }();
    (void)once;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(std::max(want, e.cp), ctx.sm_count));
    cfg.blockDim = dim3(kLoopThreads);
    cfg.dynamicSmemBytes = loop_smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void* args[] = {&g};
    int made = 0;
    // a wait that gave up ends the call with an error (Context::end_call)
    if (launch_accepted(cfg, (const void*)simpls_loop_kernel, args, made)) return;
  }
  // The phases between the products in one launch, where a chunk's S fits shared
  // memory and the chunks form a cluster or are all resident (the count of blocks
  // an SM holds decides); else (wide responses, or many fits of many chunks) as
  // launches of their own.
  UpdateLaunch up;
  {
    up.cluster = e.cp <= kClusterChunks;
    // few columns give a warp one or two, and 60 fits of a grid fill the SMs
    up.threads = std::max(b.m, b.K) <= 32 ? 256 : 512;
    up.grid = gp;
    up.args.coef_len = coef_len;
    up.smem = (coef_len + (size_t)b.m * kTile) * sizeof(double);
    const void* k = up.threads == 256 ? update_kernel<256>(up.cluster) : update_kernel<512>(up.cluster);
    bool fits = e.szp <= kTile && up.smem <= kUpdateSmem;
    if (fits && !up.cluster) {
      int per_sm = 0;
      FPLS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, up.threads, up.smem));
      fits = (long long)e.cp * b.F <= (long long)per_sm * ctx.sm_count;
    }
    if (fits) {
      up.kernel = k;
      unsigned* ctl = ar.alloc_n<unsigned>(32 * (2 * F + 1));   // each on a line of its own
      FPLS_CUDA(cudaMemsetAsync(ctl, 0xff, 32 * F * sizeof(unsigned), st));
      up.args.stop = ctl;
      if (!up.cluster) {
        FPLS_CUDA(cudaMemsetAsync(ctl + 32 * F, 0, 32 * (F + 1) * sizeof(unsigned), st));
        up.args.counter = ctl + 32 * F;
        up.args.fail = reinterpret_cast<int*>(ctl + 32 * 2 * F);
        up.args.host_fail = ctx.host_fail;
      }
    }
  }
  // The component loop as one CUDA graph once its shape has run (not while a
  // trace or the kernel-class profiler records events, nor for row-sharded
  // fits, whose all-reduce callback is the caller's).
  const std::array<long long, 9> key{b.F, b.n, b.p, b.m, b.K, e.iters, b.labels ? 1 : 0, ctx.precision,
                                     static_cast<long long>(typeid(*b.X).hash_code())};
  const bool eligible = simpls_graph_enabled() && !trace && !ctx.profile && !shard_red;
  const bool graph = eligible && simpls_seen().count(key) > 0;
  auto loop = [&]() {
  bool refreshed = up.run(e, -1, 1, st);
  if (!refreshed) {
    k_refresh_start<<<gp, tm, 0, st>>>(e); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
  }
  for (int a = 0; a < b.K; ++a) {
    if (!refreshed) {
      // Refresh: y <- S (S^T y) `iters` times from the warm start, then normalise.
      double* zin = e.zA;
      double* zout = e.zB;
      for (int it = 0; it < e.iters; ++it) {
        const int last = (it == e.iters - 1) ? 1 : 0;
        k_refresh_apply<<<gp, tm, sm_m, st>>>(e, zin, zout, last); ::fpls::note_launch();
        FPLS_CHECK_LAUNCH();
        std::swap(zin, zout);
      }
      k_refresh_finish<<<gp, kThreads, 0, st>>>(e); ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      mark("refresh");
    }
    const Partials xr = b.X->times_partials(e.Rhat, b.F, e.U);
    e.upart = const_cast<double*>(xr.w);
    e.usplits = xr.splits;
    mark("X*R");
    if (b.labels) k_scores<true><<<gn, tq, sm_m, st>>>(e, a);
    else k_scores<false><<<gn, tq, 0, st>>>(e, a);
    ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    mark("scores");
    if (shard_red) {
      b.X->t_times(e.T, b.F, e.P);   // the all-reduce takes the sums
    } else {
      const Partials pp = b.X->t_times_partials(e.T, b.F, e.P);
      e.ppart = pp.w;
      e.psplits = pp.splits;
    }
    if (shard_red) {
      k_shard_pack<<<shard_grid, kThreads, 0, st>>>(e, shard_red); ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      shard_sum(shard_red, shard_count);
      k_shard_unpack<<<shard_grid, kThreads, 0, st>>>(e, shard_red); ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
    }
    mark("X^T*T");
    refreshed = up.run(e, a, a + 1 < b.K ? 1 : 0, st);
    if (refreshed) {
      mark("update");
      continue;
    }
    k_loading<<<gp, block(a), 0, st>>>(e, a); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    mark("loading");
    k_orth<<<gp, tm, sm_k, st>>>(e, a); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    mark("orth");
    k_deflate<<<gp, tm, sm_m, st>>>(e, a, a + 1 < b.K ? 1 : 0); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    mark("deflate");
  }
  };
  if (!(graph && simpls_launch_as_graph(st, loop))) {
    loop();
    if (eligible) simpls_seen().insert(key);
  }
  if (trace) {
    FPLS_CUDA(cudaStreamSynchronize(st));
    std::map<std::string, double> acc;
    for (size_t k = 1; k < marks.size(); ++k) {
      float ms = 0.f;
      FPLS_CUDA(cudaEventElapsedTime(&ms, marks[k - 1].second, marks[k].second));
      acc[marks[k].first] += ms;
    }
    double total = 0.0;
    for (auto& kv : acc) total += kv.second;
    std::fprintf(stderr, "[fastpls trace] SIMPLS engine F=%d n=%d p=%d m=%d K=%d: %.3f ms\n", b.F, b.n,
                 b.p, b.m, b.K, total);
    for (auto& kv : acc) std::fprintf(stderr, "  %-10s %8.3f ms\n", kv.first.c_str(), kv.second);
    for (auto& mk : marks) cudaEventDestroy(mk.second);
  }
}

}  // namespace fpls
