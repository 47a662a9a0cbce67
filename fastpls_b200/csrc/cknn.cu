// Candidate-kNN classifier on the device: latent score space, class centroids,
// candidate classes by centroid similarity, and the smoothed class-kNN rerank.
//
// Reference behaviour (R package fastPLS):
//   score space / row L2 / centroids   R/main.R:657-730
//   candidate_knn_predict_cuda         src/fastPLS.cpp:1653-1711 -> 1322-1467
//   per-(row, candidate) class kNN     src/lda_cuda_kernels.cu:180-243 (at most
//                                      32 neighbour similarities are kept)
//
// The reference scores every (test row, candidate class) pair with one thread
// that walks the whole class serially.  Here the pairs are grouped by class:
// for each class the test rows that list it as a candidate form 64-row tiles,
// the class's training rows (gathered class-contiguous, row-major) are cut into
// chunks, and one CTA computes the 64 x 64 similarity tiles of a (class, tile,
// chunk) item with FP64 tensor-core MMA, folding each tile into per-row top-k
// lists held in shared memory.  A merge pass combines the chunk lists of a pair
// and applies the smoothed score; a rerank pass keeps the top classes.
#include "../../include/fastpls_b200.h"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <limits>
#include <type_traits>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "blas_f64.cuh"
#include "capi_util.cuh"
#include "cknn.cuh"
#include "context.cuh"
#include "row_topk.cuh"
#include "tc_util.cuh"

namespace fpls {
namespace {

constexpr int kKnnMax = 32;      // neighbour list cap of the replaced CUDA scorer
constexpr int kTileM = 64;       // test rows per tile
constexpr int kTileN = 64;       // training rows per similarity tile
constexpr int kBK = 16;
constexpr int kPad = 4;
constexpr int kTileThreads = 128;
constexpr int kMaxChunks = 64;   // chunk lists merged per pair
constexpr int kMinChunkRows = 2048;

// Strict '>' insertion into a descending list of length k (earlier entries win
// ties), list entries strided by `stride` (src/fastPLS.cpp:1249-1267).
template <typename V, typename I>
__device__ __forceinline__ void insert_desc(V* vals, I* idx, int k, size_t stride, V v, I id) {
  if (!(v > vals[(size_t)(k - 1) * stride])) return;
  int j = 0;
  while (!(v > vals[(size_t)j * stride])) ++j;
  for (int h = k - 1; h > j; --h) {
    vals[(size_t)h * stride] = vals[(size_t)(h - 1) * stride];
    if (idx) idx[(size_t)h * stride] = idx[(size_t)(h - 1) * stride];
  }
  vals[(size_t)j * stride] = v;
  if (idx) idx[(size_t)j * stride] = id;
}

// ---------------------------------------------------------------- fit side

// Tn = row_l2(T Ck) or row_l2(T); zero / non-finite row norms become 1
// (R/main.R:657-662).  One thread per row, sums in column order.
__global__ void row_l2_kernel(const double* __restrict__ A, int n, int k, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int j = 0; j < k; ++j) {
    const double v = A[i + (size_t)j * n];
    s += v * v;
  }
  double nr = sqrt(s);
  if (!isfinite(nr) || nr == 0.0) nr = 1.0;
  for (int j = 0; j < k; ++j) out[i + (size_t)j * n] = A[i + (size_t)j * n] / nr;
}

// Class counts and class-contiguous slots of integer codes 1..C (other codes
// are dropped).  One atomic a code on its class's counter serialises the
// frequent classes in L2: 1,200,000 codes, the most frequent of 1000 classes a
// tenth of them, took 280 us for the counts and 280 us for the slots.  So a
// block counts a range of codes in shared memory, where the count before each
// code is also its rank, and takes one range of slots a class: 12 and 17 us.
// More classes than the shared counters hold use the counters in L2 directly.
constexpr int kHistClasses = 12288;       // 48 KB of shared counters
constexpr int kSlotRows = 4096;           // codes a block ranks
constexpr int kSlotThreads = 256;
__global__ void __launch_bounds__(kSlotThreads)
class_hist_kernel(const int* __restrict__ codes, int n, int C, int in_smem, int* counts) {
  extern __shared__ int hist[];
  if (in_smem) {
    for (int c = threadIdx.x; c < C; c += kSlotThreads) hist[c] = 0;
    __syncthreads();
  }
  const long long i0 = (long long)blockIdx.x * kSlotRows;
#pragma unroll
  for (int u = 0; u < kSlotRows / kSlotThreads; ++u) {
    const long long i = i0 + u * kSlotThreads + threadIdx.x;
    const int c = i < n ? codes[i] : 0;
    if (c >= 1 && c <= C) atomicAdd((in_smem ? hist : counts) + (c - 1), 1);
  }
  if (in_smem) {
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += kSlotThreads)
      if (hist[c]) atomicAdd(counts + c, hist[c]);
  }
}

// dest[i] = slot of code i in class-contiguous order (-1 when dropped), perm
// its inverse, sorted[slot] the 0-based class; each may be null.  The order
// within a class is not fixed.
__global__ void __launch_bounds__(kSlotThreads)
class_slot_kernel(const int* __restrict__ codes, int n, int C, const int* __restrict__ offs, int in_smem,
                  int* cursor, int* __restrict__ dest, int* __restrict__ perm, int* __restrict__ sorted) {
  extern __shared__ int hist[];
  const long long i0 = (long long)blockIdx.x * kSlotRows;
  int code[kSlotRows / kSlotThreads], rank[kSlotRows / kSlotThreads];
#pragma unroll
  for (int u = 0; u < kSlotRows / kSlotThreads; ++u) {
    const long long i = i0 + u * kSlotThreads + threadIdx.x;
    const int c = i < n ? codes[i] : 0;
    code[u] = (c >= 1 && c <= C) ? c - 1 : -1;
  }
  if (in_smem) {
    for (int c = threadIdx.x; c < C; c += kSlotThreads) hist[c] = 0;
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < kSlotRows / kSlotThreads; ++u)
    rank[u] = code[u] >= 0 ? atomicAdd((in_smem ? hist : cursor) + code[u], 1) : 0;
  if (in_smem) {
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += kSlotThreads)
      if (hist[c]) hist[c] = atomicAdd(cursor + c, hist[c]);   // becomes the block's first rank
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < kSlotRows / kSlotThreads; ++u) {
    const long long i = i0 + u * kSlotThreads + threadIdx.x;
    if (i >= n) continue;
    int d = -1;
    if (code[u] >= 0) {
      d = offs[code[u]] + rank[u] + (in_smem ? hist[code[u]] : 0);
      if (perm) perm[d] = static_cast<int>(i);
      if (sorted) sorted[d] = code[u];
    }
    if (dest) dest[i] = d;
  }
}

// Column-major A (n x k) -> row-major rows out[dest[i] * k + j] (rows with
// dest < 0 dropped); dest == null keeps the order.  32 x 32 tiles through
// shared memory so both sides are coalesced.
__global__ void transpose_scatter_kernel(const double* __restrict__ A, int n, int k,
                                         const int* __restrict__ dest, double* __restrict__ out) {
  __shared__ double tile[32][33];
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int j = j0 + r, i = i0 + threadIdx.x;
    if (i < n && j < k) tile[r][threadIdx.x] = A[i + (size_t)j * n];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = i0 + r, j = j0 + threadIdx.x;
    if (i < n && j < k) {
      const int d = dest ? dest[i] : i;
      if (d >= 0) out[(size_t)d * k + j] = tile[threadIdx.x][r];
    }
  }
}

// row_l2 and the scatter above in one pass: out[dest[i] * k + j] = A[i, j] /
// norm of row i, 32 rows a CTA held in shared memory (k + 1 doubles a row) from
// the norm to the store, the sums in column order as row_l2_kernel's.  Bound by
// its one read and one write; 1,200,000 x 100: 0.48 ms, against 1.05 ms for
// the two kernels.
constexpr int kL2Rows = 32;
__global__ void __launch_bounds__(256)
row_l2_scatter_kernel(const double* __restrict__ A, int n, int k, const int* __restrict__ dest,
                      double* __restrict__ out) {
  extern __shared__ double rows_s[];   // kL2Rows x (k + 1), then the norms
  const int S = k + 1;
  double* norms = rows_s + (size_t)kL2Rows * S;
  const int i0 = blockIdx.x * kL2Rows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = i0 + lane;
#pragma unroll 8
  for (int j = warp; j < k; j += 8) rows_s[lane * S + j] = i < n ? A[i + (size_t)j * n] : 0.0;
  __syncthreads();
  if (warp == 0) {
    double s = 0.0;
#pragma unroll 8
    for (int j = 0; j < k; ++j) {
      const double v = rows_s[lane * S + j];
      s += v * v;
    }
    double nr = sqrt(s);
    if (!isfinite(nr) || nr == 0.0) nr = 1.0;
    norms[lane] = nr;
  }
  __syncthreads();
  for (int r = warp; r < kL2Rows && i0 + r < n; r += 8) {
    const int d = dest[i0 + r];
    if (d < 0) continue;
    const double nr = norms[r];
    for (int j = lane; j < k; j += 32) out[(size_t)d * k + j] = rows_s[r * S + j] / nr;
  }
}

// Class sums of class-contiguous row-major rows (R/main.R:686-698): each CTA
// walks a fixed range of rows, locating its first class by binary search in
// the class offsets; each thread keeps a column sum in registers and flushes
// it (atomicAdd into sums, C x k column-major) at class boundaries, so a very
// large class is spread over many CTAs.  The next kCentRows rows are loaded
// before they are added: a load a row, waited for, took 1.1 ms for 1,200,000
// rows of 100 columns, this 0.16 ms (960 MB).
constexpr int kCentRows = 16;
__global__ void __launch_bounds__(128) class_rowsum_kernel(const double* __restrict__ Ts, int k, int nrows,
                                                           const int* __restrict__ offs, int C, int rows,
                                                           double* __restrict__ sums) {
  const int s0 = blockIdx.x * rows;
  const int s1 = min(nrows, s0 + rows);
  const int j = blockIdx.y * 128 + threadIdx.x;
  if (j >= k) return;
  int lo = 0, hi = C - 1;  // last class with offs[c] <= s0
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (offs[mid] <= s0) lo = mid; else hi = mid - 1;
  }
  int c = lo;
  int cend = offs[c + 1];
  double acc = 0.0;
  for (int r0 = s0; r0 < s1; r0 += kCentRows) {
    double v[kCentRows];
#pragma unroll
    for (int u = 0; u < kCentRows; ++u) v[u] = r0 + u < s1 ? __ldg(Ts + (size_t)(r0 + u) * k + j) : 0.0;
#pragma unroll
    for (int u = 0; u < kCentRows; ++u) {
      if (r0 + u >= s1) break;
      if (r0 + u >= cend) {
        atomicAdd(sums + c + (size_t)j * C, acc);
        acc = 0.0;
        while (r0 + u >= offs[c + 1]) ++c;
        cend = offs[c + 1];
      }
      acc += v[u];
    }
  }
  atomicAdd(sums + c + (size_t)j * C, acc);
}

// centroid = row_l2(sums / max(count, 1)); one thread per class.
__global__ void centroid_finish_kernel(const double* __restrict__ sums, int k, const int* __restrict__ offs,
                                       int C, double* __restrict__ cent) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int cnt = offs[c + 1] - offs[c];
  const double den = cnt > 0 ? (double)cnt : 1.0;
  double sq = 0.0;
#pragma unroll 16
  for (int j = 0; j < k; ++j) {
    const double t = sums[c + (size_t)j * C] / den;
    sq += t * t;
  }
  double nr = sqrt(sq);
  if (!isfinite(nr) || nr == 0.0) nr = 1.0;
#pragma unroll 16
  for (int j = 0; j < k; ++j) cent[c + (size_t)j * C] = (sums[c + (size_t)j * C] / den) / nr;
}

// ---------------------------------------------------------------- predict side

// Top-m classes of each test row by centroid similarity (insertion order of
// src/fastPLS.cpp:1401-1415): cand = class code (1-based) or -1.
__global__ void select_candidates_kernel(const double* __restrict__ base, int ntest, int C, int top_m,
                                         int* __restrict__ cand, double* __restrict__ cbase) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ntest) return;
  double* vals = cbase + i;
  int* idx = cand + i;
  for (int j = 0; j < top_m; ++j) {
    vals[(size_t)j * ntest] = -INFINITY;
    idx[(size_t)j * ntest] = -1;
  }
  for (int c = 0; c < C; ++c)
    insert_desc(vals, idx, top_m, (size_t)ntest, base[i + (size_t)c * ntest], c + 1);
}

struct KnnItem {
  int cls;    // 0-based class
  int tile;   // 64-pair tile within the class's pair list
  int chunk;  // training-row chunk within the class
  int pad;
};

struct KnnClassInfo {
  const int* row_offs;         // C + 1 class-contiguous training row offsets
  const int* pair_offs;        // C + 1 class-sorted pair offsets
  const int* chunk_rows;       // C rows per chunk
  const int* nchunks;          // C
  const long long* part_base;  // C partial-list base offsets (in doubles)
};

// One (class, 64-pair tile, training chunk) item: 64 x 64 FP64 MMA similarity
// tiles over the chunk, folded into per-row top-k lists (two half-row lists
// per test row, merged at the end) and written as one sorted list per pair.
__global__ void __launch_bounds__(kTileThreads)
knn_tile_kernel(const KnnItem* __restrict__ items, KnnClassInfo ci, const int* __restrict__ pairs,
                int ntest, const double* __restrict__ Tq, const double* __restrict__ Ts, int K,
                int use_k, double* __restrict__ part) {
  extern __shared__ double smem[];
  double (*As)[kBK][kTileM + kPad] = reinterpret_cast<double (*)[kBK][kTileM + kPad]>(smem);
  double (*Bs)[kBK][kTileN + kPad] =
      reinterpret_cast<double (*)[kBK][kTileN + kPad]>(smem + 2 * kBK * (kTileM + kPad));
  double (*sim)[kTileN + 1] =
      reinterpret_cast<double (*)[kTileN + 1]>(smem + 2 * kBK * (kTileM + kPad) + 2 * kBK * (kTileN + kPad));
  double* lv = smem + 2 * kBK * (kTileM + kPad) + 2 * kBK * (kTileN + kPad) + kTileM * (kTileN + 1);
  __shared__ int prow[kTileM];

  const KnnItem it = items[blockIdx.x];
  const int c = it.cls;
  const int p0 = ci.pair_offs[c] + it.tile * kTileM;
  const int np = min(kTileM, ci.pair_offs[c + 1] - p0);
  const int cr = ci.chunk_rows[c];
  const int r0 = ci.row_offs[c] + it.chunk * cr;
  const int r1 = min(ci.row_offs[c + 1], r0 + cr);
  const int tid = threadIdx.x;
  if (tid < kTileM) prow[tid] = (tid < np) ? (int)(pairs[p0 + tid] % ntest) : -1;
  for (int e = 0; e < use_k; ++e) lv[e * kTileThreads + tid] = -INFINITY;
  double tail = -INFINITY;

  const int warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
  __syncthreads();

  for (int n0 = r0; n0 < r1; n0 += kTileN) {
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    double ra[8], rb[8];
    auto load = [&](int k0) {
      const int kk = tid & 15;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int mn = (tid >> 4) + 8 * i;
        const int gk = k0 + kk;
        const int tr = prow[mn];
        ra[i] = (tr >= 0 && gk < K) ? __ldg(Tq + (size_t)tr * K + gk) : 0.0;
        rb[i] = (n0 + mn < r1 && gk < K) ? __ldg(Ts + (size_t)(n0 + mn) * K + gk) : 0.0;
      }
    };
    auto store = [&](int b) {
      const int kk = tid & 15;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int mn = (tid >> 4) + 8 * i;
        As[b][kk][mn] = ra[i];
        Bs[b][kk][mn] = rb[i];
      }
    };
    load(0);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += kBK) {
      const bool has_next = k0 + kBK < K;
      if (has_next) load(k0 + kBK);
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
      if (has_next) store(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) sim[wm + i * 8 + gid][wn + j * 8 + tig * 2 + e] = acc[i][j][e];
    __syncthreads();
    {
      const int m = tid & (kTileM - 1), h = tid >> 6;
      const int ncol = min(32, r1 - n0 - h * 32);
      for (int cidx = 0; cidx < ncol; ++cidx) {
        const double v = sim[m][h * 32 + cidx];
        if (v > tail) {
          insert_desc<double, int>(lv + tid, nullptr, use_k, kTileThreads, v, 0);
          tail = lv[(use_k - 1) * kTileThreads + tid];
        }
      }
    }
    __syncthreads();
  }

  // Merge the two half-row lists of each test row; write the pair's list.
  if (tid < kTileM && tid < np) {
    const int q = p0 + tid - ci.pair_offs[c];
    double* out = part + ci.part_base[c] + ((long long)q * ci.nchunks[c] + it.chunk) * use_k;
    const double* la = lv + tid;
    const double* lb = lv + tid + kTileM;
    int ia = 0, ib = 0;
    for (int e = 0; e < use_k; ++e) {
      const double va = la[ia * kTileThreads], vb = lb[ib * kTileThreads];
      if (!(vb > va)) { out[e] = va; ++ia; } else { out[e] = vb; ++ib; }
    }
  }
}

// The same items with the whole contraction staged at once: the item's 64
// test rows are copied into shared memory once (cp.async, rows of K doubles
// at a stride S = K rounded up to 4 with S = 4 mod 16, so that the fragment
// loads of a warp hit distinct banks), the class's training rows stream
// through two 64-row buffers (the next tile's copy in flight while this one is
// multiplied), eight warps each take a 32 x 16 block of the 64 x 64 tile
// (FP64 m8n8k4), and the finished buffer holds the similarity tile for the
// top-k epilogue.  Up to K = 116.
constexpr int kV2Threads = 256;
constexpr int kV2MaxStride = 116;

__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(valid ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

template <int NB>
__global__ void __launch_bounds__(kV2Threads, NB == 1 ? 2 : 1)
knn_tile_kernel_v2(const KnnItem* __restrict__ items, KnnClassInfo ci, const int* __restrict__ pairs,
                   int ntest, const double* __restrict__ Tq, const double* __restrict__ Ts, int K, int KP, int S,
                   int use_k, double* __restrict__ part) {
  extern __shared__ double smem[];
  // a training-row buffer also holds the 64 x 65 similarity tile
  const int BS = max(S, kTileN + 1);
  double* As = smem;                   // 64 x S (test rows)
  // NB = 2: two buffers, the next tile's copy in flight during this tile;
  // NB = 1: one buffer (half the shared memory: two CTAs per SM, one CTA's
  // epilogue overlapping the other's products)
  double* Bb[2] = {smem + kTileM * S, smem + kTileM * S + (NB - 1) * kTileN * BS};   // rows of stride S
  double* lv = smem + kTileM * S + NB * kTileN * BS;                                 // use_k x 128 lists
  __shared__ int prow[kTileM];

  const KnnItem it = items[blockIdx.x];
  const int c = it.cls;
  const int p0 = ci.pair_offs[c] + it.tile * kTileM;
  const int np = min(kTileM, ci.pair_offs[c + 1] - p0);
  const int cr = ci.chunk_rows[c];
  const int r0 = ci.row_offs[c] + it.chunk * cr;
  const int r1 = min(ci.row_offs[c + 1], r0 + cr);
  const int tid = threadIdx.x;
  if (tid < kTileM) prow[tid] = (tid < np) ? (int)(pairs[p0 + tid] % ntest) : -1;
  if (tid < 2 * kTileM)
    for (int e = 0; e < use_k; ++e) lv[e * (2 * kTileM) + tid] = -INFINITY;
  double tail = -INFINITY;
  __syncthreads();

  const uint32_t sA = static_cast<uint32_t>(__cvta_generic_to_shared(As));
  const uint32_t sB[2] = {static_cast<uint32_t>(__cvta_generic_to_shared(Bb[0])),
                          static_cast<uint32_t>(__cvta_generic_to_shared(Bb[1]))};
  for (int idx = tid; idx < kTileM * KP; idx += kV2Threads) {
    const int r = idx / KP, k = idx % KP;
    const int src = prow[r];
    const bool ok = src >= 0 && k < K;
    cp_async8(sA + 8u * (r * S + k), ok ? Tq + (size_t)src * K + k : Tq, ok);
  }
  auto copy_tile = [&](int n0, int b) {
    for (int idx = tid; idx < kTileN * KP; idx += kV2Threads) {
      const int r = idx / KP, k = idx % KP;
      const bool ok = n0 + r < r1 && k < K;
      cp_async8(sB[b] + 8u * (r * S + k), ok ? Ts + (size_t)(n0 + r) * K + k : Ts, ok);
    }
  };
  copy_tile(r0, 0);
  cp_async_commit();

  const int warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * 16;
  int j = 0;
  for (int n0 = r0; n0 < r1; n0 += kTileN, ++j) {
    const int b = NB == 2 ? (j & 1) : 0;
    const bool more = n0 + kTileN < r1;
    if (NB == 2 && more) {
      copy_tile(n0 + kTileN, b ^ 1);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const double* Bs = Bb[b];
    double acc[4][2][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) acc[i][q][0] = acc[i][q][1] = 0.0;
    const double* ap = As + (wm + gid) * S + tig;
    const double* bp = Bs + (wn + gid) * S + tig;
#pragma unroll 5
    for (int kk = 0; kk < KP; kk += 4) {
      double a[4], bq[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = ap[i * 8 * S + kk];
#pragma unroll
      for (int q = 0; q < 2; ++q) bq[q] = bp[q * 8 * S + kk];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 2; ++q) dmma_8x8x4(acc[i][q][0], acc[i][q][1], a[i], bq[q]);
    }
    __syncthreads();   // every warp is done with this tile's training rows: the buffer holds the similarities
    double* sim = Bb[b];   // 64 x 65
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int e = 0; e < 2; ++e) sim[(wm + i * 8 + gid) * (kTileN + 1) + wn + q * 8 + tig * 2 + e] = acc[i][q][e];
    __syncthreads();
    if (tid < 2 * kTileM) {
      const int m = tid & (kTileM - 1), h = tid >> 6;
      const int ncol = min(32, r1 - n0 - h * 32);
      for (int cidx = 0; cidx < ncol; ++cidx) {
        const double v = sim[m * (kTileN + 1) + h * 32 + cidx];
        if (v > tail) {
          insert_desc<double, int>(lv + tid, nullptr, use_k, 2 * kTileM, v, 0);
          tail = lv[(use_k - 1) * (2 * kTileM) + tid];
        }
      }
    }
    __syncthreads();   // the buffer is refilled by the copy issued next
    if (NB == 1 && more) {
      copy_tile(n0 + kTileN, 0);
      cp_async_commit();
    }
  }

  // Merge the two half-row lists of each test row; write the pair's list.
  if (tid < kTileM && tid < np) {
    const int q = p0 + tid - ci.pair_offs[c];
    double* out = part + ci.part_base[c] + ((long long)q * ci.nchunks[c] + it.chunk) * use_k;
    const double* la = lv + tid;
    const double* lb = lv + tid + kTileM;
    int ia = 0, ib = 0;
    for (int e = 0; e < use_k; ++e) {
      const double va = la[ia * (2 * kTileM)], vb = lb[ib * (2 * kTileM)];
      if (!(vb > va)) { out[e] = va; ++ia; } else { out[e] = vb; ++ib; }
    }
  }
}

// ----------------------------------------------------- tensor-core filter
// The same (class, pair tile, training chunk) items on the 16-bit tensor
// cores, with results equal to the FP64 tiles': the products below only choose
// which training rows are scored, the scores and lists are FP64.
//   pass 1  128 pairs x 128 training rows of approximate similarities per tile
//           (tcgen05.mma kind::f16, M128 N128 K16, FP32 accumulation in TMEM,
//           double-buffered so the epilogue overlaps the next tile); each pair
//           row keeps running maxima of 64 disjoint buckets of its values and
//           writes the k largest of them per chunk;
//   bar     per pair, theta = the k-th largest of those values over all its
//           chunks.  They are approximate values of distinct training rows, so
//           theta is at most the k-th largest approximate value of the class.
//           Every approximate value is within eps of the exact dot, so each
//           row of the pair's exact top k has an approximate value of at least
//           theta - 2 eps;
//   pass 2  the same products again; every training row whose approximate
//           value reaches that bar is scored exactly (FP64 dot of the two score
//           rows, knn_exact_kernel) and the pair's k largest go to the list
//           that knn_merge_kernel reads.
// Two forms of the products, by PLANES:
//   1  one FP16 product of rows scaled by powers of two: each test row into
//      norm [1/2, 1), the training rows by one power so that their largest
//      norm is in [1/2, 1].  Rounding each factor to FP16 leaves
//      2^-11 |x_k| + 2^-25 a factor, so (2^-10 + 2^-22) |x||y| and at most
//      2 sqrt(128) 2^-25 a dot, which is below 2^-18.5 |x| max|y|; the 128
//      products are exact in FP32, and their accumulation loses at most
//      128 2^-23 |x||y| even with every addition truncated.  In all below
//      1.02 2^-10 |x| max|y|; eps = 17/16 2^-10 |x| max|y|.
//   2  both rows split into BF16 planes hi = bf16(x), lo = bf16(x - hi), three
//      products hi.hi + hi.lo + lo.hi: the split leaves x - hi - lo below
//      2^-18 |x| and drops terms below 3 2^-18 |x||y| in all (1.2e-5 |x||y|),
//      the accumulation of 3 x 128 products loses at most 4.6e-5 |x||y|;
//      5.7e-5 < eps = 2^-14 |x| max|y|.
// In large calls the FP16 form runs first: a third of the MMA work, half the bytes
// through L2 and shared memory, and two CTAs on an SM.  Its wider bar costs more
// exact scores.  Where the similarities of a class to a test row crowd within it, the
// candidate slots of that pair fill up: pass 2 raises a flag, at which the CTAs that
// start later and the exact scores return at once, and all products of the call run
// again as split BF16, and after that on the FP64 tiles.  2 classes of 15000 rows of
// 128 scores, spread 0.01, 5000 test rows: 1455 us with every FP16 candidate scored,
// 665 with the flag.
// What bounds it: a 128 x 128 tile brings 32 KB out of L2, 16384 values out of
// TMEM, one max or compare a value, and 128 x 128 x 112 products, each a third
// to a half of the tile's time; two CTAs overlap them.  1,200,000 training rows
// of 100 scores, 10^6 pairs, 7.9e9 similarities: pass 1 1.84 ms, pass 2
// 1.64 ms (1.06 ms is the MMA work of one pass at the measured 1670 TFLOP/s);
// with split BF16 throughout, a search of the maxima in shared memory and an
// atomic a hit, one CTA an SM: 5.65 and 7.55 ms.
// Score rows up to 128 wide, neighbour lists up to 16 long, less than 2^31 padded
// training rows and pairs.  Warp 0 loads (TMA, SWIZZLE_128B boxes of 64 x 128 values:
// the A tile once, the B tiles through two stages), warp 1 issues the MMAs,
// warps 2..9 are the epilogue (two per TMEM lane quarter).  Every mbarrier
// wait is bounded; no cluster multicast.
constexpr int kFT = 128;                  // pairs per tile = training rows per tile
constexpr int kFK = 128;                  // widest score row
constexpr int kFBox = 64 * kFT * 2;       // one 64-wide box of 128 16-bit rows: 16 KB
constexpr int kFEpiWarps = 8;             // two per TMEM lane quarter, half the columns each
constexpr int kFThreads = 64 + 32 * kFEpiWarps;
constexpr int kFList = 16;                // longest neighbour list of the filter
constexpr int kFBuckets = 32;             // pass 1: running maxima per thread
constexpr int kFCap = 128;                // pass 2: candidate rows kept per pair
template <int PLANES>
struct FilterTile {
  static constexpr int kOperand = PLANES * 2 * kFBox;   // planes x two boxes
  static constexpr int kBarOff = 3 * kOperand;          // A, then two B stages
  static constexpr int kSmem = kBarOff + 256 + 1024;
  static constexpr int kCtas = PLANES == 1 ? 2 : 1;     // per SM
  // D FP32; A and B FP16 (one plane) or BF16 (two)
  static constexpr uint32_t kIdesc = (1u << 4) | (PLANES == 1 ? 0u : (1u << 7) | (1u << 10)) |
                                     (uint32_t(kFT >> 3) << 17) | (uint32_t(kFT >> 4) << 24);
};
static_assert(FilterTile<2>::kSmem <= 227 * 1024 && 2 * (FilterTile<1>::kSmem + 1024) <= 228 * 1024,
              "filter tiles exceed shared memory");

__device__ __forceinline__ void umma_16bit_f32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}

// Compare-exchange steps of a bitonic merge of N values into descending order.
template <int N>
__device__ __forceinline__ void bitonic_merge_desc(float (&x)[N]) {
#pragma unroll
  for (int d = N / 2; d > 0; d >>= 1)
#pragma unroll
    for (int i = 0; i < N; ++i)
      if ((i & d) == 0) {
        const float a = x[i], b = x[i + d];
        x[i] = fmaxf(a, b);
        x[i + d] = fminf(a, b);
      }
}

// The kFList values of x[OFF ..] in descending order (bitonic network).
template <int OFF, int M>
__device__ __forceinline__ void sort16_desc(const float (&x)[M], float (&out)[kFList]) {
#pragma unroll
  for (int i = 0; i < kFList; ++i) out[i] = x[OFF + i];
#pragma unroll
  for (int size = 2; size <= kFList; size <<= 1)
#pragma unroll
    for (int d = size / 2; d > 0; d >>= 1)
#pragma unroll
      for (int i = 0; i < kFList; ++i)
        if ((i & d) == 0) {
          const bool desc = (i & size) == 0;
          const float a = out[i], b = out[i + d];
          out[i] = desc ? fmaxf(a, b) : fminf(a, b);
          out[i + d] = desc ? fminf(a, b) : fmaxf(a, b);
        }
}

template <int PASS, int PLANES>
__global__ void __launch_bounds__(kFThreads, FilterTile<PLANES>::kCtas)
knn_filter_kernel(const __grid_constant__ CUtensorMap mA0, const __grid_constant__ CUtensorMap mA1,
                  const __grid_constant__ CUtensorMap mB0, const __grid_constant__ CUtensorMap mB1,
                  const KnnItem* __restrict__ items, KnnClassInfo ci, int K, int use_k, float* __restrict__ apart,
                  const float* __restrict__ bar, int* __restrict__ ccount, int* __restrict__ crow, int* err,
                  int* inexact) {
  using Tile = FilterTile<PLANES>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Tile::kBarOff);
  uint64_t* fullA = bars;
  uint64_t* full = bars + 1;     // [2]
  uint64_t* empty = bars + 3;    // [2]
  uint64_t* tfull = bars + 5;    // [2]
  uint64_t* tempty = bars + 7;   // [2]
  uint64_t* done = bars + 9;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const KnnItem it = items[blockIdx.x];
  const int c = it.cls;
  const int p0 = ci.pair_offs[c] + it.tile * kFT;
  const int np = min(kFT, ci.pair_offs[c + 1] - p0);
  const int r0 = ci.row_offs[c] + it.chunk * ci.chunk_rows[c];
  const int r1 = min(ci.row_offs[c + 1], r0 + ci.chunk_rows[c]);
  const int ntiles = (r1 - r0 + kFT - 1) / kFT;
  // the lists of this form are known not to be exact: another form follows
  if (PASS == 2 && __syncthreads_or(threadIdx.x == 0 && *(volatile int*)inexact != 0)) return;
  const int nbox = (K + 63) / 64;        // 64-wide boxes a plane holds
  const int ksteps = (K + 15) / 16;      // columns past K are zero: their steps add nothing

  if (threadIdx.x == 0) {
    tc::mbar_init(tc::smem_u32(fullA), 1);
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(tc::smem_u32(&full[b]), 1);
      tc::mbar_init(tc::smem_u32(&empty[b]), 1);
      tc::mbar_init(tc::smem_u32(&tfull[b]), 1);
      tc::mbar_init(tc::smem_u32(&tempty[b]), 32 * kFEpiWarps);
    }
    tc::mbar_init(tc::smem_u32(done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(tmem_slot)),
                 "r"(2 * kFT)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---------------------------------------------------------- producer
    const uint32_t sa = tc::smem_u32(smem);
    auto load = [&](const CUtensorMap* m0, const CUtensorMap* m1, uint32_t dst, uint32_t fb, int row) {
      tc::mbar_expect_tx(fb, PLANES * nbox * kFBox);
      for (int x = 0; x < nbox; ++x) {
        tc::tma_load_2d(m0, dst + x * kFBox, fb, x * 64, row);
        if (PLANES == 2) tc::tma_load_2d(m1, dst + (2 + x) * kFBox, fb, x * 64, row);
      }
    };
    load(&mA0, &mA1, sa, tc::smem_u32(fullA), p0);
    int issued = 0;
    for (int t = 0; t < ntiles; ++t) {
      const int s = t & 1;
      if (!tc::mbar_wait(tc::smem_u32(&empty[s]), ((t >> 1) & 1) ^ 1, err)) break;
      load(&mB0, &mB1, sa + (1 + s) * Tile::kOperand, tc::smem_u32(&full[s]), r0 + t * kFT);
      issued = t + 1;
    }
    // the copies in flight land before the CTA exits (bounded waits)
    tc::mbar_wait(tc::smem_u32(fullA), 0, err, false);
    for (int d = 1; d <= 2 && issued - d >= 0; ++d) {
      const int u = issued - d;
      tc::mbar_wait(tc::smem_u32(&full[u & 1]), (u >> 1) & 1, err, false);
    }
  } else if (warp == 1 && lane == 0) {
    // ---------------------------------------------------------- MMA issuer
    bool ok = tc::mbar_wait(tc::smem_u32(fullA), 0, err);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t sa = tc::smem_u32(smem);
    for (int t = 0; t < ntiles && ok; ++t) {
      const int b = t & 1;
      if (!tc::mbar_wait(tc::smem_u32(&tempty[b]), ((t >> 1) & 1) ^ 1, err)) { ok = false; break; }
      if (!tc::mbar_wait(tc::smem_u32(&full[b]), (t >> 1) & 1, err)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sb = sa + (1 + b) * Tile::kOperand;
      const uint32_t acc = tmem + static_cast<uint32_t>(b * kFT);
#pragma unroll
      for (int kk = 0; kk < kFK / 16; ++kk) {
        if (kk >= ksteps) break;
        const uint32_t off = (kk >> 2) * kFBox + (kk & 3) * 32;   // box, then 32 bytes per K16 step
        const uint64_t a0 = tc::sw128_desc(sa + off), b0 = tc::sw128_desc(sb + off);
        umma_16bit_f32(acc, a0, b0, Tile::kIdesc, kk > 0 ? 1u : 0u);
        if (PLANES == 2) {
          const uint64_t a1 = tc::sw128_desc(sa + 2 * kFBox + off), b1 = tc::sw128_desc(sb + 2 * kFBox + off);
          umma_16bit_f32(acc, a0, b1, Tile::kIdesc, 1u);
          umma_16bit_f32(acc, a1, b0, Tile::kIdesc, 1u);
        }
      }
      tc::umma_commit(tc::smem_u32(&empty[b]));
      tc::umma_commit(tc::smem_u32(&tfull[b]));
    }
    // every MMA issued has completed before TMEM is released
    tc::umma_commit(tc::smem_u32(done));
    tc::mbar_wait(tc::smem_u32(done), 0, err, false);
  }
  // ------------------------------------------------------------ epilogue
  // Two warps per TMEM lane quarter, each with half of the tile's columns:
  // thread (row r, half h) loads its 64 values in two rounds and releases the
  // accumulator before it uses the second.
  //   pass 1: 32 running maxima of disjoint buckets of the half row's values
  //           (one max per value).  They are values of distinct training rows,
  //           so the k-th largest of them is at most the k-th largest
  //           approximate value, which is all the bar needs.  A sorting
  //           network in registers orders them at the end, and the two halves
  //           of a pair row meet in shared memory;
  //   pass 2: the columns that reach the bar become bits of a mask; one atomic
  //           a tile reserves their places in the pair's candidate slots, and
  //           the rows are written while the next tile is compared (with an
  //           atomic a hit, waited for, pass 2 took 1.3 times pass 1).
  const int q = warp & 3;
  const int h = (warp - 2) / 4;
  const int r = q * 32 + lane;          // pair row of the tile (TMEM lane)
  float top[kFList];
  if (warp >= 2) {
    const bool row_ok = r < np;
    float M[kFBuckets];
#pragma unroll
    for (int e = 0; e < kFBuckets; ++e) M[e] = -INFINITY;
    // the rows past np are other pairs' or padding: their maxima are not
    // written, and nothing reaches a bar that is not a number
    float thr = (PASS == 2 && row_ok) ? bar[p0 + r] : __int_as_float(0x7fffffff);
    uint32_t held[2] = {0u, 0u};   // the last tile's hits, not yet written
    int slot = 0, hbase = 0;
    auto write_hits = [&]() {
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        while (held[x]) {
          const int i = __ffs(held[x]) - 1;
          held[x] &= held[x] - 1;
          if (slot < kFCap) {
            crow[(size_t)(p0 + r) * kFCap + slot] = hbase + 32 * x + i;
          } else if (thr == thr) {   // more candidates than slots: the pair looks for no more
            atomicMax(inexact, 1);
            thr = __int_as_float(0x7fffffff);
          }
          ++slot;
        }
      }
    };
    for (int t = 0; t < ntiles; ++t) {
      const int b = t & 1;
      if (!__all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&tfull[b]), (t >> 1) & 1, err))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int n0 = r0 + t * kFT + h * 64;
      const int ncol = min(64, r1 - n0);   // columns of this half that are rows of the class (may be <= 0)
      const uint32_t base = tmem + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(b * kFT + h * 64);
      uint32_t hits[2] = {0u, 0u};
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        uint32_t v[2][16];
        tc::tmem_ld16_raw(base + x * 32, v[0]);
        tc::tmem_ld16_raw(base + x * 32 + 16, v[1]);
        tc::tmem_wait_ld();
        if (x == 1) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          tc::mbar_arrive(tc::smem_u32(&tempty[b]));
        }
        if (PASS == 1) {
          if (ncol == 64) {
#pragma unroll
            for (int i = 0; i < 32; ++i) M[i] = fmaxf(M[i], __uint_as_float(v[i >> 4][i & 15]));
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (x * 32 + i < ncol) M[i] = fmaxf(M[i], __uint_as_float(v[i >> 4][i & 15]));
          }
        } else {
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            float mx = __uint_as_float(v[g][0]);
#pragma unroll
            for (int i = 1; i < 16; ++i) mx = fmaxf(mx, __uint_as_float(v[g][i]));
            if (mx >= thr) {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (__uint_as_float(v[g][i]) >= thr) hits[x] |= 1u << (g * 16 + i);
            }
          }
        }
      }
      if (PASS == 2) {
        if (ncol < 64) {   // columns past the class's last training row
          hits[0] = ncol <= 0 ? 0u : (ncol >= 32 ? hits[0] : hits[0] & ((1u << ncol) - 1u));
          hits[1] = ncol <= 32 ? 0u : hits[1] & ((1u << (ncol - 32)) - 1u);
        }
        write_hits();
        held[0] = hits[0];
        held[1] = hits[1];
        hbase = n0;
        const int n = __popc(hits[0]) + __popc(hits[1]);
        if (n) slot = atomicAdd(ccount + p0 + r, n);
      }
    }
    if (PASS == 2) write_hits();
    if (PASS == 1) {
      // the kFList largest of this half's maxima, descending
      float other[kFList];
      sort16_desc<0>(M, top);
      sort16_desc<16>(M, other);
#pragma unroll
      for (int e = 0; e < kFList; ++e) top[e] = fmaxf(top[e], other[kFList - 1 - e]);
      bitonic_merge_desc(top);
      // every MMA that reads the A tile has completed (the last accumulator
      // was waited for), so its buffer takes the second half's list
      float* ls = reinterpret_cast<float*>(smem);
      if (h == 1) {
#pragma unroll
        for (int e = 0; e < kFList; ++e) ls[e * kFT + r] = top[e];
      }
    }
  }
  // every MMA has completed (the issuer waited for them) and every epilogue
  // thread has stored its values: one thread per pair row writes its list
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PASS == 1 && warp >= 2 && h == 0 && r < np) {
    const float* ls = reinterpret_cast<const float*>(smem);
#pragma unroll
    for (int e = 0; e < kFList; ++e) top[e] = fmaxf(top[e], ls[(kFList - 1 - e) * kFT + r]);
    bitonic_merge_desc(top);
    const int qi = p0 + r - ci.pair_offs[c];
    const long long o = ci.part_base[c] + ((long long)qi * ci.nchunks[c] + it.chunk) * use_k;
#pragma unroll
    for (int e = 0; e < kFList; ++e)
      if (e < use_k) apart[o + e] = top[e];
  }
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kFT) : "memory");
  }
}

// Row i of the FP16 plane (rows_pad x kw, zero padded) = row src(i) of S
// (row-major, K doubles a row) times a power of two, one warp a row: src(i) =
// pairs[i] % ntest when pairs is given (the test row of class-sorted pair i;
// the power takes its norm into [1/2, 1), and slack[i] = 2 eps in the scaled
// units, rounded up), else i (the power takes the largest norm of the rows,
// *ymax_bits, into [1/2, 1]).  A norm that is not finite raises *flag to 2 and
// leaves zeros, except that of a test row with a NaN, which has no similarity
// to anything: zeros, and a slack of -inf that lets no row through.
__global__ void __launch_bounds__(256)
knn_half_rows_kernel(const double* __restrict__ S, int rows, int K, const int* __restrict__ pairs, int ntest,
                     int rows_pad, int kw, const unsigned* __restrict__ ymax_bits, __half* __restrict__ plane,
                     float* __restrict__ slack, int* flag) {
  const int lane = threadIdx.x & 31;
  const double ymax = static_cast<double>(__uint_as_float(*ymax_bits));
  int ey = 0;
  const bool y_ok = isfinite(ymax);
  if (y_ok) frexp(ymax, &ey);
  const int nq = kw / 64;
  for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < rows_pad; i += gridDim.x * 8) {
    double x[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    if (i < rows) {
      const double* row = S + (size_t)(pairs ? pairs[i] % ntest : i) * K;
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (m * 64 + lane * 2 + u < K) x[m][u] = row[m * 64 + lane * 2 + u];
    }
    int e = ey;
    bool ok = y_ok;
    if (pairs) {   // warp-uniform
      double s2 = 0.0;
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int u = 0; u < 2; ++u) s2 = fma(x[m][u], x[m][u], s2);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      const double norm = sqrt(s2);
      ok = isfinite(norm);
      e = 0;
      if (ok) frexp(norm, &e);
      if (lane == 0 && i < rows) {
        // 2 (17/16 2^-10) |x| max|y|
        slack[i] = ok ? __double2float_ru(ldexp(norm, -e) * ldexp(ymax, -ey) * (17.0 / 8192.0))
                      : (norm != norm ? -INFINITY : INFINITY);
        if (!ok && norm == norm) atomicMax(flag, 2);
      }
    }
    if (!y_ok && i == 0 && lane == 0) atomicMax(flag, 2);
    // 2^-e as two factors, each of which a double holds
    const double f1 = ok ? ldexp(1.0, -(e / 2)) : 0.0, f2 = ok ? ldexp(1.0, -(e - e / 2)) : 0.0;
#pragma unroll
    for (int m = 0; m < 2; ++m)
      if (m < nq) {
        const __half2 v = ok ? __halves2half2(__double2half(x[m][0] * f1 * f2), __double2half(x[m][1] * f1 * f2))
                             : __halves2half2(__half(0.0f), __half(0.0f));
        *reinterpret_cast<__half2*>(plane + (size_t)i * kw + m * 64 + lane * 2) = v;
      }
  }
}

// Row i of the BF16 planes (rows_pad x kw, zero padded) = the hi / lo split
// of row src(i) of S (row-major, K doubles per row): src(i) = pairs[i] % ntest
// when pairs is given (the test row of class-sorted pair i; slack[i] = 2 eps,
// rounded up; a row with a NaN, as above), else i.  These planes are not scaled:
// where the products may leave the range of FP32, or a factor that of BF16, far
// enough that the error is no longer below eps, *flag becomes 2 (the FP64 tiles).
__global__ void __launch_bounds__(256)
knn_split_rows_kernel(const double* __restrict__ S, int rows, int K, const int* __restrict__ pairs, int ntest,
                      int rows_pad, int kw, const unsigned* __restrict__ ymax_bits, __nv_bfloat16* __restrict__ hi,
                      __nv_bfloat16* __restrict__ lo, float* __restrict__ slack, int* flag) {
  const int lane = threadIdx.x & 31;
  for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < rows_pad; i += gridDim.x * 8) {
    const double* row = S + (size_t)(i < rows ? (pairs ? pairs[i] % ntest : i) : 0) * K;
    double s2 = 0.0;
    for (int k = lane; k < kw; k += 32) {
      const double x = (i < rows && k < K) ? row[k] : 0.0;
      s2 = fma(x, x, s2);
      const __nv_bfloat16 h = __double2bfloat16(x);
      hi[(size_t)i * kw + k] = h;
      lo[(size_t)i * kw + k] = __double2bfloat16(x - static_cast<double>(__bfloat162float(h)));
    }
    if (pairs && i < rows) {
      for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      if (lane == 0) {
        const double norm = sqrt(s2), ymax = static_cast<double>(__uint_as_float(*ymax_bits));
        const double largest = norm * ymax;
        slack[i] = norm != norm ? -INFINITY : __double2float_ru(ldexp(largest, -13));
        // lo rounds to a multiple of 2^-133: at most sqrt(128) 2^-134 of a row, 5.3e-7 of
        // 1e-33, in both factors; products below 2^-126 add at most 3 128 2^-126, 4.6e-7 of
        // 1e-29.  With these, 5.9e-5 < eps = 6.1e-5.
        const bool in_range = norm >= 1e-33 && ymax >= 1e-33 && largest >= 1e-29 && largest <= 1e38;
        if (!isfinite(ymax) || (norm > 0.0 && ymax > 0.0 && !in_range)) atomicMax(flag, 2);
      }
    }
  }
}

// Largest row norm of S (rows x K, row-major), rounded up, as float bits
// (non-negative floats order as their bit patterns; a NaN norm wins): one warp
// a row, four rows' loads in flight.
__global__ void __launch_bounds__(256)
knn_row_norm_max_kernel(const double* __restrict__ S, int rows, int K, unsigned* out) {
  const int lane = threadIdx.x & 31;
  const int stride = gridDim.x * 8;
  unsigned best = 0u;
  for (int i0 = blockIdx.x * 8 + (threadIdx.x >> 5); i0 < rows; i0 += 4 * stride) {
    double x[4][kFK / 32];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int m = 0; m < kFK / 32; ++m) {
        const long long i = i0 + (long long)u * stride;
        x[u][m] = (i < rows && lane + 32 * m < K) ? S[(size_t)i * K + lane + 32 * m] : 0.0;
      }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      double s2 = 0.0;
#pragma unroll
      for (int m = 0; m < kFK / 32; ++m) s2 = fma(x[u][m], x[u][m], s2);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      best = max(best, __float_as_uint(__double2float_ru(sqrt(s2))) & 0x7fffffffu);
    }
  }
  if (lane == 0 && best) atomicMax(out, best);
}

// Per class-sorted pair: theta = the k-th largest approximate similarity over
// all its chunk lists, bar = theta - 2 eps (rounded down), -inf when the
// class has fewer than k rows.  The running list stays in registers: a sorted
// chunk list merges into it as max against the reverse, then a bitonic merge.
__global__ void __launch_bounds__(256)
knn_filter_bar_kernel(const float* __restrict__ apart, KnnClassInfo ci, int C, long long total_pairs, int use_k,
                      const float* __restrict__ slack, float* __restrict__ bar) {
  const long long P = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (P >= total_pairs) return;
  int lo = 0, hi = C - 1;   // the last class whose pair offset is <= P
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (ci.pair_offs[mid] <= P) lo = mid;
    else hi = mid - 1;
  }
  const int c = lo;
  const long long qi = P - ci.pair_offs[c];
  const int nch = ci.nchunks[c];
  float lst[kFList];
#pragma unroll
  for (int e = 0; e < kFList; ++e) lst[e] = -INFINITY;
  for (int s = 0; s < nch; ++s) {
    const float* l = apart + ci.part_base[c] + (qi * nch + s) * use_k;
    float in[kFList];
#pragma unroll
    for (int e = 0; e < kFList; ++e) in[e] = e < use_k ? l[e] : -INFINITY;
#pragma unroll
    for (int e = 0; e < kFList; ++e) lst[e] = fmaxf(lst[e], in[kFList - 1 - e]);
    bitonic_merge_desc(lst);
  }
  float theta = lst[0];
#pragma unroll
  for (int e = 1; e < kFList; ++e)
    if (e == use_k - 1) theta = lst[e];
  // a slack of -inf marks a test row with a NaN: nothing reaches its bar, not a number
  const float sl = slack[P];
  bar[P] = sl == -INFINITY ? __int_as_float(0x7fffffff) : (theta == -INFINITY ? -INFINITY : __fadd_rd(theta, -sl));
}

// Exact scores of the candidates of every pair, one warp per class-sorted pair:
// the lanes split every FP64 dot (four candidates at a time, the test row loaded
// once) and lane c keeps the values of candidates c, c + 32, ...  The use_k
// largest go to plist[P * use_k ..] in descending order (-inf when there are
// fewer).  Nothing is scored where a pair has more candidates than its slots
// hold (*inexact, raised by pass 2): another form of the products follows.
// What bounds it: the candidates' rows, 8 K bytes each, out of L2.  A lane
// a candidate past 32 of them took 32 lines a load: 100,000 pairs with 50 candidates
// of 128 scores, the call 808 us so, 358 with the dots split.
__global__ void knn_exact_kernel(const int* __restrict__ ccount, const int* __restrict__ crow,
                                 const int* __restrict__ pairs, long long total_pairs, int ntest,
                                 const double* __restrict__ Tq, const double* __restrict__ Ts, int K, int use_k,
                                 double* __restrict__ plist, const int* __restrict__ inexact) {
  const long long P = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (P >= total_pairs) return;   // whole warps
  if (*inexact != 0) return;
  const int cnt = ccount[P];   // at most kFCap
  const double* xr = Tq + (size_t)(pairs[P] % ntest) * K;
  double xv[kFK / 32];
#pragma unroll
  for (int m = 0; m < kFK / 32; ++m) xv[m] = (lane + 32 * m < K) ? xr[lane + 32 * m] : 0.0;
  double v[kFCap / 32];
#pragma unroll
  for (int u = 0; u < kFCap / 32; ++u) {
    v[u] = -INFINITY;
    const int end = min(cnt, 32 * u + 32);
    for (int c0 = 32 * u; c0 < end; c0 += 4) {
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (c0 + c < end) {
          const double* yr = Ts + (size_t)crow[(size_t)P * kFCap + c0 + c] * K;
#pragma unroll
          for (int m = 0; m < kFK / 32; ++m)
            if (lane + 32 * m < K) acc[c] = fma(xv[m], yr[lane + 32 * m], acc[c]);
        }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (32 * u + lane == c0 + c && c0 + c < end) v[u] = acc[c];
    }
    if (!(v[u] == v[u])) v[u] = -INFINITY;   // a NaN never enters a list
  }
  if (cnt <= 32) {
    // each value goes to its rank in the descending list (ties by lane)
    int rank = 0;
    for (int j = 0; j < 32; ++j) {
      const double vj = __shfl_sync(0xffffffffu, v[0], j);
      rank += (vj > v[0] || (vj == v[0] && j < lane)) ? 1 : 0;
    }
    if (rank < use_k) plist[P * use_k + rank] = v[0];
    return;
  }
  for (int e = 0; e < use_k; ++e) {
    // the warp's largest remaining value; the lowest lane holding it gives it up
    double m = v[0];
#pragma unroll
    for (int u = 1; u < kFCap / 32; ++u) m = fmax(m, v[u]);
    double wm = m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wm = fmax(wm, __shfl_xor_sync(0xffffffffu, wm, o));
    const unsigned holders = __ballot_sync(0xffffffffu, m == wm && wm > -INFINITY);
    if (holders && lane == __ffs(holders) - 1) {
      bool done = false;
#pragma unroll
      for (int u = 0; u < kFCap / 32; ++u)
        if (!done && v[u] == wm) {
          v[u] = -INFINITY;
          done = true;
        }
    }
    if (lane == 0) plist[P * use_k + e] = holders ? wm : -INFINITY;
  }
}

// A plane of 16-bit score rows, kw (64 or 128) wide, in boxes of 64 x 128.
CUtensorMap make_rows_map(CUtensorMapDataType type, const void* p, int rows_pad, int kw) {
  CUtensorMap m;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(kw), static_cast<cuuint64_t>(rows_pad)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(kw) * 2};
  cuuint32_t box[2] = {64, static_cast<cuuint32_t>(kFT)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = tc::encode_fn()(&m, type, 2, const_cast<void*>(p), dims, strides,
                               box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw Error(kErrCuda, "cuTensorMapEncodeTiled failed (cKNN score planes)");
  return m;
}

// Per pair: merge its chunk lists, smoothed class score (src/fastPLS.cpp:1287-1320,
// src/lda_cuda_kernels.cu:225-242), add alpha * base + bias.
__global__ void knn_merge_kernel(const int* __restrict__ pairs, long long total_pairs,
                                 const int* __restrict__ cand, const double* __restrict__ cbase,
                                 KnnClassInfo ci, const double* __restrict__ part, int use_k,
                                 double tau, double alpha, const double* __restrict__ bias,
                                 double* __restrict__ cscore) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= total_pairs) return;
  const int flat = pairs[q];
  const int c = cand[flat] - 1;
  const int found = ci.row_offs[c + 1] - ci.row_offs[c];
  double top[kKnnMax];
  for (int e = 0; e < use_k; ++e) top[e] = -INFINITY;
  const int S = ci.nchunks[c];
  const double* src = part + ci.part_base[c] + (q - ci.pair_offs[c]) * (long long)S * use_k;
  for (int s = 0; s < S; ++s)
    for (int e = 0; e < use_k; ++e) {
      const double v = src[(size_t)s * use_k + e];
      if (!(v > top[use_k - 1])) break;  // lists are sorted: the rest is smaller
      insert_desc<double, int>(top, nullptr, use_k, 1, v, 0);
    }
  double local;
  if (found < 1 || !isfinite(top[0])) {
    local = -INFINITY;
  } else {
    const int denom = max(1, min(use_k, found));
    const double mx = top[0];
    double acc = 0.0;
    for (int j = 0; j < denom; ++j) acc += exp((top[j] - mx) / tau);
    local = mx + tau * log(acc / (double)denom);
  }
  cscore[flat] = __dadd_rn(__dadd_rn(local, __dmul_rn(alpha, cbase[flat])), bias[c]);
}

// Rerank the candidates of each row by score (src/fastPLS.cpp:1447-1466).
__global__ void knn_rerank_kernel(const int* __restrict__ cand, const double* __restrict__ cscore,
                                  int ntest, int C, int top_m, int top_k, int* __restrict__ top_index,
                                  double* __restrict__ top_score) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ntest) return;
  for (int j = 0; j < top_k; ++j) {
    top_score[i + (size_t)j * ntest] = -INFINITY;
    top_index[i + (size_t)j * ntest] = -1;
  }
  for (int j = 0; j < top_m; ++j) {
    const int cls = cand[i + (size_t)j * ntest];
    if (cls < 1 || cls > C) continue;
    insert_desc(top_score + i, top_index + i, top_k, (size_t)ntest, cscore[i + (size_t)j * ntest], cls);
  }
}

void class_hist(const int* codes, int n, int C, int* counts) {
  Context& ctx = Context::get();
  FPLS_CUDA(cudaMemsetAsync(counts, 0, C * sizeof(int), ctx.stream));
  if (n <= 0) return;
  const int in_smem = C <= kHistClasses;
  class_hist_kernel<<<ceil_div(n, kSlotRows), kSlotThreads, in_smem ? C * sizeof(int) : 0, ctx.stream>>>(
      codes, n, C, in_smem, counts);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

}  // namespace

void class_slots(const int* codes, int n, int C, const int* d_offs, int* dest, int* perm, int* sorted) {
  Context& ctx = Context::get();
  int* cursor = ctx.arena.alloc_n<int>(C);
  FPLS_CUDA(cudaMemsetAsync(cursor, 0, C * sizeof(int), ctx.stream));
  if (n <= 0) return;
  const int in_smem = C <= kHistClasses;
  class_slot_kernel<<<ceil_div(n, kSlotRows), kSlotThreads, in_smem ? C * sizeof(int) : 0, ctx.stream>>>(
      codes, n, C, d_offs, in_smem, cursor, dest, perm, sorted);
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

ClassRows group_rows_by_class(const double* dT, int n, int k, const int* dcodes, int C) {
  Context& ctx = Context::get();
  ClassRows cr;
  int* counts = ctx.arena.alloc_n<int>(C);
  int* dest = ctx.arena.alloc_n<int>(std::max(n, 1));
  class_hist(dcodes, n, C, counts);
  std::vector<int> h(C);
  d2h(h.data(), counts, C * sizeof(int));
  ctx.sync();
  cr.offs.assign(C + 1, 0);
  for (int c = 0; c < C; ++c) cr.offs[c + 1] = cr.offs[c] + h[c];
  int* d_offs = ctx.arena.alloc_n<int>(C + 1);
  h2d(d_offs, cr.offs.data(), (C + 1) * sizeof(int));
  cr.d_offs = d_offs;
  class_slots(dcodes, n, C, d_offs, dest, nullptr, nullptr);
  cr.Ts = ctx.arena.alloc_n<double>((size_t)std::max(cr.offs[C], 1) * k);
  dim3 grid(ceil_div(n, 32), ceil_div(k, 32));
  transpose_scatter_kernel<<<grid, dim3(32, 8), 0, ctx.stream>>>(dT, n, k, dest, cr.Ts); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  return cr;
}

using capi::upload;

void candidate_scores_device(const double* dT, int n, int k, const double* dCk, double* dTn) {
  Context& ctx = Context::get();
  const double* src = dT;
  if (dCk) {
    double* prod = ctx.arena.alloc_n<double>((size_t)n * k);
    gemm(false, false, n, k, k, 1.0, dT, n, dCk, k, 0.0, prod, n);
    src = prod;
  }
  row_l2_kernel<<<ceil_div(n, 128), 128, 0, ctx.stream>>>(src, n, k, dTn); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void candidate_score_rows_device(const double* dT, int n, int k, const double* dCk, const int* dest, double* dTs) {
  Context& ctx = Context::get();
  double* prod = ctx.arena.alloc_n<double>((size_t)n * k);
  gemm(false, false, n, k, k, 1.0, dT, n, dCk, k, 0.0, prod, n);
  const size_t smem = sizeof(double) * kL2Rows * ((size_t)k + 2);
  // two CTAs an SM still hide a row's norm behind the other's copies; wider
  // rows go through memory between the two steps
  if (smem <= 100 * 1024) {
    static bool attr = false;
    if (!attr) {
      FPLS_CUDA(cudaFuncSetAttribute(row_l2_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
      attr = true;
    }
    row_l2_scatter_kernel<<<ceil_div(n, kL2Rows), 256, smem, ctx.stream>>>(prod, n, k, dest, dTs);
  } else {
    double* Tn = ctx.arena.alloc_n<double>((size_t)n * k);
    row_l2_kernel<<<ceil_div(n, 128), 128, 0, ctx.stream>>>(prod, n, k, Tn); ::fpls::note_launch();
    dim3 grid(ceil_div(n, 32), ceil_div(k, 32));
    transpose_scatter_kernel<<<grid, dim3(32, 8), 0, ctx.stream>>>(Tn, n, k, dest, dTs);
  }
  ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void candidate_centroids_device(const ClassRows& cr, int k, int C, double* dCent) {
  Context& ctx = Context::get();
  const int nvalid = cr.offs[C];
  double* sums = ctx.arena.alloc_n<double>((size_t)C * k);
  fill(sums, (size_t)C * k, 0.0);
  if (nvalid > 0) {
    const int rows = std::min(2048, std::max(64, ceil_div(ceil_div(nvalid, 16 * ctx.sm_count), kCentRows) * kCentRows));
    class_rowsum_kernel<<<dim3(ceil_div(nvalid, rows), ceil_div(k, 128)), 128, 0, ctx.stream>>>(
        cr.Ts, k, nvalid, cr.d_offs, C, rows, sums); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
  }
  centroid_finish_kernel<<<ceil_div(C, 32), 32, 0, ctx.stream>>>(sums, k, cr.d_offs, C, dCent); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void candidate_knn_predict_device(const double* dTt, int ntest, const ClassRows& cr, int kdim, const double* dC,
                                  int C, const double* dbias, int top_k, int top_m, int knn_k, double tau,
                                  double alpha, int* d_ti, double* d_ts) {
  Context& ctx = Context::get();
  const int tk = std::max(1, std::min(top_k, C));
  const int tm = std::max(tk, std::min(std::max(1, top_m), C));
  const int use_k = std::max(1, std::min(std::max(1, knn_k), kKnnMax));
  const double tau_e = (std::isfinite(tau) && tau > 0.0) ? tau : 0.2;
  const double alpha_e = std::isfinite(alpha) ? alpha : 0.5;
  const long long npairs = (long long)ntest * tm;
  FPLS_REQUIRE(npairs < (1ll << 31), "candidate-kNN: ntest * top_m must stay below 2^31");
  double* bias0 = nullptr;
  if (!dbias) {
    bias0 = ctx.arena.alloc_n<double>(C);
    fill(bias0, C, 0.0);
    dbias = bias0;
  }
  PhaseTimer pt("candidate-kNN predict");
  // base scores and candidate classes
  double* base = ctx.arena.alloc_n<double>((size_t)ntest * C);
  gemm(false, true, ntest, C, kdim, 1.0, dTt, ntest, dC, C, 0.0, base, ntest);
  int* cand = ctx.arena.alloc_n<int>((size_t)npairs);
  double* cbase = ctx.arena.alloc_n<double>((size_t)npairs);
  if (tm <= kRowTopkMax) {
    row_topk_launch(base, ntest, C, nullptr, tm, -1, false, cand, cbase);
  } else {   // longer candidate lists than the register lists hold
    select_candidates_kernel<<<ceil_div(ntest, 128), 128, 0, ctx.stream>>>(base, ntest, C, tm, cand, cbase);
    ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
  }

  // test rows row-major, as the training rows are
  pt.mark("base scores + candidates");
  double* Tq = ctx.arena.alloc_n<double>((size_t)ntest * kdim);
  {
    dim3 grid(ceil_div(ntest, 32), ceil_div(kdim, 32));
    transpose_scatter_kernel<<<grid, dim3(32, 8), 0, ctx.stream>>>(dTt, ntest, kdim, nullptr, Tq); ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
  }

  // (row, candidate) pairs grouped by class
  int* pcount = ctx.arena.alloc_n<int>(C);
  class_hist(cand, (int)npairs, C, pcount);
  std::vector<int> hp(C);
  d2h(hp.data(), pcount, C * sizeof(int));
  ctx.sync();
  // Tile kernel (FASTPLS_CKNN_TILES): 4 or unset the tensor-core filter with
  // exact FP64 rescoring (score rows up to 128 wide), 5 / 6 the filter with the
  // FP16 / the split BF16 products first at any size, 1 the 16-wide k-step FP64
  // kernel, 2 / 3 the staged FP64 kernels with two / one training-row buffers.
  const char* tv = std::getenv("FASTPLS_CKNN_TILES");
  const char sel = (tv && tv[0]) ? tv[0] : '4';
  const bool use_filter = sel >= '4' && kdim <= kFK && use_k <= kFList;
  std::vector<int> poffs(C + 1, 0);
  for (int c = 0; c < C; ++c) poffs[c + 1] = poffs[c] + hp[c];
  // the (class, pair tile, row chunk) items of a tile kernel and the places of
  // their lists: tile_m pairs an item, chunks of a multiple of gran rows
  std::vector<int> chunk_rows(C), nchunks(C);
  std::vector<long long> part_base(C);
  std::vector<KnnItem> items;
  long long part_total = 0;
  auto make_items = [&](int tile_m, int gran) {
    items.clear();
    part_total = 0;
    for (int c = 0; c < C; ++c) {
      const int rows = cr.offs[c + 1] - cr.offs[c];
      int S = 0, cr_rows = 0;
      if (rows > 0) {
        S = std::min(kMaxChunks, std::max(1, ceil_div(rows, kMinChunkRows)));
        cr_rows = ceil_div(ceil_div(rows, S), gran) * gran;
        S = ceil_div(rows, cr_rows);
      }
      chunk_rows[c] = cr_rows;
      nchunks[c] = S;
      part_base[c] = part_total;
      part_total += (long long)hp[c] * S * use_k;
      if (rows > 0 && hp[c] > 0) {
        const int tiles = ceil_div(hp[c], tile_m);
        for (int t = 0; t < tiles; ++t)
          for (int s = 0; s < S; ++s) items.push_back(KnnItem{c, t, s, 0});
      }
    }
    FPLS_REQUIRE(items.size() < (1u << 31), "candidate-kNN: too many work items");
  };
  make_items(use_filter ? kFT : kTileM, use_filter ? kFT : kTileN);
  const long long total_pairs = poffs[C];
  double work = 0.0;   // (pair, training row) products
  for (int c = 0; c < C; ++c) work += (double)hp[c] * (cr.offs[c + 1] - cr.offs[c]);
  if (pt.enabled()) {
    std::fprintf(stderr, "[fastpls trace] candidate-kNN: %lld pairs, %.3e pair-rows (%.3e flop), %zu items\n",
                 total_pairs, work, 2.0 * work * kdim, items.size());
  }
  int* pairs = ctx.arena.alloc_n<int>((size_t)std::max<long long>(total_pairs, 1));
  int* d_poffs = ctx.arena.alloc_n<int>(C + 1);
  h2d(d_poffs, poffs.data(), (C + 1) * sizeof(int));
  class_slots(cand, (int)npairs, C, d_poffs, nullptr, pairs, nullptr);

  KnnClassInfo ci;
  ci.row_offs = cr.d_offs;
  ci.pair_offs = d_poffs;
  auto upload_items = [&] {
    ci.chunk_rows = upload(chunk_rows.data(), C);
    ci.nchunks = upload(nchunks.data(), C);
    ci.part_base = upload(part_base.data(), C);
  };
  upload_items();
  double* cscore = ctx.arena.alloc_n<double>((size_t)npairs);
  pt.mark("class rows + pair lists");
  // the lists the merge reads: one exact list per pair from the filter, or
  // (pair, chunk) lists of the FP64 tiles
  KnnClassInfo ci_merge = ci;
  const double* merge_part = nullptr;
  bool scored = false;
  if (!items.empty() && use_filter) {
    const KnnItem* ditems = upload(items.data(), items.size());
    const int slot = ctx.prof_begin("cknn_filter", ctx.stream);
    const int nvalid = cr.offs[C];
    const long long a_rows = (total_pairs + kFT - 1) / kFT * kFT + kFT;
    const long long b_rows = ((long long)nvalid + kFT - 1) / kFT * kFT + kFT;
    FPLS_REQUIRE(a_rows < (1ll << 31) && b_rows < (1ll << 31), "candidate-kNN: too many rows for the filter");
    const int kw = kdim <= 64 ? 64 : kFK;
    unsigned* ymax = ctx.arena.alloc_n<unsigned>(1);
    dzero(ymax, sizeof(unsigned));
    const int gs = 8 * ctx.sm_count;
    if (nvalid > 0) {
      knn_row_norm_max_kernel<<<std::min(gs, ceil_div(nvalid, 8)), 256, 0, ctx.stream>>>(cr.Ts, nvalid, kdim, ymax);
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
    }
    float* apart = ctx.arena.alloc_n<float>((size_t)std::max<long long>(part_total, 1));
    float* barv = ctx.arena.alloc_n<float>((size_t)total_pairs);
    float* slack = ctx.arena.alloc_n<float>((size_t)total_pairs);
    int* ccount = ctx.arena.alloc_n<int>((size_t)total_pairs);
    int* crow = ctx.arena.alloc_n<int>((size_t)total_pairs * kFCap);
    double* plist = ctx.arena.alloc_n<double>((size_t)total_pairs * use_k);
    uint16_t* aplane = ctx.arena.alloc_n<uint16_t>((size_t)a_rows * kw);
    uint16_t* bplane = ctx.arena.alloc_n<uint16_t>((size_t)b_rows * kw);
    int* ferr = ctx.d_status + 24;    // [0] a pipeline wait ran out, [1] the lists are not exact
    const unsigned ng = (unsigned)items.size();
    const unsigned bar_grid = (unsigned)ceil_div(total_pairs, 256);
    const unsigned exact_grid = (unsigned)ceil_div(total_pairs * 32, 256);
    // both passes, the bar and the exact scores with planes of one form;
    // returns [1]: 0 when every list is exact, 1 when a pair had more rows
    // within the error bar than its slots hold, 2 when a row's norm is not finite
    auto passes = [&](auto planes, const CUtensorMap& mA0, const CUtensorMap& mA1, const CUtensorMap& mB0,
                      const CUtensorMap& mB1) {
      constexpr int PLANES = decltype(planes)::value;
      static bool fattr = false;
      if (!fattr) {
        FPLS_CUDA(cudaFuncSetAttribute(knn_filter_kernel<1, PLANES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       FilterTile<PLANES>::kSmem));
        FPLS_CUDA(cudaFuncSetAttribute(knn_filter_kernel<2, PLANES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       FilterTile<PLANES>::kSmem));
        fattr = true;
      }
      dzero(ccount, (size_t)total_pairs * sizeof(int));
      knn_filter_kernel<1, PLANES><<<ng, kFThreads, FilterTile<PLANES>::kSmem, ctx.stream>>>(
          mA0, mA1, mB0, mB1, ditems, ci, kdim, use_k, apart, nullptr, nullptr, nullptr, ferr, ferr + 1);
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      pt.mark("filter pass 1");
      knn_filter_bar_kernel<<<bar_grid, 256, 0, ctx.stream>>>(apart, ci, C, total_pairs, use_k, slack, barv);
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      pt.mark("filter bar");
      knn_filter_kernel<2, PLANES><<<ng, kFThreads, FilterTile<PLANES>::kSmem, ctx.stream>>>(
          mA0, mA1, mB0, mB1, ditems, ci, kdim, use_k, nullptr, barv, ccount, crow, ferr, ferr + 1);
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      pt.mark("filter pass 2");
      knn_exact_kernel<<<exact_grid, 256, 0, ctx.stream>>>(ccount, crow, pairs, total_pairs, ntest, Tq, cr.Ts, kdim,
                                                          use_k, plist, ferr + 1);
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      pt.mark("filter exact scores");
      int flags[2] = {0, 0};
      d2h(flags, ferr, 2 * sizeof(int));
      ctx.sync();
      if (flags[0]) throw Error(kErrCuda, "candidate-kNN: a filter tile's pipeline wait timed out");
      return flags[1];
    };
    dzero(ferr, 2 * sizeof(int));
    // FP16 products first only where they are most of the call and a crowded pair's
    // exact scores little of it.  Measured, us, FP16 first / split BF16 first, where
    // the FP16 slots hold and where similarities crowd (unit-norm rows, 5 candidate
    // classes, or both of 2):
    //   2 x 15000 rows, 64 scores, 5000 test rows (1.9e10): 354 / 408, 568 / 419
    //   2 x 3000, 110, 5000 (6.6e9): 281 / 303, 435 / 329
    //   20 x 50, 100, 10000 (1e8 and less): 3 % apart at most, 1.1 to 2 times
    //   200 x 100, 128, 100000 (1.3e10): 1704 / 1828, 4467 / 1883 (every row of a
    //   class within the FP16 bar, and its slots hold them)
    const bool half_first =
        sel == '5' || (sel == '4' && 2.0 * work * kdim >= 1e10 && work >= 2048.0 * (double)total_pairs);
    int left = 1;
    if (half_first) {
      __half* a16 = reinterpret_cast<__half*>(aplane);
      __half* b16 = reinterpret_cast<__half*>(bplane);
      knn_half_rows_kernel<<<gs, 256, 0, ctx.stream>>>(Tq, (int)total_pairs, kdim, pairs, ntest, (int)a_rows, kw,
                                                       ymax, a16, slack, ferr + 1);
      ::fpls::note_launch();
      knn_half_rows_kernel<<<gs, 256, 0, ctx.stream>>>(cr.Ts, nvalid, kdim, nullptr, 1, (int)b_rows, kw, ymax, b16,
                                                       nullptr, ferr + 1);
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      pt.mark("filter planes");
      const CUtensorMap mA = make_rows_map(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a16, (int)a_rows, kw);
      const CUtensorMap mB = make_rows_map(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, b16, (int)b_rows, kw);
      left = passes(std::integral_constant<int, 1>{}, mA, mA, mB, mB);
      if (left == 1) dzero(ferr, 2 * sizeof(int));
    }
    if (left == 1) {
      // the first form, or similarities crowd within the FP16 bar: this one is 17 times narrower
      __nv_bfloat16* ah = reinterpret_cast<__nv_bfloat16*>(aplane);
      __nv_bfloat16* bh = reinterpret_cast<__nv_bfloat16*>(bplane);
      __nv_bfloat16* al = ctx.arena.alloc_n<__nv_bfloat16>((size_t)a_rows * kw);
      __nv_bfloat16* bl = ctx.arena.alloc_n<__nv_bfloat16>((size_t)b_rows * kw);
      knn_split_rows_kernel<<<gs, 256, 0, ctx.stream>>>(Tq, (int)total_pairs, kdim, pairs, ntest, (int)a_rows, kw,
                                                        ymax, ah, al, slack, ferr + 1);
      ::fpls::note_launch();
      knn_split_rows_kernel<<<gs, 256, 0, ctx.stream>>>(cr.Ts, nvalid, kdim, nullptr, 1, (int)b_rows, kw, ymax, bh,
                                                        bl, nullptr, nullptr);
      ::fpls::note_launch();
      FPLS_CHECK_LAUNCH();
      pt.mark("filter planes");
      const CUtensorMapDataType bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
      left = passes(std::integral_constant<int, 2>{}, make_rows_map(bf, ah, (int)a_rows, kw),
                    make_rows_map(bf, al, (int)a_rows, kw), make_rows_map(bf, bh, (int)b_rows, kw),
                    make_rows_map(bf, bl, (int)b_rows, kw));
    }
    if (slot >= 0) {
      // algorithmic work: the FP16 products of both passes over every
      // (candidate pair, class row); bytes: the score planes of every class's
      // training rows once per 128-pair tile and pass, the pair planes once a
      // pass (the class's time includes the planes, the bar, the exact scores
      // and the split BF16 products where they run)
      double bytes = 2.0 * 2.0 * kw * (double)total_pairs;
      for (int c = 0; c < C; ++c)
        bytes += 2.0 * 2.0 * kw * (double)(cr.offs[c + 1] - cr.offs[c]) * (double)ceil_div(hp[c], kFT);
      ctx.prof_end(slot, ctx.stream, bytes, 2.0 * 2.0 * work * kdim);
    }
    if (left == 0) {
      std::vector<int> ones(C, 1);
      std::vector<long long> pbase(C);
      for (int c = 0; c < C; ++c) pbase[c] = (long long)poffs[c] * use_k;
      ci_merge.nchunks = upload(ones.data(), C);
      ci_merge.part_base = upload(pbase.data(), C);
      merge_part = plist;
      scored = true;
    } else {
      // the FP64 tiles score every row
      make_items(kTileM, kTileN);
      upload_items();
      ci_merge = ci;
    }
  }
  if (!items.empty() && !scored) {
    const KnnItem* ditems = upload(items.data(), items.size());
    double* part = ctx.arena.alloc_n<double>((size_t)std::max<long long>(part_total, 1));
    merge_part = part;
    const int slot = ctx.prof_begin("cknn_tiles", ctx.stream);
    // stride of the staged rows: K rounded up to 4, then to 4 mod 16
    const int KP = (kdim + 3) / 4 * 4;
    const int S = KP + (4 - KP % 16 + 16) % 16;
    // FP64 tile kernels: on the large-class workload (K = 100) the
    // similarity tiles took 123.4 ms (k-step), 162.6 ms (two buffers: one
    // 8-warp CTA per SM, the tensor pipe idles while the top-k epilogue runs)
    // and 107.2 ms (one buffer: two CTAs per SM, one CTA's epilogue overlapping
    // the other's products).  The filter takes score rows up to 128 wide and
    // lists up to 16 long; past that the staged kernel runs, and rows wider
    // than 116 doubles take the k-step kernel.
    if (S <= kV2MaxStride && sel != '1') {
      const int nb = sel == '2' ? 2 : 1;
      const size_t smem = sizeof(double) * ((size_t)kTileM * S + nb * (size_t)kTileN * std::max(S, kTileN + 1) +
                                            (size_t)use_k * 2 * kTileM);
      const int smem_max = (int)(sizeof(double) * ((size_t)(kTileM + nb * kTileN) * kV2MaxStride +
                                                   (size_t)kKnnMax * 2 * kTileM));
      static bool attr2[2] = {false, false};
      if (!attr2[nb - 1]) {
        if (nb == 2)
          FPLS_CUDA(cudaFuncSetAttribute(knn_tile_kernel_v2<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
        else {
          FPLS_CUDA(cudaFuncSetAttribute(knn_tile_kernel_v2<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
          // all of the SM's unified memory as shared memory: two 113 KB CTAs at K = 100
          FPLS_CUDA(cudaFuncSetAttribute(knn_tile_kernel_v2<1>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared));
        }
        attr2[nb - 1] = true;
      }
      if (nb == 2)
        knn_tile_kernel_v2<2><<<(unsigned)items.size(), kV2Threads, smem, ctx.stream>>>(
            ditems, ci, pairs, ntest, Tq, cr.Ts, kdim, KP, S, use_k, part);
      else
        knn_tile_kernel_v2<1><<<(unsigned)items.size(), kV2Threads, smem, ctx.stream>>>(
            ditems, ci, pairs, ntest, Tq, cr.Ts, kdim, KP, S, use_k, part);
    } else {
      const size_t smem = sizeof(double) * (2 * kBK * (kTileM + kPad) + 2 * kBK * (kTileN + kPad) +
                                            kTileM * (kTileN + 1) + (size_t)kKnnMax * kTileThreads);
      static bool attr_set = false;
      if (!attr_set) {
        FPLS_CUDA(cudaFuncSetAttribute(knn_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set = true;
      }
      knn_tile_kernel<<<(unsigned)items.size(), kTileThreads, smem, ctx.stream>>>(
          ditems, ci, pairs, ntest, Tq, cr.Ts, kdim, use_k, part);
    }
    ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
    if (slot >= 0) {
      // algorithmic work: one kdim-long FP64 dot per (candidate pair, class row);
      // bytes: every class's training rows once per 64-row tile of its pairs,
      // the test rows once
      double work = 0.0, bytes = 8.0 * (double)ntest * kdim;
      for (int c = 0; c < C; ++c) {
        const double rows = cr.offs[c + 1] - cr.offs[c];
        work += (double)hp[c] * rows;
        bytes += 8.0 * kdim * rows * (double)ceil_div(hp[c], kTileM);
      }
      ctx.prof_end(slot, ctx.stream, bytes, 2.0 * work * kdim);
    }
  }
  pt.mark("similarity tiles");
  fill(cscore, (size_t)npairs, -INFINITY);
  if (total_pairs > 0) {
    knn_merge_kernel<<<ceil_div(total_pairs, 128), 128, 0, ctx.stream>>>(
        pairs, total_pairs, cand, cbase, ci_merge, merge_part, use_k, tau_e, alpha_e, dbias, cscore);
    ::fpls::note_launch();
    FPLS_CHECK_LAUNCH();
  }
  knn_rerank_kernel<<<ceil_div(ntest, 128), 128, 0, ctx.stream>>>(cand, cscore, ntest, C, tm, tk, d_ti, d_ts); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
  pt.mark("merge + rerank");
  pt.report();
}

}  // namespace fpls

using namespace fpls;

extern "C" {

int fpls_candidate_scores(const double* T, int n, int k, const double* Ck, double* Tn, char* err,
                          size_t errlen) {
  return capi::guarded(err, errlen, [&] {
    FPLS_REQUIRE(n > 0 && k > 0, "candidate-kNN requires at least one latent component");
    Context& ctx = Context::get();
    ctx.begin_call();
    const double* dT = upload(T, (size_t)n * k);
    const double* dC = Ck ? upload(Ck, (size_t)k * k) : nullptr;
    double* out = ctx.arena.alloc_n<double>((size_t)n * k);
    candidate_scores_device(dT, n, k, dC, out);
    d2h(Tn, out, (size_t)n * k * sizeof(double));
    ctx.sync();
  });
}

int fpls_candidate_centroids(const double* Tn, int n, int k, const int* y_codes, int n_classes,
                             double* centroids, char* err, size_t errlen) {
  return capi::guarded(err, errlen, [&] {
    FPLS_REQUIRE(n > 0 && k > 0, "candidate centroids: empty score matrix");
    FPLS_REQUIRE(n_classes >= 1, "candidate-kNN requires at least one class");
    Context& ctx = Context::get();
    ctx.begin_call();
    const double* dT = upload(Tn, (size_t)n * k);
    const int* dy = upload(y_codes, n);
    double* dC = ctx.arena.alloc_n<double>((size_t)n_classes * k);
    candidate_centroids_device(group_rows_by_class(dT, n, k, dy, n_classes), k, n_classes, dC);
    d2h(centroids, dC, (size_t)n_classes * k * sizeof(double));
    ctx.sync();
  });
}

int fpls_candidate_knn_predict(const double* Ttest_norm, int ntest, const double* Ttrain_norm,
                               int ntrain, int kdim, const int* y_codes, const double* centroids,
                               int n_classes, const double* candidate_bias, int top_k, int top_m,
                               int knn_k, double tau, double alpha, int* top_index,
                               double* top_score, char* err, size_t errlen) {
  return capi::guarded(err, errlen, [&] {
    FPLS_REQUIRE(n_classes >= 1, "candidate-kNN requires at least one class");
    FPLS_REQUIRE(ntest > 0 && ntrain > 0 && kdim > 0, "candidate-kNN: empty score matrices");
    Context& ctx = Context::get();
    ctx.begin_call();
    const int C = n_classes;
    const int tk = std::max(1, std::min(top_k, C));
    const double* dTt = upload(Ttest_norm, (size_t)ntest * kdim);
    const double* dTr = upload(Ttrain_norm, (size_t)ntrain * kdim);
    const int* dy = upload(y_codes, ntrain);
    const double* dC = upload(centroids, (size_t)C * kdim);
    const double* dbias = candidate_bias ? upload(candidate_bias, C) : nullptr;
    int* d_ti = ctx.arena.alloc_n<int>((size_t)ntest * tk);
    double* d_ts = ctx.arena.alloc_n<double>((size_t)ntest * tk);
    candidate_knn_predict_device(dTt, ntest, group_rows_by_class(dTr, ntrain, kdim, dy, C), kdim, dC, C, dbias, top_k,
                                 top_m, knn_k, tau, alpha, d_ti, d_ts);
    d2h(top_index, d_ti, (size_t)ntest * tk * sizeof(int));
    d2h(top_score, d_ts, (size_t)ntest * tk * sizeof(double));
    ctx.sync();
  });
}

}  // extern "C"
