// Gaussian sketches on the device, drawn exactly as the reference's host code
// draws them: std::mt19937(seed) feeding std::normal_distribution<double>(0, 1)
// as implemented by libstdc++ (src/svd_cpu_rsvd.cpp:10-22), column-major fill.
//
// One CTA replays one stream, in batches of kBatch words.  The words follow
// one recurrence, w[n] = w[n - 227] ^ g(w[n - 624], w[n - 623]), so 227 of them
// are independent; the first kGen threads make one word a step each (w[n - 227]
// is the thread's own last word) and need a barrier only every second step,
// while the other threads turn the batch before into variates.  Four words are
// two 53-bit canonical doubles (two 32-bit words each, low word first) and form
// one polar-method attempt (x, y), accepted when 0 < x^2 + y^2 <= 1.  An
// accepted attempt yields y * mult and then x * mult (the distribution returns
// y first and keeps x for the next call).  The arithmetic is IEEE double with
// every product and sum rounded separately (no contraction), so the stream
// matches the host bit for bit except where the device log differs from the
// host's in the last place.
// Bound by the polar arithmetic (a divide, a root and a log in FP64 on one SM),
// about 3000 cycles a batch of 681 attempts.  110,000 variates: 168 us;
// twisting 624 words in three phases and then consuming them, fourteen
// barriers a pass, took 560 us.
#include "gaussian.cuh"

#include "../../include/fastpls_b200.h"

#include <algorithm>
#include <vector>

#include "capi_util.cuh"
#include "context.cuh"

namespace fpls {
namespace {

constexpr int kN = 624;
constexpr int kStep = 227;                 // words whose recurrences are independent (624 - 397)
constexpr int kSteps = 12;                 // a batch, even so that its barriers pair the steps
constexpr int kBatch = kStep * kSteps;     // 2724 words
constexpr int kAttempts = kBatch / 4;      // 681
constexpr int kGen = 256;                  // threads that make words
constexpr int kPolarWarps = (kAttempts + 31) / 32;
constexpr int kPolar = 32 * kPolarWarps;   // threads that consume them
constexpr int kThreads = kGen + kPolar;
static_assert(kBatch % 4 == 0 && kSteps % 2 == 0 && kThreads <= 1024, "batch layout");

// The 624 words std::mt19937 holds after seeding.
struct MtState {
  uint32_t w[kN];
};

__host__ __device__ __forceinline__ uint32_t seed_word(uint32_t before, uint32_t i) {
  return 1812433253u * (before ^ (before >> 30)) + i;
}

// g of the recurrence: the upper bit of one word with the rest of the next.
__device__ __forceinline__ uint32_t twist_bits(uint32_t cur, uint32_t next) {
  const uint32_t y = (cur & 0x80000000u) | (next & 0x7fffffffu);
  return (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
}

__device__ __forceinline__ void group_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ uint32_t temper(uint32_t y) {
  y ^= y >> 11;
  y ^= (y << 7) & 0x9d2c5680u;
  y ^= (y << 15) & 0xefc60000u;
  y ^= y >> 18;
  return y;
}

// generate_canonical<double, 53>: (lo + hi * 2^32) / 2^64, clamped below 1.
__device__ __forceinline__ double canonical53(uint32_t lo, uint32_t hi) {
  const double sum = __dadd_rn((double)lo, __dmul_rn((double)hi, 4294967296.0));
  double r = __ddiv_rn(sum, 18446744073709551616.0);
  if (r >= 1.0) r = 0.99999999999999988898;  // nextafter(1, 0)
  return r;
}

// SEEDED: every stream's seed is on the device and one thread expands it (a
// serial chain, 4.6 us); otherwise the one stream's state comes with the launch.
template <bool SEEDED>
__global__ void __launch_bounds__(kThreads)
mt_gaussian_kernel(double* __restrict__ out, long long len, long long ld, const unsigned int* __restrict__ seeds,
                   const __grid_constant__ MtState state) {
  __shared__ __align__(16) uint32_t ring[2 * kBatch];   // batch b in half b & 1
  __shared__ int wsum[kPolarWarps];
  __shared__ int accepted[2];
  double* dst = out + (long long)blockIdx.x * ld;
  const int tid = threadIdx.x;
  // the state stands where the batch before the first one would end
  if (SEEDED) {
    if (tid == 0) {
      uint32_t x = seeds[blockIdx.x];
      ring[2 * kBatch - kN] = x;
      for (int i = 1; i < kN; ++i) {
        x = seed_word(x, (uint32_t)i);
        ring[2 * kBatch - kN + i] = x;
      }
    }
  } else {
    for (int i = tid; i < kN; i += kThreads) ring[2 * kBatch - kN + i] = state.w[i];
  }
  __syncthreads();
  uint32_t own = tid < kStep ? ring[2 * kBatch - kStep + tid] : 0u;   // w[n - 227] of the thread's next word
  auto make_batch = [&](int half) {
    for (int s = 0; s < kSteps; s += 2) {
      if (tid < kStep) {
        // both steps read words of earlier pairs of steps only
        const int n = half * kBatch + s * kStep + tid;
        int i0 = n - kN, i1 = n + 1 - kN, i2 = n + kStep - kN, i3 = n + 1 + kStep - kN;
        if (i0 < 0) i0 += 2 * kBatch;
        if (i1 < 0) i1 += 2 * kBatch;
        if (i2 < 0) i2 += 2 * kBatch;
        if (i3 < 0) i3 += 2 * kBatch;
        const uint32_t a = twist_bits(ring[i0], ring[i1]), b = twist_bits(ring[i2], ring[i3]);
        own ^= a;
        ring[n] = own;
        own ^= b;
        ring[n + kStep] = own;
      }
      group_sync(1, kGen);
    }
  };
  if (tid < kGen) make_batch(0);
  __syncthreads();
  long long produced = 0;
  for (int batch = 0;; ++batch) {
    if (tid < kGen) {
      make_batch((batch + 1) & 1);
    } else {
      // polar attempts over the tempered words
      const int j = tid - kGen, lane = j & 31, w = j >> 5;
      bool ok = false;
      double vx = 0.0, vy = 0.0;
      if (j < kAttempts) {
        const uint4 q = *reinterpret_cast<const uint4*>(ring + (batch & 1) * kBatch + 4 * j);
        const double u1 = canonical53(temper(q.x), temper(q.y));
        const double u2 = canonical53(temper(q.z), temper(q.w));
        const double x = __dsub_rn(__dmul_rn(2.0, u1), 1.0);
        const double y = __dsub_rn(__dmul_rn(2.0, u2), 1.0);
        const double r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
        ok = !(r2 > 1.0 || r2 == 0.0);
        if (ok) {
          const double mult = __dsqrt_rn(__ddiv_rn(__dmul_rn(-2.0, log(r2)), r2));
          vx = __dmul_rn(x, mult);
          vy = __dmul_rn(y, mult);
        }
      }
      // place of each accepted attempt: a ballot per warp, the warps before added in order
      const unsigned votes = __ballot_sync(0xffffffffu, ok);
      if (lane == 0) wsum[w] = __popc(votes);
      group_sync(2, kPolar);
      int before = 0;
      for (int u = 0; u < w; ++u) before += wsum[u];
      if (ok) {
        const long long o = produced + 2ll * (before + __popc(votes & ((1u << lane) - 1u)));
        if (o < len) dst[o] = vy;
        if (o + 1 < len) dst[o + 1] = vx;
      }
      if (w == kPolarWarps - 1 && lane == 0) accepted[batch & 1] = before + __popc(votes);
    }
    __syncthreads();
    produced += 2ll * accepted[batch & 1];
    if (produced >= len) break;
  }
}

}  // namespace

void device_gaussian_streams(double* out, long long len, long long ld, const unsigned int* d_seeds, int nstreams,
                             cudaStream_t stream) {
  if (nstreams <= 0 || len <= 0) return;
  mt_gaussian_kernel<true><<<nstreams, kThreads, 0, stream>>>(out, len, ld, d_seeds, MtState{}); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

void device_gaussian(double* out, long long n_elem, unsigned int seed) {
  if (n_elem <= 0) return;
  Context& ctx = Context::get();
  MtState st;
  st.w[0] = seed;
  for (int i = 1; i < kN; ++i) st.w[i] = seed_word(st.w[i - 1], (uint32_t)i);
  mt_gaussian_kernel<false><<<1, kThreads, 0, ctx.stream>>>(out, n_elem, n_elem, nullptr, st); ::fpls::note_launch();
  FPLS_CHECK_LAUNCH();
}

}  // namespace fpls

extern "C" int fpls_gaussian_sketch(int rows, int cols, unsigned int seed, double* out, char* err,
                                    size_t errlen) {
  return fpls::capi::guarded(err, errlen, [&] {
    FPLS_REQUIRE(rows >= 0 && cols >= 0, "gaussian_sketch: negative size");
    fpls::Context& ctx = fpls::Context::get();
    ctx.begin_call();
    const long long n = (long long)rows * cols;
    if (n == 0) return;
    double* d = ctx.arena.alloc_n<double>((size_t)n);
    fpls::device_gaussian(d, n, seed);
    fpls::d2h(out, d, (size_t)n * sizeof(double));
    ctx.sync();
  });
}
