"""The phases of a SIMPLS component on a chunk in shared memory, compiled for the host with a thread per CUDA
thread, one warp held back after every barrier: what one warp still reads, no other may write before the next
barrier, so the results do not depend on which warp is late."""
import os
import shutil
import subprocess

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastpls_b200", "csrc",
                   "simpls_engine.cu")

SHIM = r"""
#include <algorithm>
#include <barrier>
#include <chrono>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
using std::isfinite;
using std::max;
using std::min;
#define __device__
#define __forceinline__ inline
#define __align__(n) alignas(n)
struct double2 { double x, y; };
static double2 make_double2(double x, double y) { return {x, y}; }
static constexpr int NT = 256;
static thread_local struct { unsigned x; } threadIdx;
static std::barrier<> block_bar(NT);
static std::vector<std::barrier<>*> warp_bar;
static double lanes[NT];
static int late;
static void __syncthreads() {
  block_bar.arrive_and_wait();
  if ((int)(threadIdx.x >> 5) == late) std::this_thread::sleep_for(std::chrono::milliseconds(15));
}
static void __syncwarp() { warp_bar[threadIdx.x >> 5]->arrive_and_wait(); }
static double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) {
    lanes[threadIdx.x] = v;
    __syncwarp();
    v += lanes[threadIdx.x ^ o];
    __syncwarp();
  }
  return v;
}
constexpr int kSumThreads = 256;
constexpr int kSumWarps = kSumThreads / 32;
constexpr int kAhead = 16;
struct Eng {
  int n, p, m, F, K, cp, cn, iters, m1_mode, psplits;
  const int* labels;
  const double *mY_all, *delta, *colscale, *dY, *omega, *ppart;
  double *S, *R, *Q, *V, *tnorm, *y, *zA, *zB, *npart, *r, *tpart, *qpart, *P, *wpart, *vpart, *vSpart;
  int *ncomp_done, *status;
};
static double sum_parts(const double* parts, int count, size_t stride) {
  double s = 0.0;
  for (int c = 0; c < count; ++c) s += parts[c * stride];
  return s;
}
"""

MAIN = r"""
int main(int argc, char** argv) {
  late = std::atoi(argv[1]);
  const int m = std::atoi(argv[2]), a = 2, rows = 201;
  for (int w = 0; w < NT / 32; ++w) warp_bar.push_back(new std::barrier<>(32));
  Eng e{};
  e.n = 5; e.p = rows; e.m = m; e.F = 1; e.K = 4; e.cp = 1; e.cn = 1; e.iters = 1;
  unsigned seed = 7;
  auto fill = [&](size_t count) {
    double* d = new double[count];
    for (size_t i = 0; i < count; ++i) { seed = seed * 1664525u + 1013904223u; d[i] = (double)(seed >> 8) / (1 << 23) - 1.0; }
    return d;
  };
  e.S = fill((size_t)rows * m); e.R = fill(rows * 4); e.Q = fill(m * 4); e.V = fill(rows * 4); e.tnorm = fill(4);
  e.y = fill(rows); e.zA = fill(m); e.zB = fill(m); e.npart = fill(1); e.r = fill(rows); e.tpart = fill(2);
  e.tpart[0] = 2.0; e.qpart = fill(m); e.P = fill(rows); e.wpart = fill(4); e.vpart = fill(1); e.vSpart = fill(m);
  int done = 0, status = 0;
  e.ncomp_done = &done; e.status = &status;
  std::vector<double> S((size_t)kTile * m, 0.0), coef(std::max(m, 4));
  for (int j = 0; j < m; ++j) for (int i = 0; i < rows; ++i) S[j * kTile + i] = e.S[j * rows + i];
  static TileShared sh;
  const TileView w{0, rows, S.data(), e.V, rows};
  std::vector<std::thread> threads;
  for (int t = 0; t < NT; ++t)
    threads.emplace_back([&, t] {
      threadIdx.x = t;
      tile_loading<NT, true>(e, w, a, 0, 0, sh);
      __syncthreads();
      tile_orth<NT, true>(e, w, a, 0, 0, coef.data(), sh);
      __syncthreads();
      tile_deflate<NT>(e, w, a, 1, 0, 0, coef.data(), sh, nullptr, e.S);
      __syncthreads();
      tile_apply<NT>(e, w, e.zA, e.zB, 1, 0, 0, coef.data(), sh);
    });
  for (auto& t : threads) t.join();
  auto put = [](const double* d, int n) { for (int i = 0; i < n; ++i) std::printf("%a\n", d[i]); };
  put(e.vpart, 1); put(e.npart, 1); put(e.vSpart, m); put(e.wpart, a); put(e.V + a * rows, rows); put(e.S, rows * m);
  put(e.R + a * rows, rows); put(e.Q + a * m, m); put(e.y, rows); put(e.zA, m);
}
"""


@pytest.fixture(scope="module")
def phases(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    text = open(SRC).read()
    body = text[text.index("constexpr int kTile = 256;"):text.index("// The chunk's S into shared memory, asynchronously")]
    d = tmp_path_factory.mktemp("phases")
    (d / "phases.cpp").write_text(SHIM + body + MAIN)
    subprocess.run([gxx, "-std=c++20", "-O1", "-pthread", "-w", "-ffp-contract=off", "-o", str(d / "phases"),
                    str(d / "phases.cpp")], check=True)

    def run(late, m):
        r = subprocess.run([str(d / "phases"), str(late), str(m)], check=True, capture_output=True, text=True, timeout=60)
        return np.array([float.fromhex(v) for v in r.stdout.split()])
    return run


# fewer responses than warps (several warps share a column and meet in shared memory), one each, and more
@pytest.mark.parametrize("m", [1, 3, 7, 8, 12])
def test_no_phase_depends_on_a_late_warp(phases, m):
    ref = phases(-1, m)
    assert np.all(np.isfinite(ref))
    for late in (0, 1, 7):
        assert np.array_equal(phases(late, m), ref), late
