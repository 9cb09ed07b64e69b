// The one-warp-per-pair all-pairs DTW kernel (approximateMedoidIndices'
// launch loop, dba.hpp:67-161, with DTWDistance's pair-distance epilogue,
// dtw.hpp:116-125, 242-257) and its launch-shape helpers.
//
// Private to the library's .cu files: everything is in an anonymous
// namespace, so every translation unit that includes this header compiles its
// own copy of the kernel into its own module.  dtw_pairwise.cu launches it
// with a caller workspace, dtw_pairwise_noalloc.cu with the scratch array it
// owns (a module of its own, so that only callers of that entry point load
// the array).
#ifndef ODBA_PAIRWISE_KERNEL_CUH
#define ODBA_PAIRWISE_KERNEL_CUH

#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>

#include "dtw_warp.cuh"

namespace odba {
namespace {

constexpr int kWarpsPerBlock = 4;
// 12 warps per SM: 300 float series of 2000-8000 samples take 140 ms, with 8
// warps 155, with 16 (128 registers: the widest swaths spill) 152.
constexpr int kMinBlocksPerSM = 3;

template <typename T>
struct PairwiseArgs {
  const T *series;
  const uint64_t *offsets;
  const uint64_t *lens;
  int n;
  unsigned long long pbeg;    // first pair of the range (upper-triangle index)
  unsigned long long npairs;  // pairs in the range
  T *dists;
  unsigned long long *counter;
  T *edges;
  unsigned long long edge_stride;  // elements per edge buffer
  int open_start, open_end;
  int classes;                     // passes over the pairs, largest first (size_classes)
};

// Largest pairs first, without a sort: the warps go over the range
// kSizeClasses times and take, each time, the pairs of one class of matrix
// size (sixteenths of max_len^2, the largest class first), so that the pairs
// left for the end are the small ones.  A skipped pair costs an atomic and two
// loads, so it has to be a small part of the longest pair's time, which is what
// the order can save: max_len^2 of at least kClassLen2 per pair of the launch.
// One class / sixteen: float, 100 series (4950 pairs) of 100-300 samples 0.096 /
// 0.130 ms, 500-1000 0.464 / 0.492, 1000-2000 1.710 / 1.714; 300 of 2000-8000
// 142.0 / 141.3; double, 100 of 500-1000 1.496 / 1.492, 1000-2000 5.21 / 5.02,
// 1000-4000 13.4 / 12.6.  Below two pairs per warp nearly all start at once;
// above kClassWaves the tail is less than the skips.
constexpr int kSizeClasses = 16;
constexpr unsigned long long kClassWaves = 64, kClassLen2 = 400;

inline int size_classes(unsigned long long npairs, int warps, unsigned long long max_len) {
  return npairs >= 2ull * warps && npairs <= kClassWaves * warps &&
                 max_len * max_len >= kClassLen2 * npairs
             ? kSizeClasses
             : 1;
}

__device__ __forceinline__ long long row_start(long long s, long long n) {
  return s * n - s * (s + 1) / 2;
}

// Upper-triangle pair index -> (s, j).
__device__ __forceinline__ void pair_of(long long p, long long n, int &s_out, int &j_out) {
  const double b = 2.0 * double(n) - 1.0;
  long long s = (long long)((b - sqrt(b * b - 8.0 * double(p))) * 0.5);
  if (s < 0) s = 0;
  if (s > n - 2) s = n - 2;
  while (s + 1 <= n - 2 && row_start(s + 1, n) <= p) ++s;
  while (s > 0 && row_start(s, n) > p) --s;
  s_out = int(s);
  j_out = int(s + 1 + (p - row_start(s, n)));
}

template <typename T>
__device__ __forceinline__ T pair_distance(T corner, int m, int n, int os, int oe) {
  float v;
  if ((oe && !os) || (!oe && os)) {
    v = __fdiv_rn(__fsqrt_rn(float(corner)), float(m));
  } else {
    v = __fsqrt_rn(float(corner));
  }
  return T(v);
}

// The reference's open-end shortcut (dtw.hpp:74-129, open end without open
// start) is checked on the left edge of every 1024-column reference swath that
// starts past the last row: if that edge's value on the last row equals its
// shortcut minimum (ShortcutRows), the swath and all later ones stop and the
// distance is taken from that value -- from the sentinel it has just stored
// when the matrix has one row (dtw.hpp:113, 121).  swath_checks_shortcut: the
// swath [c0, c0 + W) whose right edge is such a left edge.
template <typename T>
__device__ __forceinline__ bool swath_checks_shortcut(int c0, int W, int m, int n, bool oe, int r0) {
  const int cnext = c0 + W;
  return oe && r0 == 0 && cnext < n && (cnext % kRefSwath) == 0 && cnext > m;
}

template <typename T>
__device__ __forceinline__ bool shortcut_fires(const EdgeStat<T> &st, int m, T &corner) {
  if (st.etop != st.emin) return false;
  corner = m == 1 ? Num<T>::big() : st.etop;
  return true;
}

// Full swaths use RF registers per lane (swath width 32*RF); the last, partial
// swath uses the smallest multiple of RQ registers that covers it, and a matrix of
// up to 128 columns 4 (200 series of 20-60 samples: 0.16 ms with 8, 0.087 so).
// RQ = 8: every width is code of its own, and the warps of an SM run different
// widths next to each other.  With RQ = 4 (8 float widths) and five copies of the
// step per width they spend half of their time waiting for instructions: pairs of
// 8-48 series of 200-2000 samples took 4.46 ms, with two copies and RQ = 8 1.57,
// RQ = 16 1.54; full-width work pays 0.4% for RQ = 8 and 2% for 16.
template <typename T, int RF, int RQ>
__device__ void sweep_pair(SwathJob<T> job, WarpSmem<T> &sm, T *e0, T *e1, T &corner) {
  constexpr int W = 32 * RF;
  int k = 0;
  for (int c0 = 0; c0 < job.n; c0 += W, ++k) {
    const int width = job.n - c0 < W ? job.n - c0 : W;
    const bool last = c0 + W >= job.n;
    job.c0 = c0;
    job.track = swath_checks_shortcut<T>(c0, W, job.m, job.n, job.open_end, job.r0);
    // ping-pong: swath k writes buffer k%2 and reads buffer (k+1)%2
    job.edge_in = c0 ? ((k & 1) ? e0 : e1) : nullptr;
    job.edge_out = last ? nullptr : ((k & 1) ? e1 : e0);
    job.free_diag0 = c0 > 0 && (c0 % kRefSwath) == 0;
    job.corner_init = c0 == 0 ? (job.r0 ? Num<T>::big() : T(0)) : (job.r0 ? T(0) : Num<T>::big());
    const int rneed = (width + 31) / 32;
    const int rq = (rneed + RQ - 1) / RQ * RQ;
    EdgeStat<T> st{Num<T>::big(), Num<T>::big()};
    if (job.n <= 128) {
      st = sweep_warp<T, 4>(job, sm, last, corner);
    } else if (rq >= RF) {
      st = sweep_warp<T, RF>(job, sm, last, corner);
    } else {
      switch (rq / RQ) {
#define ODBA_CASE(K)                                                       \
  case K:                                                                  \
    if constexpr (K * RQ < RF) st = sweep_warp<T, K * RQ>(job, sm, last, corner); \
    break;
        ODBA_CASE(1)
        ODBA_CASE(2)
        ODBA_CASE(3)
        ODBA_CASE(4)
        ODBA_CASE(5)
        ODBA_CASE(6)
        ODBA_CASE(7)
#undef ODBA_CASE
        default:
          break;
      }
    }
    // the next swath reads what this swath's lanes stored
    __syncwarp();
    if (job.track && shortcut_fires<T>(st, job.m, corner)) return;
  }
}

template <typename T, int RF, int RQ>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, kMinBlocksPerSM)
    pairwise_kernel(PairwiseArgs<T> a) {
  __shared__ WarpSmem<T> sm[kWarpsPerBlock];
  const int lane = threadIdx.x & 31;
  const long long slot = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  T *e0 = a.edges + slot * 2 * a.edge_stride;
  T *e1 = e0 + a.edge_stride;
  for (;;) {
    unsigned long long q = 0;
    if (lane == 0) q = atomicAdd(a.counter, 1ull);
    q = __shfl_sync(kFull, q, 0);
    int cls = 0;
    while (q >= a.npairs && cls < a.classes) {
      q -= a.npairs;
      ++cls;
    }
    if (cls == a.classes) break;
    const long long p = (long long)(a.pbeg + a.npairs - 1 - q);
    int s, j;
    pair_of(p, a.n, s, j);
    if (a.classes > 1) {
      const float top = float(a.edge_stride - 32);
      const float part = float(a.lens[s]) * float(a.lens[j]) / (top * top);  // of the largest matrix
      const int c = a.classes - 1 - int(part * float(a.classes));
      if ((c < 0 ? 0 : c) != cls) continue;
    }
    SwathJob<T> job;
    job.x = a.series + a.offsets[s];
    job.m = int(a.lens[s]);
    job.y = a.series + a.offsets[j];
    job.n = int(a.lens[j]);
    job.r0 = a.open_start ? 1 : 0;
    job.open_end = a.open_end != 0;
    if ((unsigned long long)job.m + 32 > a.edge_stride) {
      // a first series longer than the max_len the edge buffers were sized
      // for: its edges would run into the next warp's buffers
      if (lane == 0) a.dists[p] = Num<T>::quiet_nan();
      continue;
    }
    T corner = T(0);
    sweep_pair<T, RF, RQ>(job, sm[threadIdx.x >> 5], e0, e1, corner);
    if (lane == 0) a.dists[p] = pair_distance<T>(corner, job.m, job.n, a.open_start, a.open_end);
  }
}

template <typename T>
struct Tune;
template <>
struct Tune<float> {
  static constexpr int RF = 32, RQ = 8;
};
template <>
struct Tune<double> {
  static constexpr int RF = 16, RQ = 8;
};

// Resident blocks of pairwise_kernel on the current device, cached per device
// index (host threads may call at once: the cache entries are atomics, and a
// race only computes the same value twice).
template <typename T>
int grid_size() {
  static std::atomic<int> cached[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    const int c = cached[dev].load(std::memory_order_relaxed);
    if (c) return c;
  }
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &per_sm, pairwise_kernel<T, Tune<T>::RF, Tune<T>::RQ>, kWarpsPerBlock * 32, 0);
  if (per_sm < 1) per_sm = 1;
  if (sms < 1) sms = 1;
  const int g = sms * per_sm;
  if (dev >= 0 && dev < 64) cached[dev].store(g, std::memory_order_relaxed);
  return g;
}

}  // namespace
}  // namespace odba

#endif  // ODBA_PAIRWISE_KERNEL_CUH
