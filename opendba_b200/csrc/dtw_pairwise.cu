// All-vs-all DTW distances for the medoid pass: the work of
// approximateMedoidIndices' launch loop (dba.hpp:67-161) and the pair-distance
// epilogue of DTWDistance (dtw.hpp:116-125, 242-257), as one persistent launch.
//
// Every warp of the grid pulls pairs from a device work counter, largest pair
// index first (with length-sorted input that is roughly largest cost first),
// and sweeps the pair swath by swath with the register wavefront of
// dtw_warp.cuh; few pairs go through the swath pipeline below, a block per
// swath (dtw_block.cuh).  The swath right-edge column goes through a per-warp
// (per-pair) ping-pong buffer in global memory (L2-resident in practice).
//
// Output: the reference's upper-triangle layout, pair (s, j), s < j, at
// index s*n - s*(s+1)/2 + (j - s - 1) (clustering.cuh:4-6), with
//   dist = (T) sqrtf(C[m-1][n-1])           global / open modes
//   dist = (T)(sqrtf(C[m-1][n-1]) / m)      exactly one open end
// computed in float like the reference (sqrtf even for double, dtw.hpp:121,251,254).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <vector>

#include "dtw_block.cuh"
#include "dtw_device.cuh"
#include "dtw_pipe.cuh"
#include "odba_internal.h"
#include "pairwise_kernel.cuh"

namespace odba {

// Workspace of the one-warp-per-pair launches: the work counter and two edge
// buffers per resident warp.
template <typename T>
size_t whole_workspace_bytes(uint64_t max_len) {
  const unsigned long long stride = (max_len + 32 + 31) / 32 * 32;
  const size_t slots = size_t(grid_size<T>()) * kWarpsPerBlock;
  return 256 + slots * 2 * stride * sizeof(T);
}

template <typename T, int RF>
int whole_pairwise_launch(const T *series, const uint64_t *offsets, const uint64_t *lens, int n,
                          uint64_t max_len, int os, int oe, unsigned long long pbeg,
                          unsigned long long npairs, T *dists, void *workspace, size_t ws_bytes,
                          cudaStream_t stream) {
  if (n < 2 || npairs == 0) return ODBA_OK;
  const size_t need = whole_workspace_bytes<T>(max_len);
  if (ws_bytes < need) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "workspace too small");
  PairwiseArgs<T> a;
  a.series = series;
  a.offsets = offsets;
  a.lens = lens;
  a.n = n;
  a.pbeg = pbeg;
  a.npairs = npairs;
  a.dists = dists;
  a.counter = static_cast<unsigned long long *>(workspace);
  a.edges = reinterpret_cast<T *>(static_cast<char *>(workspace) + 256);
  a.edge_stride = (max_len + 32 + 31) / 32 * 32;
  a.open_start = os;
  a.open_end = oe;
  a.classes = size_classes(a.npairs, grid_size<T>() * kWarpsPerBlock, max_len);
  cudaMemsetAsync(a.counter, 0, 16, stream);  // work counter and error word
  pairwise_kernel<T, RF, Tune<T>::RQ><<<grid_size<T>(), kWarpsPerBlock * 32, 0, stream>>>(a);
  return check_launch("pairwise DTW kernel");
}

}  // namespace odba

// ---------------------------------------------------------------------------
// Pairs from a task list: many independent jobs (each its own set of series,
// its own alignment mode) in one persistent launch.  The caller orders the
// tasks (largest m*n first keeps the tail short); each warp takes the next
// task from the device counter.
namespace odba {
namespace {

template <typename T, int RF, int RQ>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, kMinBlocksPerSM)
    pairlist_kernel(const T *series, const uint64_t *offsets, const uint64_t *lens,
                    const odba_pair_task *tasks, unsigned long long ntasks, T *dists,
                    unsigned long long *counter, T *edges, unsigned long long edge_stride) {
  __shared__ WarpSmem<T> sm[kWarpsPerBlock];
  const int lane = threadIdx.x & 31;
  const long long slot = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  T *e0 = edges + slot * 2 * edge_stride;
  T *e1 = e0 + edge_stride;
  for (;;) {
    unsigned long long q = 0;
    if (lane == 0) q = atomicAdd(counter, 1ull);
    q = __shfl_sync(kFull, q, 0);
    if (q >= ntasks) break;
    const odba_pair_task task = tasks[q];
    const int os = int((task.out >> 62) & 1ull), oe = int((task.out >> 63) & 1ull);
    const unsigned long long out = task.out & ((1ull << 62) - 1);
    SwathJob<T> job;
    job.x = series + offsets[task.first];
    job.m = int(lens[task.first]);
    job.y = series + offsets[task.second];
    job.n = int(lens[task.second]);
    job.r0 = os;
    job.open_end = oe != 0;
    if ((unsigned long long)job.m + 32 > edge_stride) {  // longer than max_len (pairwise_kernel)
      if (lane == 0) dists[out] = Num<T>::quiet_nan();
      continue;
    }
    T corner = T(0);
    sweep_pair<T, RF, RQ>(job, sm[threadIdx.x >> 5], e0, e1, corner);
    if (lane == 0) dists[out] = pair_distance<T>(corner, job.m, job.n, os, oe);
  }
}

}  // namespace

template <typename T, int RF>
int whole_pairlist_launch(const T *series, const uint64_t *offsets, const uint64_t *lens,
                          const odba_pair_task *tasks, unsigned long long ntasks, uint64_t max_len,
                          T *dists, void *workspace, size_t ws_bytes, cudaStream_t stream) {
  if (ntasks == 0) return ODBA_OK;
  const size_t need = whole_workspace_bytes<T>(max_len);
  if (ws_bytes < need) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "workspace too small");
  auto *counter = static_cast<unsigned long long *>(workspace);
  T *edges = reinterpret_cast<T *>(static_cast<char *>(workspace) + 256);
  const unsigned long long stride = (max_len + 32 + 31) / 32 * 32;
  cudaMemsetAsync(counter, 0, 16, stream);  // work counter and error word
  unsigned long long blocks = (ntasks + kWarpsPerBlock - 1) / kWarpsPerBlock;
  int grid = grid_size<T>();
  if (blocks < (unsigned long long)grid) grid = int(blocks);
  pairlist_kernel<T, RF, Tune<T>::RQ><<<grid, kWarpsPerBlock * 32, 0, stream>>>(
      series, offsets, lens, tasks, ntasks, dists, counter, edges, stride);
  return check_launch("pair-list DTW kernel");
}

}  // namespace odba

// ---------------------------------------------------------------------------
// Few pairs: swath-pipelined sweeps.
//
// With fewer pairs than warps (16 series of 1M-4M samples give 120 pairs for
// ~1776 resident warps), one warp per pair would leave most of the GPU idle.
// Here the unit of work is one 1024-column swath of one pair, swept by a block
// (sweep_block): task k is a swath of pair k % P (P pairs) in turn k / P, so swath s of a pair
// is always handed out after swath s - 1 of the same pair.  Each pair owns
// two edge buffers (swath s writes buffer s % 2 and reads buffer (s - 1) % 2),
// and every swath of every pair has its own progress word (rows stored so far),
// which the producing block's feeder publishes with a gpu-scope release every
// 8 or 16 row pairs and at the end of its swath.  The consuming block's feeder
// acquires the word before reading rows it has not seen published.  Why this
// cannot deadlock: a block waits only on the previous swath of its pair, which
// was handed out earlier to a block that is already running and waits only on
// earlier tasks, so the earliest unfinished task never waits.  Why two buffers
// suffice: swath s + 1 overwrites row r of buffer (s - 1) % 2 only after swath
// s has published row r, and swath s reads its input rows before it computes
// (and publishes) them; swaths s and s + 2 do write one buffer at the same
// time, at different rows, which is why the progress words are per swath and
// not per buffer.
//
// Every wait is bounded: a block whose feeder could not go on for limit_ns
// (%globaltimer) raises the launch's error word and continues; every other
// waiting block sees the word and stops waiting, so a fault in the hand-off
// ends the launch quickly with the pairs it touched written as NaN.
namespace odba {
namespace {

// Blocks per SM of the swath pipeline.
constexpr int kPipeBlocksF32 = 4, kPipeBlocksF64 = 3;

template <typename T>
struct PipeArgs {
  const T *series;
  const uint64_t *offsets;
  const uint64_t *lens;
  int n;                         // series (all-vs-all) when list is null
  const odba_pair_task *list;    // pair list, or null for the upper triangle of n series
  unsigned long long pbeg;       // first pair of the range (upper triangle only)
  unsigned long long npairs;
  unsigned long long max_swaths;
  T *dists;
  unsigned long long *counter;
  unsigned *err;
  unsigned long long *progress;  // one word per (pair, swath): progress[pair * max_swaths + s]
  T *bstat;                      // per (pair, reference swath boundary): shortcut value or -1
  unsigned long long max_bounds;
  T *edges;                      // two buffers of edge_stride elements per pair
  unsigned long long edge_stride;
  int open_start, open_end;      // all-vs-all modes (a list carries its own)
  unsigned long long limit_ns;
};

// One pair of a launch: its series (rows, columns), modes and output.  Without
// an open end the matrix of (b, a) is the transpose of (a, b)'s, in float with
// the same costs bit for bit (the differences change sign, the cell rule is
// symmetric), so the shorter series takes the rows: a pair's time is the steps
// down its rows plus about 200 steps for each swath after the first, and 1024
// columns cost less than 1024 rows.  Not in double: its compare-and-select
// minimum is not symmetric in NaN, so a pair with a NaN (or two infinities)
// would depend on the plan.  The same order of the minimum in a second copy of
// the sweep costs more than the exchange gives (15 series of 10000-30000: 24.4
// ms exchanged, 25.2 not, 27.9 with the copy).
//
// fits: the first series (before the exchange) is within the max_len the
// launch sized its edge buffers for; a longer one's edges would run into the
// next pair's buffers, so its pair is given NaN, as in the one-warp plans.
struct PipePair {
  int s, j, os, oe;
  unsigned long long out;
  uint64_t m, n;
  bool fits;
};
template <typename T>
__device__ __forceinline__ PipePair pipe_pair(const PipeArgs<T> &a, unsigned long long qi) {
  PipePair p;
  if (a.list) {
    const odba_pair_task task = a.list[qi];
    p.s = int(task.first);
    p.j = int(task.second);
    p.os = int((task.out >> 62) & 1ull);
    p.oe = int((task.out >> 63) & 1ull);
    p.out = task.out & ((1ull << 62) - 1);
  } else {
    const long long i = (long long)(a.pbeg + a.npairs - 1 - qi);
    pair_of(i, a.n, p.s, p.j);
    p.os = a.open_start;
    p.oe = a.open_end;
    p.out = (unsigned long long)i;
  }
  p.m = a.lens[p.s];
  p.n = a.lens[p.j];
  p.fits = p.m + 32 <= a.edge_stride;
  if (sizeof(T) == 4 && !p.os && !p.oe && p.m > p.n) {
    const int t = p.s;
    p.s = p.j;
    p.j = t;
    const uint64_t l = p.m;
    p.m = p.n;
    p.n = l;
  }
  return p;
}

// A block per swath (sweep_block).  TRACK: some pair may take the open-end
// shortcut (see sweep_pair).  A pair with more swaths than the launch counts
// (a list's second series may be longer than its longest first one) has the
// rest of them swept by the block of its last counted one, in turn.
template <typename T, bool TRACK>
__global__ void __launch_bounds__(kBlkThreads, sizeof(T) == 4 ? kPipeBlocksF32 : kPipeBlocksF64)
    swathpipe_kernel(PipeArgs<T> a) {
  __shared__ BlockSmem<T> sm;
  const int lane = threadIdx.x & 31;
  const bool feeder = (threadIdx.x >> 5) == kBlkWarps;
  const unsigned long long ntasks = a.npairs * a.max_swaths;
  // The turn of a pair's first swath: the last swaths of all pairs share the
  // last turn, so the longest chains start first (28 pairs of 40000-80000
  // samples: 13.95 ms with the first swaths in one turn, 13.3 so; 15 in double
  // of 30000-50000 17.2 and 16.6; 435 pairs of 200-900, one swath each, 172 us
  // both ways).
  auto late = [&](const PipePair &p) {
    const unsigned swaths = unsigned(p.n + kBlkCols - 1) / kBlkCols, most = unsigned(a.max_swaths);
    return swaths < most ? most - swaths : 0u;
  };
  for (;;) {
    if (feeder && lane == 0) {
      // the next task that exists
      unsigned long long q;
      for (;;) {
        q = atomicAdd(a.counter, 1ull);
        if (q >= ntasks) break;
        const unsigned long long turn = q / a.npairs;
        if (turn >= late(pipe_pair(a, q - turn * a.npairs))) break;
      }
      sm.task = q;
    }
    __syncthreads();
    const unsigned long long q = sm.task;
    if (q >= ntasks) break;
    const unsigned long long turn = q / a.npairs, qi = q - turn * a.npairs;
    const PipePair p = pipe_pair(a, qi);
    const unsigned long long first = turn - late(p);
    if (!p.fits) {
      if (first == 0 && threadIdx.x == 0) a.dists[p.out] = Num<T>::quiet_nan();
      __syncthreads();  // the task word is free again
      continue;
    }
    const int m = int(p.m), n = int(p.n);
    T *b0 = a.edges + qi * 2 * a.edge_stride;
    T *b1 = b0 + a.edge_stride;
    unsigned long long *words = a.progress + qi * a.max_swaths;
    const bool to_end = first + 1 == a.max_swaths;
    bool stop = false;  // the shortcut fired past the counted boundaries
    for (unsigned long long sw = first;; ++sw) {
      const int c0 = int(sw) * kBlkCols;
      const bool last = c0 + kBlkCols >= n;
      BlockJob<T> job;
      job.x = a.series + a.offsets[p.s];
      job.y = a.series + a.offsets[p.j];
      job.m = m;
      job.n = n;
      job.c0 = c0;
      job.r0 = p.os;
      job.edge_in = sw ? (((sw - 1) & 1) ? b1 : b0) : nullptr;
      job.edge_out = last ? nullptr : ((sw & 1) ? b1 : b0);
      job.open_end = p.oe != 0;
      job.free_diag0 = c0 > 0;
      job.corner_init = c0 == 0 ? (p.os ? Num<T>::big() : T(0)) : (p.os ? T(0) : Num<T>::big());
      job.words = nullptr;
      job.word_steps = 0;
      PipeGate gate;
      gate.prog_in = words + (first ? first - 1 : 0);
      gate.prog_out = words + first;
      gate.err = a.err;
      gate.limit_ns = a.limit_ns;
      gate.avail = sw == first ? 0 : 0x7fffffff;
      T corner = T(0);
      EdgeStat<T> st;
      bool mine = sweep_block<T, false, false, false, true>(
          job, sm, gate, CkptOut<T>{nullptr, 0, 1}, last, corner, st);
      if (TRACK && swath_checks_shortcut<T>(c0, kBlkCols, m, n, p.oe != 0, p.os)) {
        // this swath's right edge is the left edge of reference swath k + 1
        const unsigned long long k = sw;
        T v = T(-1);
        if (feeder && lane == 0) {
          if (!shortcut_fires<T>(st, m, v)) v = T(-1);
          if (k < a.max_bounds) a.bstat[qi * a.max_bounds + k] = v;
        }
        if (k >= a.max_bounds) {
          if (feeder && lane == 0) sm.task = v >= T(0) ? 1ull : 0ull;
          __syncthreads();
          if (sm.task) {
            stop = true;
            mine = feeder && lane == 0;
            corner = v;
          }
        }
      }
      if (m <= p.os && last) mine = threadIdx.x == 0;  // open start over a single row: all zeros
      if (mine) {
        const bool bad = *reinterpret_cast<volatile unsigned *>(a.err) != 0;
        a.dists[p.out] = bad ? T(NAN) : pair_distance<T>(corner, m, n, p.os, p.oe);
      }
      __syncthreads();  // the task word and the rings are free again
      if (last || stop || !to_end) break;
    }
  }
}

// Resident blocks of swathpipe_kernel on the current device (cached like
// grid_size).
template <typename T>
int pipe_grid() {
  static std::atomic<int> cached[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    const int c = cached[dev].load(std::memory_order_relaxed);
    if (c) return c;
  }
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, swathpipe_kernel<T, false>, kBlkThreads, 0);
  constexpr int want = sizeof(T) == 4 ? kPipeBlocksF32 : kPipeBlocksF64;
  if (per_sm > want) per_sm = want;
  if (per_sm < 1) per_sm = 1;
  if (sms < 1) sms = 1;
  const int g = sms * per_sm;
  if (dev >= 0 && dev < 64) cached[dev].store(g, std::memory_order_relaxed);
  return g;
}

// After the pipeline: a pair whose open-end shortcut fired on some checked
// edge takes its distance from the first such edge (the swaths after it ran
// anyway; the reference's stop there).  One thread per pair.
template <typename T>
__global__ void pipe_shortcut_kernel(PipeArgs<T> a) {
  const unsigned long long qi = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (qi >= a.npairs) return;
  if (*reinterpret_cast<volatile unsigned *>(a.err) != 0) return;
  const PipePair p = pipe_pair(a, qi);  // (never exchanged with an open end)
  if (!p.oe || p.os || !p.fits) return;
  const int m = int(p.m), n = int(p.n);
  for (int cnext = kRefSwath; cnext < n; cnext += kRefSwath) {
    if (cnext <= m) continue;
    if ((unsigned long long)(cnext / kRefSwath - 1) >= a.max_bounds) return;
    const T v = a.bstat[qi * a.max_bounds + (unsigned long long)(cnext / kRefSwath - 1)];
    if (v >= T(0)) {
      a.dists[p.out] = pair_distance<T>(v, m, n, p.os, p.oe);
      return;
    }
  }
}

}  // namespace

// counter and error word | progress words | shortcut values | edge buffers
template <typename T>
size_t swathpipe_progress_bytes(unsigned long long npairs, uint64_t max_len) {
  const unsigned long long max_swaths = (max_len + kBlkCols - 1) / kBlkCols;
  return (size_t(npairs) * max_swaths * 8 + 255) / 256 * 256;
}

inline unsigned long long swathpipe_max_bounds(uint64_t max_len) { return max_len / kRefSwath + 1; }

template <typename T>
size_t swathpipe_head_bytes(unsigned long long npairs, uint64_t max_len) {
  return 256 + swathpipe_progress_bytes<T>(npairs, max_len) +
         (size_t(npairs) * swathpipe_max_bounds(max_len) * sizeof(T) + 255) / 256 * 256;
}

template <typename T>
size_t swathpipe_workspace_bytes(unsigned long long npairs, uint64_t max_len) {
  const unsigned long long stride = (max_len + 32 + 31) / 32 * 32;
  return swathpipe_head_bytes<T>(npairs, max_len) + size_t(npairs) * 2 * stride * sizeof(T);
}

template <typename T>
int swathpipe_launch(const T *series, const uint64_t *offsets, const uint64_t *lens, int n,
                     const odba_pair_task *list, unsigned long long pbeg, unsigned long long npairs,
                     uint64_t max_len, int os, int oe, T *dists, void *workspace, size_t ws_bytes,
                     cudaStream_t stream, unsigned long long limit_ns) {
  if (npairs == 0) return ODBA_OK;
  if (ws_bytes < swathpipe_workspace_bytes<T>(npairs, max_len))
    return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "workspace too small for the swath pipeline");
  PipeArgs<T> a;
  a.series = series;
  a.offsets = offsets;
  a.lens = lens;
  a.n = n;
  a.list = list;
  a.pbeg = pbeg;
  a.npairs = npairs;
  a.max_swaths = (max_len + kBlkCols - 1) / kBlkCols;
  a.dists = dists;
  char *base = static_cast<char *>(workspace);
  a.counter = reinterpret_cast<unsigned long long *>(base);
  a.err = reinterpret_cast<unsigned *>(base + 8);
  a.progress = reinterpret_cast<unsigned long long *>(base + 256);
  a.bstat = reinterpret_cast<T *>(base + 256 + swathpipe_progress_bytes<T>(npairs, max_len));
  a.max_bounds = swathpipe_max_bounds(max_len);
  const size_t head = swathpipe_head_bytes<T>(npairs, max_len);
  a.edges = reinterpret_cast<T *>(base + head);
  a.edge_stride = (max_len + 32 + 31) / 32 * 32;
  a.open_start = os;
  a.open_end = oe;
  a.limit_ns = limit_ns ? limit_ns : kWaitLimitNs;
  // the shortcut values need no clearing: every checked edge writes its entry
  if (cudaMemsetAsync(base, 0, 256 + swathpipe_progress_bytes<T>(npairs, max_len), stream) != cudaSuccess)
    return fail(ODBA_ERR_CUDA, "clearing the pipeline state failed");
  const bool track = list || (oe && !os);
  const unsigned long long tasks = npairs * a.max_swaths;
  const int resident = pipe_grid<T>();
  const int grid = tasks < (unsigned long long)resident ? int(tasks) : resident;
  if (track) {
    swathpipe_kernel<T, true><<<grid, kBlkThreads, 0, stream>>>(a);
    pipe_shortcut_kernel<T><<<unsigned((npairs + 127) / 128), 128, 0, stream>>>(a);
  } else {
    swathpipe_kernel<T, false><<<grid, kBlkThreads, 0, stream>>>(a);
  }
  return check_launch("swath-pipelined DTW kernel");
}

template size_t swathpipe_workspace_bytes<float>(unsigned long long, uint64_t);
template size_t swathpipe_workspace_bytes<double>(unsigned long long, uint64_t);
template int swathpipe_launch<float>(const float *, const uint64_t *, const uint64_t *, int,
                                     const odba_pair_task *, unsigned long long, unsigned long long,
                                     uint64_t, int, int, float *, void *, size_t, cudaStream_t,
                                     unsigned long long);
template int swathpipe_launch<double>(const double *, const uint64_t *, const uint64_t *, int,
                                      const odba_pair_task *, unsigned long long, unsigned long long,
                                      uint64_t, int, int, double *, void *, size_t, cudaStream_t,
                                      unsigned long long);

}  // namespace odba

// ---------------------------------------------------------------------------
// Launch plans and the autotuner.
//
// Three plans compute the same distances (bit for bit): one warp per pair with
// 1024-column swaths (float; 512 for double), the same with half-width swaths,
// and the swath pipeline above (many warps per pair).  The plan is chosen per
// key (element size, floor(log2 max_len), floor(log2 pairs)): a plan pinned by
// odba_tune_set; else, in tuning mode, every eligible plan not yet measured for
// the key, in turn; else the fastest measured plan; else a rule of thumb
// (rule_of_thumb).  Measured throughput is pair-cells per
// second with max_len^2 per pair standing in for the cells (the lengths live
// on the device); CUDA events around each tuning launch are read back on the
// next call or by odba_tune_flush.
namespace odba {

namespace {

struct TuneCell {
  int pinned = 0;                        // a plan, or 0
  double rate[ODBA_PLAN_COUNT] = {0, 0, 0, 0};
};

struct Pending {
  int elem, lb, cb, plan;
  double cells;
  cudaEvent_t start, stop;
};

std::mutex g_tune_mu;
TuneCell g_tune[2][64][64];
bool g_tune_mode = false;
std::vector<Pending> g_pending;

int bucket_of(unsigned long long v) { return v ? 63 - __builtin_clzll(v) : 0; }

void harvest_locked(bool block) {
  std::vector<Pending> keep;
  for (auto &p : g_pending) {
    cudaError_t q = block ? cudaEventSynchronize(p.stop) : cudaEventQuery(p.stop);
    if (q == cudaErrorNotReady) {
      keep.push_back(p);
      continue;
    }
    float ms = 0;
    if (q == cudaSuccess && cudaEventElapsedTime(&ms, p.start, p.stop) == cudaSuccess && ms > 0) {
      double &r = g_tune[p.elem][p.lb][p.cb].rate[p.plan];
      const double rate = p.cells / (ms * 1e-3);
      if (rate > r) r = rate;
    } else {
      cudaGetLastError();
    }
    cudaEventDestroy(p.start);
    cudaEventDestroy(p.stop);
  }
  g_pending.swap(keep);
}

template <typename T>
bool plan_fits(int plan, unsigned long long npairs, uint64_t max_len, size_t ws_bytes) {
  const unsigned long long slots = (unsigned long long)grid_size<T>() * kWarpsPerBlock;
  switch (plan) {
    case ODBA_PLAN_WHOLE_PAIR:
    case ODBA_PLAN_WHOLE_PAIR_HALF_SWATH:
      return ws_bytes >= whole_workspace_bytes<T>(max_len);
    case ODBA_PLAN_SWATH_PIPELINE:
      return npairs <= 2 * slots && ws_bytes >= swathpipe_workspace_bytes<T>(npairs, max_len);
    default:
      return false;
  }
}

// The pipeline pays while its blocks are few enough to run a pair's swaths side
// by side: it takes a pair's steps a third to two thirds of the one-warp sweep's
// time, but fills the GPU with a third as many pairs, and a second swath that is
// nearly empty costs it a block all the same.  Series of up to 160 samples are
// swept by one warp in narrow lanes as fast.  Measured on one B200 (one-warp
// time / pipeline time, all pairs of n series), float:
//   2000-4000 samples  1128 / 1431 / 1770 pairs         1.54 / 1.28 / 1.18
//   1000-2000          1128 / 1431 / 1653 / 1770        1.40 / 1.14 / 1.03 / 0.97
//   1200-1500          780 / 946 / 1128 / 1431          1.33 / 1.16 / 1.00 / 0.77
//   900-1100           861 / 1035 / 1128                1.14 / 1.02 / 0.96
//   512-1024           861 / 1128 / 1431                1.21 / 1.09 / 0.85
//   150-400            435 / 630 / 780                  1.14 / 1.07 / 0.96
//   180-250            190 / 378 / 561                  1.09 / 1.07 / 0.96
//   129-160            66 / 378                         0.96 / 0.99
//   64-128             190 / 378                        0.86 / 0.86
//   20-40              190 / 435                        0.88 / 0.83
// double:
//   2000-4000          1431 / 1653 / 1770               1.53 / 1.39 / 1.13
//   1000-2000          1431 / 1653 / 1770               1.22 / 1.09 / 1.04
//   1200-1500          946 / 1128 / 1431                1.24 / 1.09 / 0.84
//   900-1100           861 / 1035 / 1128                1.23 / 1.05 / 0.94
//   512-1024           1035 / 1128 / 1431               1.23 / 1.05 / 0.94
//   150-400            435 / 630 / 780                  1.33 / 1.06 / 0.98
//   180-250            190 / 378 / 561                  1.13 / 1.14 / 0.72
//   129-160            66 / 378                         0.83 / 0.99
//   64-128             190 / 378                        0.78 / 0.78
// A pair list (reads against one or a few series) gains less: the one-warp kernel
// starts no more blocks than it has tasks for, the pipeline adds the launch that
// applies the open-end shortcut.  Reads against one series of their median
// length, float / double:
//   500-5000 samples   300 / 1200 tasks         2.66 / 1.22    2.66 / 1.43
//   1000-2000          300 / 700 / 1200         1.66 / 1.27 / 0.82    1.67 / 1.36 / 0.86
//   700-1000           100 / 300 / 700          1.42 / 1.20 / 0.81    1.57 / 1.31 / 0.98
//   512-700            100 / 300                1.10 / 0.96    1.25 / 1.04
//   300-500            30 / 300                 0.99 / 0.90    0.85 / 0.76
//   150-250            30 / 300                 0.80 / 0.78    0.67 / 0.66
// Above one pair per resident warp (1776) the workspace that does not know the
// number of pairs would not hold the pipeline's edges, so the rule ends there.
template <typename T>
int rule_of_thumb(unsigned long long npairs, uint64_t max_len, bool list = false) {
  const unsigned long long slots = (unsigned long long)grid_size<T>() * kWarpsPerBlock;
  const uint64_t swaths = (max_len + kBlkCols - 1) / kBlkCols;
  unsigned long long most;
  if (swaths >= 3)
    most = slots;
  else if (list)
    most = swaths == 2 ? slots / 2 : max_len >= 512 ? slots / 6 : 0;
  else if (swaths == 2)
    most = max_len < 1536 ? slots * 5 / 8 : sizeof(T) == 4 ? slots * 15 / 16 : slots;
  else if (max_len >= 256)
    most = max_len >= 512 ? slots * 2 / 3 : slots * 2 / 5;
  else
    most = max_len > 160 ? slots / 4 : 0;
  return npairs < most ? ODBA_PLAN_SWATH_PIPELINE : ODBA_PLAN_WHOLE_PAIR;
}

// Chooses the plan; *measure tells the caller to time the launch for the table.
template <typename T>
int choose_plan(unsigned long long npairs, uint64_t max_len, size_t ws_bytes, bool *measure,
                bool list = false) {
  const int e = sizeof(T) == 8 ? 1 : 0, lb = bucket_of(max_len), cb = bucket_of(npairs);
  std::lock_guard<std::mutex> g(g_tune_mu);
  harvest_locked(false);
  TuneCell &c = g_tune[e][lb][cb];
  *measure = false;
  if (c.pinned && plan_fits<T>(c.pinned, npairs, max_len, ws_bytes)) return c.pinned;
  if (g_tune_mode) {
    for (int p = 1; p < ODBA_PLAN_COUNT; ++p) {
      if (c.rate[p] > 0 || !plan_fits<T>(p, npairs, max_len, ws_bytes)) continue;
      bool queued = false;
      for (auto &q : g_pending)
        if (q.elem == e && q.lb == lb && q.cb == cb && q.plan == p) queued = true;
      if (queued) continue;
      *measure = true;
      return p;
    }
  }
  int best = 0;
  for (int p = 1; p < ODBA_PLAN_COUNT; ++p)
    if (c.rate[p] > 0 && plan_fits<T>(p, npairs, max_len, ws_bytes) && (!best || c.rate[p] > c.rate[best]))
      best = p;
  if (best) return best;
  const int r = rule_of_thumb<T>(npairs, max_len, list);
  if (plan_fits<T>(r, npairs, max_len, ws_bytes)) return r;
  for (int p = 1; p < ODBA_PLAN_COUNT; ++p)
    if (plan_fits<T>(p, npairs, max_len, ws_bytes)) return p;
  return 0;
}

template <typename T>
void record_pending(unsigned long long npairs, uint64_t max_len, int plan, cudaEvent_t a,
                    cudaEvent_t b) {
  std::lock_guard<std::mutex> g(g_tune_mu);
  g_pending.push_back(Pending{sizeof(T) == 8 ? 1 : 0, bucket_of(max_len), bucket_of(npairs), plan,
                              double(npairs) * double(max_len) * double(max_len), a, b});
}

template <typename T, typename F>
int run_planned(unsigned long long npairs, uint64_t max_len, size_t ws_bytes, cudaStream_t stream,
                bool list, F &&launch) {
  bool measure = false;
  const int plan = choose_plan<T>(npairs, max_len, ws_bytes, &measure, list);
  if (!plan) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "workspace too small");
  cudaEvent_t a = nullptr, b = nullptr;
  if (measure && (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess)) {
    cudaGetLastError();
    measure = false;
  }
  if (measure) cudaEventRecord(a, stream);
  const int rc = launch(plan);
  if (measure) {
    cudaEventRecord(b, stream);
    if (rc == ODBA_OK) {
      record_pending<T>(npairs, max_len, plan, a, b);
    } else {
      cudaEventDestroy(a);
      cudaEventDestroy(b);
    }
  }
  return rc;
}

}  // namespace

template <typename T>
size_t pairwise_workspace_bytes(uint64_t max_len) {
  // enough for every plan when there are at most as many pairs as resident warps
  const size_t slots = size_t(grid_size<T>()) * kWarpsPerBlock;
  return whole_workspace_bytes<T>(max_len) + swathpipe_head_bytes<T>(slots, max_len);
}

template <typename T>
size_t pairwise_workspace_bytes_n(unsigned long long npairs, uint64_t max_len) {
  const int r = rule_of_thumb<T>(npairs, max_len);
  return r == ODBA_PLAN_SWATH_PIPELINE ? swathpipe_workspace_bytes<T>(npairs, max_len)
                                       : whole_workspace_bytes<T>(max_len);
}

template <typename T>
int pairwise_range_launch(const T *series, const uint64_t *offsets, const uint64_t *lens, int n,
                          uint64_t max_len, int os, int oe, unsigned long long pbeg,
                          unsigned long long pend, T *dists, void *workspace, size_t ws_bytes,
                          cudaStream_t stream) {
  if (n < 2 || pend <= pbeg) return ODBA_OK;
  const unsigned long long npairs = pend - pbeg;
  return run_planned<T>(npairs, max_len, ws_bytes, stream, false, [&](int plan) {
    switch (plan) {
      case ODBA_PLAN_WHOLE_PAIR_HALF_SWATH:
        return whole_pairwise_launch<T, Tune<T>::RF / 2>(series, offsets, lens, n, max_len, os, oe,
                                                          pbeg, npairs, dists, workspace, ws_bytes,
                                                          stream);
      case ODBA_PLAN_SWATH_PIPELINE:
        return swathpipe_launch<T>(series, offsets, lens, n, nullptr, pbeg, npairs, max_len, os, oe,
                                   dists, workspace, ws_bytes, stream, 0);
      default:
        return whole_pairwise_launch<T, Tune<T>::RF>(series, offsets, lens, n, max_len, os, oe,
                                                      pbeg, npairs, dists, workspace, ws_bytes,
                                                      stream);
    }
  });
}

template <typename T>
int pairwise_launch(const T *series, const uint64_t *offsets, const uint64_t *lens, int n,
                    uint64_t max_len, int os, int oe, T *dists, void *workspace, size_t ws_bytes,
                    cudaStream_t stream) {
  if (n < 2) return ODBA_OK;
  return pairwise_range_launch<T>(series, offsets, lens, n, max_len, os, oe, 0,
                                  (unsigned long long)n * (n - 1) / 2, dists, workspace, ws_bytes,
                                  stream);
}

template <typename T>
int pairlist_launch(const T *series, const uint64_t *offsets, const uint64_t *lens,
                    const odba_pair_task *tasks, unsigned long long ntasks, uint64_t max_len,
                    T *dists, void *workspace, size_t ws_bytes, cudaStream_t stream) {
  if (ntasks == 0) return ODBA_OK;
  return run_planned<T>(ntasks, max_len, ws_bytes, stream, true, [&](int plan) {
    switch (plan) {
      case ODBA_PLAN_WHOLE_PAIR_HALF_SWATH:
        return whole_pairlist_launch<T, Tune<T>::RF / 2>(series, offsets, lens, tasks, ntasks,
                                                          max_len, dists, workspace, ws_bytes, stream);
      case ODBA_PLAN_SWATH_PIPELINE:
        return swathpipe_launch<T>(series, offsets, lens, 0, tasks, 0, ntasks, max_len, 0, 0, dists,
                                   workspace, ws_bytes, stream, 0);
      default:
        return whole_pairlist_launch<T, Tune<T>::RF>(series, offsets, lens, tasks, ntasks, max_len,
                                                      dists, workspace, ws_bytes, stream);
    }
  });
}

namespace {
// The self-test's buffer: the error word, the progress words, samples, an edge.
constexpr int kSelfRows = 64, kSelfCols = 1024 + 300;
struct SelfTest {
  unsigned err[4];
  unsigned long long prog[2];
  float x[kSelfRows], y[kSelfCols], edge[kSelfRows + 32];
};

// A block sweeps the second swath of a pair whose first swath nobody sweeps:
// the pipeline's own wait on a progress word that nothing publishes.
__device__ __forceinline__ BlockJob<float> selftest_job(SelfTest *t) {
  BlockJob<float> job;
  job.x = t->x;
  job.y = t->y;
  job.m = kSelfRows;
  job.n = kSelfCols;
  job.c0 = kBlkCols;
  job.r0 = 0;
  job.edge_in = t->edge;
  job.edge_out = nullptr;
  job.open_end = false;
  job.free_diag0 = true;
  job.corner_init = Num<float>::big();
  job.words = nullptr;
  job.word_steps = 0;
  return job;
}
__global__ void __launch_bounds__(kBlkThreads) gate_selftest_kernel(SelfTest *t,
                                                                    unsigned long long limit_ns) {
  __shared__ BlockSmem<float> sm;
  PipeGate gate;
  gate.prog_in = t->prog;
  gate.prog_out = t->prog + 1;
  gate.err = t->err;
  gate.limit_ns = limit_ns;
  gate.avail = 0;
  float corner = 0.f;
  EdgeStat<float> st;
  sweep_block<float, false, false, false, true>(selftest_job(t), sm, gate,
                                                CkptOut<float>{nullptr, 0, 1}, true, corner, st);
}

// The same swath with nothing to wait for outside the block, by the compute
// warps alone (kBlkThreads - 32 threads): their wait for a feeder that is not
// there.
__global__ void __launch_bounds__(kBlkThreads) block_selftest_kernel(SelfTest *t,
                                                                     unsigned long long limit_ns) {
  __shared__ BlockSmem<float> sm;
  float corner = 0.f;
  EdgeStat<float> st;
  sweep_block<float, false, false, false, true>(selftest_job(t), sm, NoGate(t->err + 1, limit_ns),
                                                CkptOut<float>{nullptr, 0, 1}, true, corner, st);
}

// The same swath by one warp (the one-warp pipeline of the rounds).
__global__ void __launch_bounds__(32) warp_selftest_kernel(SelfTest *t, unsigned long long limit_ns) {
  __shared__ WarpSmem<float> sm;
  const BlockJob<float> b = selftest_job(t);
  SwathJob<float> job;
  job.x = b.x;
  job.y = b.y;
  job.m = b.m;
  job.n = b.n;
  job.c0 = b.c0;
  job.r0 = b.r0;
  job.edge_in = b.edge_in;
  job.edge_out = nullptr;
  job.open_end = false;
  job.free_diag0 = true;
  job.corner_init = b.corner_init;
  PipeGate gate;
  gate.prog_in = t->prog;
  gate.prog_out = t->prog + 1;
  gate.err = t->err + 2;
  gate.limit_ns = limit_ns;
  gate.avail = 0;
  float corner = 0.f;
  sweep_warp<float, 16, false, PipeGate>(job, sm, true, corner, gate);
}
}  // namespace

int gate_selftest(unsigned long long limit_ns, cudaStream_t stream) {
  if (limit_ns == 0 || limit_ns > 10000000000ull)
    return fail(ODBA_ERR_INVALID_ARGUMENT, "limit must be in (0, 10 s]");
  if (int rc = require_sm100()) return rc;
  SelfTest *t = nullptr;
  if (cudaMallocAsync(reinterpret_cast<void **>(&t), sizeof *t, stream) != cudaSuccess)
    return fail(ODBA_ERR_OUT_OF_MEMORY, "self-test buffer");
  unsigned err[4] = {0u, 0u, 0u, 0u};
  cudaMemsetAsync(t, 0, sizeof *t, stream);
  gate_selftest_kernel<<<1, kBlkThreads, 0, stream>>>(t, limit_ns);
  block_selftest_kernel<<<1, kBlkThreads - 32, 0, stream>>>(t, limit_ns);
  warp_selftest_kernel<<<1, 32, 0, stream>>>(t, limit_ns);
  int rc = check_launch("wait self-test kernel");
  cudaMemcpyAsync(err, t->err, sizeof err, cudaMemcpyDeviceToHost, stream);
  cudaFreeAsync(t, stream);
  if (cudaStreamSynchronize(stream) != cudaSuccess) return fail(ODBA_ERR_CUDA, "wait self-test");
  if (rc) return rc;
  if (err[0] && err[1] && err[2]) return fail(ODBA_ERR_TIMEOUT, "the waits ran out and raised the error words");
  return fail(ODBA_ERR_CUDA, !err[0]   ? "the wait returned without the word or a timeout"
                             : !err[1] ? "a wait inside a block returned without a timeout"
                                       : "the one-warp wait returned without a timeout");
}

int tune_set(int elem_size, int len_bucket, int count_bucket, int plan) {
  if ((elem_size != 4 && elem_size != 8) || len_bucket < 0 || len_bucket > 63 || count_bucket < 0 ||
      count_bucket > 63 || plan < 0 || plan >= ODBA_PLAN_COUNT)
    return fail(ODBA_ERR_INVALID_ARGUMENT, "bad tuning key or plan");
  std::lock_guard<std::mutex> g(g_tune_mu);
  g_tune[elem_size == 8][len_bucket][count_bucket].pinned = plan;
  return ODBA_OK;
}

int tune_query(int elem_size, uint64_t max_len, unsigned long long npairs, size_t ws_bytes, int *plan,
               double *rates) {
  if (elem_size != 4 && elem_size != 8) return fail(ODBA_ERR_INVALID_ARGUMENT, "elem_size must be 4 or 8");
  bool measure = false;
  const int p = elem_size == 8 ? choose_plan<double>(npairs, max_len, ws_bytes, &measure)
                               : choose_plan<float>(npairs, max_len, ws_bytes, &measure);
  if (plan) *plan = p;
  if (rates) {
    std::lock_guard<std::mutex> g(g_tune_mu);
    const TuneCell &c = g_tune[elem_size == 8][bucket_of(max_len)][bucket_of(npairs)];
    for (int i = 0; i < ODBA_PLAN_COUNT; ++i) rates[i] = c.rate[i];
  }
  return ODBA_OK;
}

void tune_mode(int on) {
  std::lock_guard<std::mutex> g(g_tune_mu);
  g_tune_mode = on != 0;
}

int tune_flush() {
  std::lock_guard<std::mutex> g(g_tune_mu);
  harvest_locked(true);
  return ODBA_OK;
}

int tune_save(const char *path) {
  std::lock_guard<std::mutex> g(g_tune_mu);
  harvest_locked(true);
  FILE *f = std::fopen(path, "w");
  if (!f) return fail(ODBA_ERR_IO, "cannot write the tuning table");
  std::fprintf(f, "# elem len_bucket count_bucket pinned rate_whole rate_half rate_pipeline\n");
  for (int e = 0; e < 2; ++e)
    for (int l = 0; l < 64; ++l)
      for (int c = 0; c < 64; ++c) {
        const TuneCell &t = g_tune[e][l][c];
        if (!t.pinned && !t.rate[1] && !t.rate[2] && !t.rate[3]) continue;
        std::fprintf(f, "%d %d %d %d %.6e %.6e %.6e\n", e ? 8 : 4, l, c, t.pinned, t.rate[1],
                     t.rate[2], t.rate[3]);
      }
  std::fclose(f);
  return ODBA_OK;
}

int tune_load(const char *path) {
  FILE *f = std::fopen(path, "r");
  if (!f) return fail(ODBA_ERR_IO, "cannot read the tuning table");
  std::lock_guard<std::mutex> g(g_tune_mu);
  char line[512];
  int rc = ODBA_OK;
  while (std::fgets(line, sizeof line, f)) {
    if (line[0] == '#' || line[0] == '\n') continue;
    int e, l, c, pin;
    double r1, r2, r3;
    if (std::sscanf(line, "%d %d %d %d %lf %lf %lf", &e, &l, &c, &pin, &r1, &r2, &r3) != 7 ||
        (e != 4 && e != 8) || l < 0 || l > 63 || c < 0 || c > 63 || pin < 0 || pin >= ODBA_PLAN_COUNT) {
      rc = fail(ODBA_ERR_IO, "malformed tuning table line");
      break;
    }
    TuneCell &t = g_tune[e == 8][l][c];
    t.pinned = pin;
    t.rate[1] = r1;
    t.rate[2] = r2;
    t.rate[3] = r3;
  }
  std::fclose(f);
  return rc;
}

template size_t pairwise_workspace_bytes<float>(uint64_t);
template size_t pairwise_workspace_bytes<double>(uint64_t);
template size_t pairwise_workspace_bytes_n<float>(unsigned long long, uint64_t);
template size_t pairwise_workspace_bytes_n<double>(unsigned long long, uint64_t);
template int pairwise_launch<float>(const float *, const uint64_t *, const uint64_t *, int,
                                    uint64_t, int, int, float *, void *, size_t, cudaStream_t);
template int pairwise_range_launch<float>(const float *, const uint64_t *, const uint64_t *, int,
                                          uint64_t, int, int, unsigned long long, unsigned long long,
                                          float *, void *, size_t, cudaStream_t);
template int pairwise_range_launch<double>(const double *, const uint64_t *, const uint64_t *, int,
                                           uint64_t, int, int, unsigned long long, unsigned long long,
                                           double *, void *, size_t, cudaStream_t);
template int pairwise_launch<double>(const double *, const uint64_t *, const uint64_t *, int,
                                     uint64_t, int, int, double *, void *, size_t, cudaStream_t);
template int pairlist_launch<float>(const float *, const uint64_t *, const uint64_t *,
                                    const odba_pair_task *, unsigned long long, uint64_t, float *,
                                    void *, size_t, cudaStream_t);
template int pairlist_launch<double>(const double *, const uint64_t *, const uint64_t *,
                                     const odba_pair_task *, unsigned long long, uint64_t,
                                     double *, void *, size_t, cudaStream_t);

}  // namespace odba
