// One DBA round on the device: DBAUpdate (dba.hpp:432-848) with the centroid
// update of updateCentroid (dba.hpp:374-423), for all members in one pass.
//
//  1. plan:      per member the orientation (the centroid goes on the Y axis
//                when open_end and it is the shorter one, dba.hpp:497-501),
//                the size and offset of its 2-bit path, and its path-file slot.
//  2. path DTW:  persistent launch, a block per swath (dtw_block.cuh) or, in
//                large rounds, a warp (dtw_warp.cuh); records every move and
//                the right-edge minima the open-end shortcut needs.
//  3. backtrack: one warp per member walks its path from the end cell back to
//                (0, 0) (updateCentroid's loop) and stores, per centroid index,
//                the contiguous range of member samples that index receives --
//                a path crosses every centroid index in one contiguous run.
//                Optionally it also emits the path as (i, j, move) triples in
//                the order of the reference's path file (io_utils.hpp:287-323).
//  4. reduce:    one warp per centroid index adds the member samples in the
//                reference's exact order -- members in order, each member's
//                samples from its last path row down to its first -- then
//                divides by the pile-up count in T (dba.hpp:820-822) and takes
//                max |old - new| in double (dba.hpp:830-836).
// The float sums are therefore bit-identical to the reference's serialized
// single-thread atomicAdd sequence, without atomics.
#include <cuda_runtime.h>

#include <atomic>
#include <climits>
#include <cstdint>
#include <vector>

#include "dtw_block.cuh"
#include "dtw_path.cuh"
#include "dtw_pipe.cuh"
#include "dtw_warp.cuh"
#include "odba_internal.h"

namespace odba {

namespace {

constexpr int kRoundWarps = 4;
constexpr int kReduceWarps = 4;  // centroid indices per block of the ordered reducer
constexpr int kReduceThreads = kReduceWarps * 32;
constexpr int kReduceBlocksF32 = 6, kReduceBlocksF64 = 4;
constexpr int kPlanThreads = 1024;  // members per step of the plan's prefix sums
constexpr int kRankMembers = 16384;  // longest-first task order computed up to this many members
// move codes of the reference's path matrix (dtw.hpp:10-16); kMoveDiag,
// kMoveRight and kMoveUp come with the path sweep (dtw_path.cuh)
constexpr int kMaxMoveNil = 255, kMoveOpenRight = 4, kMoveNilOpenRight = 5;

// Non-negative costs order like their bit patterns.
template <typename T>
struct CostBits;
template <>
struct CostBits<float> {
  using U = unsigned;
  static __device__ __forceinline__ U of(float v) { return __float_as_uint(v); }
};
template <>
struct CostBits<double> {
  using U = unsigned long long;
  static __device__ __forceinline__ U of(double v) { return (U)__double_as_longlong(v); }
};

// Geometry of one member's cost matrix, identical on host and device.
struct MemberGeom {
  int flip, m, n, r0, swaths, steps;
  unsigned long long words;
};

template <typename T>
__host__ __device__ inline MemberGeom member_geom(uint64_t len, uint64_t Lc, int os, int oe,
                                                  int centroid_rows = 0) {
  MemberGeom g;
  g.flip = ((oe && Lc < len) || centroid_rows) ? 1 : 0;
  g.m = int(g.flip ? Lc : len);
  g.n = int(g.flip ? len : Lc);
  g.r0 = os ? 1 : 0;
  g.swaths = (g.n + kBlkCols - 1) / kBlkCols;
  g.steps = block_steps(g.m - g.r0);
  g.words = (unsigned long long)g.swaths * g.steps * 64ull;
  return g;
}

// Rows of a swath-pipeline task.  With nbands > 1 each member's rows r0 ..
// m-1 are cut into bands of an even height of at least kMinBandRows (so a
// band's steps are the whole swath's steps from (rb - r0) / 2 on); count is
// the member's number of bands, band b covers rows rb .. re-1.
constexpr int kMinBandRows = 1024;
struct Band {
  int rb, re, count;
};
__host__ __device__ inline Band member_band(const MemberGeom &g, int nbands, int b) {
  const int rows = g.m - g.r0;
  Band o;
  int h = rows;
  if (nbands > 1 && rows > 0) {
    h = (rows + nbands - 1) / nbands;
    h = (h + 1) & ~1;
    if (h < kMinBandRows) h = kMinBandRows;
  }
  o.count = (rows > 0 && h > 0) ? (rows + h - 1) / h : 1;
  o.rb = g.r0 + b * h;
  o.re = b >= o.count - 1 ? g.m : o.rb + h;
  return o;
}

// Jobs share one launch: job J owns centroid centroids[coff[J] .. + clen[J]),
// flags (bit 0 open start, bit 1 open end, bit 2 active, bit 3 centroid on
// the rows whatever the lengths -- the prefix-chop orientation) and the members
// job_mbeg[J] .. job_mend[J]-1 of the member list (member k is series
// mem_series[k] of the series table).  Members of a job are contiguous and in
// the job's order, which is the order their samples are added.
template <typename T>
struct RoundArgs {
  const T *centroids;
  const unsigned long long *coff;
  const int *clen;
  const int *jflags;
  const int *mbeg, *mend;
  int njobs;
  const T *series;
  const uint64_t *offsets;
  const uint64_t *lens;
  const int *mseries, *mjob, *order;
  int nmem;
  unsigned long long *counter;
  unsigned long long *path_off;  // word offset of member k's path
  unsigned long long *trip_off;  // triple offset of member k's path listing
  unsigned long long *rng_off;   // offset of member k's per-centroid-index ranges
  // backtrack without a path listing: per member, per row, the column
  // interval of the row's contributing cells (runs_off[k] = member k's first)
  unsigned long long *runs_off = nullptr;
  int2 *runs = nullptr;
  int *shortcut;                 // first column of the open-end shortcut, or 0
  int2 *ranges;
  T *edges;
  unsigned long long edge_stride;
  unsigned long long *words;
  // swath pipeline (many warps per member): one progress word and the right
  // edge's minimum and top-row value per (member, swath)
  unsigned long long *prog;
  T *emtop;  // per (band, member, swath)
  unsigned *err;
  int max_swaths;
  int one_warp = 0;  // a warp per swath, whose moves are laid out as WarpMap has them
  // row bands of the swath pipeline (member_band): per (member, swath) the
  // last row and edge corner of the band done so far, and that band's count
  int nbands = 1;
  T *rowbuf = nullptr;
  unsigned long long *bdone = nullptr;
  // the backtrack's row walk inside the path DTW: a member's last task to
  // finish walks its path (per member, the count of its tasks done)
  int walk_in_sweep = 0;
  unsigned long long *mdone = nullptr;
  T *means;
  uint32_t *counts;
  double *deltas;
  int32_t *triples;
  int64_t *triple_counts;
  // stripe mode with an open end: one more sample index per (member, centroid
  // index), added after its range (-1: none)
  const int *extra = nullptr;
};

template <typename T>
__device__ __forceinline__ MemberGeom geom_of(const RoundArgs<T> &a, int k, int &job) {
  job = a.mjob[k];
  const int f = a.jflags[job];
  return member_geom<T>(a.lens[a.mseries[k]], uint64_t(a.clen[job]), f & 1, (f >> 1) & 1,
                        (f >> 3) & 1);
}

// Members of inactive jobs take no path words and no ranges (a caller can run
// a large set of jobs in waves with a workspace sized for one wave); the path
// listing keeps a slot for every member so its layout does not depend on the
// flags.
template <typename T>
__global__ void __launch_bounds__(kPlanThreads) plan_kernel(RoundArgs<T> a) {
  // exclusive prefix sums over the members, kPlanThreads at a time: path
  // words, path-listing triples (every member), ranges and rows (active
  // members only)
  __shared__ unsigned long long s_warp[4][kPlanThreads / 32];
  __shared__ unsigned long long s_carry[4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x < 4) s_carry[threadIdx.x] = 0;
  __syncthreads();
  for (int base = 0; base < a.nmem; base += kPlanThreads) {
    const int k = base + threadIdx.x;
    unsigned long long v[4] = {0ull, 0ull, 0ull, 0ull}, x[4];
    if (k < a.nmem) {
      int job;
      const MemberGeom g = geom_of<T>(a, k, job);
      v[1] = (unsigned long long)(g.m + g.n + 1);
      if (a.jflags[job] & 4) {
        v[0] = g.words;
        v[2] = (unsigned long long)a.clen[job];
        v[3] = (unsigned long long)g.m;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      x[q] = v[q];
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long y = __shfl_up_sync(kFull, x[q], off);
        if (lane >= off) x[q] += y;
      }
      if (lane == 31) s_warp[q][wid] = x[q];
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const unsigned long long t = lane < kPlanThreads / 32 ? s_warp[q][lane] : 0ull;
        unsigned long long y = t;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const unsigned long long z = __shfl_up_sync(kFull, y, off);
          if (lane >= off) y += z;
        }
        if (lane < kPlanThreads / 32) s_warp[q][lane] = y - t;  // exclusive over warps
      }
    }
    __syncthreads();
    unsigned long long ex[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) ex[q] = s_carry[q] + s_warp[q][wid] + x[q] - v[q];
    if (k < a.nmem) {
      a.path_off[k] = ex[0];
      a.trip_off[k] = ex[1];
      a.rng_off[k] = ex[2];
      if (a.runs_off) a.runs_off[k] = ex[3];
    }
    __syncthreads();
    // the last thread's inclusive sums are the next chunk's carries
    if (threadIdx.x == kPlanThreads - 1) {
#pragma unroll
      for (int q = 0; q < 4; ++q) s_carry[q] = ex[q] + v[q];
    }
    __syncthreads();
  }
  for (int j = threadIdx.x; j < a.njobs; j += kPlanThreads)
    if (a.jflags[j] & 4) a.deltas[j] = 0.0;
}

// Longest first: member k's place in the swath pipeline's task order is the
// number of members with more rows, or as many and a lower index (inactive
// members last).  The last tasks taken, and with the row walk in the sweep
// the last walks, are then the shortest.  Rows come in tiles of the block's
// size through shared memory.
template <typename T>
__global__ void __launch_bounds__(256) rank_members_kernel(RoundArgs<T> a, int *order) {
  __shared__ int s_rows[256];
  auto rows_of = [&](int i) {
    int jb;
    const MemberGeom g = geom_of<T>(a, i, jb);
    return (a.jflags[jb] & 4) ? g.m : -1;
  };
  const int k = blockIdx.x * 256 + threadIdx.x;
  const int mine = k < a.nmem ? rows_of(k) : -1;
  int rank = 0;
  for (int base = 0; base < a.nmem; base += 256) {
    const int i = base + threadIdx.x;
    s_rows[threadIdx.x] = i < a.nmem ? rows_of(i) : -1;
    __syncthreads();
    const int lim = a.nmem - base < 256 ? a.nmem - base : 256;
    for (int u = 0; u < lim; ++u) {
      const int ri = s_rows[u];
      rank += int(ri > mine) | int(ri == mine && base + u < k);
    }
    __syncthreads();
  }
  if (k < a.nmem) order[rank] = k;
}

__global__ void fill_ranges_kernel(int2 *r, unsigned long long count) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < count;
       i += (unsigned long long)gridDim.x * blockDim.x)
    r[i] = make_int2(1, 0);
}

// The open-end shortcut of swath-pipeline member k, from the per-swath
// right-edge minima (a swath's minimum is the least of its bands', its top-row
// value the top band's, the other bands leaving theirs at big).  The reference
// checks, at every swath start past the first series' length, whether the top
// row already holds the column minimum; from the first hit on, the rest of the
// top row is OPEN_RIGHT: the first qualifying swath boundary, or 0.
template <typename T>
__device__ __forceinline__ int member_shortcut(const RoundArgs<T> &a, int k, const MemberGeom &g,
                                               int flags, int cols) {
  const int os = flags & 1, oe = (flags >> 1) & 1;
  if (!oe || os) return 0;
  const int nb = member_band(g, a.nbands, 0).count;
  const unsigned long long layer = (unsigned long long)a.nmem * a.max_swaths;
  for (int s = 0; (s + 1) * cols < g.n; ++s) {
    const int cnext = (s + 1) * cols;  // (a swath of `cols` columns)
    if (cnext % kRefSwath || cnext <= g.m) continue;
    T emin = Num<T>::big(), etop = Num<T>::big();
    for (int b = 0; b < nb; ++b) {
      const T *et = a.emtop + ((unsigned long long)b * layer + (unsigned long long)k * a.max_swaths + s) * 2;
      emin = Num<T>::min2(emin, et[0]);
      etop = Num<T>::min2(etop, et[1]);
    }
    if (etop == emin) return cnext;
  }
  return 0;
}

// The moves of one row's 32 columns cb .. cb + 31 (cb a multiple of 32): bit
// j of d (u) is column cb + j's D (U) bit.
struct RowMoves {
  unsigned d, u;
};

// Where a matrix's moves are, as the block sweep lays them out (from column cmin,
// a multiple of the swath, on): four lanes of 8 columns hold a row's 32 columns,
// each a step behind its left neighbour.  Rows r >= 1.
struct BlockMap {
  const unsigned short *w;
  int r0, steps, cmin;
  struct At {
    const unsigned short *p;
  };
  __device__ __forceinline__ At at(int r, int cb) const {
    const int k = r - r0, l = ((cb - cmin) / kBlkR) & 31;
    return At{w + (((size_t)((cb - cmin) / kBlkWarpCols) * steps + (k >> 1) + l) * 32 + l) * 2 + (k & 1)};
  }
  // the 32 columns cb .. to the left of a's, and the rows 32 below a's
  __device__ __forceinline__ At left(At a, int r, int cb) const {
    return ((cb - cmin + 32) & (kBlkWarpCols - 1)) ? At{a.p - 4 * 66} : at(r, cb);
  }
  static __device__ __forceinline__ At below(At a) { return At{a.p - 16 * 64}; }
  static __device__ __forceinline__ RowMoves load(At a) {
    const unsigned lo = unsigned(a.p[0]) | unsigned(a.p[66]) << 16;
    const unsigned hi = unsigned(a.p[132]) | unsigned(a.p[198]) << 16;
    return RowMoves{__byte_perm(lo, hi, 0x6420), __byte_perm(lo, hi, 0x7531)};
  }
};

// The one-warp sweep: columns per lane of a full swath, and of a last one of
// `width` columns (the least of 8, 16 and 32 that covers it: a row's 32 columns
// are then 1, 2 or 4 lanes').
template <typename T>
constexpr int kWarpR = sizeof(T) == 4 ? 32 : 16;
template <typename T>
__host__ __device__ inline int warp_cols() {
  return 32 * kWarpR<T>;
}
template <typename T>
__host__ __device__ inline int warp_regs(int width) {
  return width <= 256 ? 8 : width <= 512 ? 16 : kWarpR<T>;
}
template <typename T>
struct WarpMap {
  static constexpr int KW = WarpMoves<T>::kWords;
  const unsigned *w;
  int r0, steps, n;
  struct At {
    const unsigned *p;
    int lanes;
  };
  __device__ __forceinline__ At at(int r, int cb) const {
    const int k = r - r0, s = cb / warp_cols<T>(), c = cb - s * warp_cols<T>();
    const int R = warp_regs<T>(n - cb + c), l = c / R;
    return At{w + (((size_t)s * steps + (k >> 1) + l) * 64 + l * 2 + (k & 1)) * KW, 32 / R};
  }
  __device__ __forceinline__ At left(At a, int r, int cb) const {
    return (cb + 32) % warp_cols<T>() ? At{a.p - a.lanes * 66 * KW, a.lanes} : at(r, cb);
  }
  static __device__ __forceinline__ At below(At a) { return At{a.p - 16 * 64 * KW, a.lanes}; }
  static __device__ __forceinline__ RowMoves load(At a) {
    RowMoves m{0u, 0u};
    const int R = 32 / a.lanes;
    for (int i = 0; i < a.lanes; ++i) {
      const unsigned *p = a.p + i * 66 * KW;
      const unsigned d = KW == 2 ? p[0] : p[0] & 0xffffu, u = KW == 2 ? p[1] : p[0] >> 16;
      m.d |= d << (i * R);
      m.u |= u << (i * R);
    }
    return m;
  }
};

template <typename T>
__device__ __forceinline__ BlockMap block_map(const RoundArgs<T> &a, const MemberGeom &g, int k) {
  return BlockMap{reinterpret_cast<const unsigned short *>(a.words + a.path_off[k]), g.r0, g.steps, 0};
}
template <typename T>
__device__ __forceinline__ WarpMap<T> warp_map(const RoundArgs<T> &a, const MemberGeom &g, int k) {
  return WarpMap<T>{reinterpret_cast<const unsigned *>(a.words + a.path_off[k]), g.r0, g.steps, g.n};
}

template <typename T, typename Map>
__device__ __forceinline__ bool walk_member_runs(const RoundArgs<T> &a, const Map &map,
                                                 const MemberGeom &g, int k, int os, int oe,
                                                 int2 *runs);

// Path DTW, a block per swath (sweep_block): task q is band
// q / (nmem * max_swaths) of a swath of the (q % nmem)-th member in alignment
// order, in turn (q / nmem) % max_swaths, so a member's swaths run in different
// blocks at once (few or long members keep the GPU busy).  The last swaths of
// all members share the last turn: a member of one swath does not go before the
// second swath of a longer one, whose chain ends later (690 members of 200-2000
// samples in 24 jobs, three blocks per SM: 480 us with the first swaths in one
// turn, 441 so; where all members have the same swaths nothing changes).  The right edge of swath s
// goes to buffer s % 2 of the member with one progress word per (member,
// swath), as in the all-pairs swath pipeline.  BAND (odba_round_set_bands,
// member_band): a band starts from the last row and edge corner the band below
// left in the (member, swath)'s row buffer, once that band has raised the
// (member, swath)'s band word; the recorded moves are the same.  Each band
// also stores its right edge's minimum and top-row value for the open-end
// shortcut, which never changes a recorded move.  Every wait is on a task
// taken earlier from the counter.
//
// The block's cost per cell is the one-warp sweep's plus about 14 instructions
// per 16 cells (loads of samples and edge, shuffles, stores); what it buys is
// a step a quarter as long where a member's chain of swaths, and not the GPU's
// throughput, sets a round's time.  One B200, one warp per swath against a
// block per swath: 64 members of 512-1024 samples 0.73 -> 0.29 ms a round, 100
// of 1000-4000 in double 2.51 -> 1.53, 400 of 3000-8000 (which fill the GPU)
// 6.57 -> 5.86.
//
// Blocks per SM: four (two for double).  More, which the registers would allow,
// only spread the issue slots over more chains, and each chain's last swath then
// ends later; three are a little better where one wave of chains is all there
// is, but lose on larger rounds.  Float, with three / four / five / six: 400
// members of 3000-8000 samples 5.79 / 5.86 / 6.24 / 6.54 ms, 600 8.61 / 8.11 /
// 8.39 / 8.67, 1000 13.75 / 12.95 / 13.06 / 13.09, 512 of 1000-2000 (open end)
// 1.10 / 1.00 / 1.07 / 1.14; double 1.71 with four, 1.53 with two.
constexpr int kRoundBlocksF32 = 4, kRoundBlocksF64 = 2;
template <typename T, bool BAND>
__global__ void
__launch_bounds__(kBlkThreads, sizeof(T) == 4 ? kRoundBlocksF32 : kRoundBlocksF64)
    path_block_kernel(RoundArgs<T> a) {
  __shared__ BlockSmem<T> sm;
  const int lane = threadIdx.x & 31;
  const bool feeder = (threadIdx.x >> 5) == kBlkWarps;
  const unsigned long long layer = (unsigned long long)a.nmem * a.max_swaths;
  const unsigned long long ntasks = layer * a.nbands;
  auto member_of = [&](unsigned long long qi) {
    return a.order ? a.order[qi] : a.nmem - 1 - int(qi);
  };
  // the turn of a member's first swath
  auto late = [&](const MemberGeom &g) { return g.swaths < a.max_swaths ? a.max_swaths - g.swaths : 0; };
  for (;;) {
    if (feeder && lane == 0) {
      // the next task that exists
      unsigned long long q;
      for (;;) {
        q = atomicAdd(a.counter, 1ull);
        if (q >= ntasks) break;
        const unsigned long long ql = q % layer;
        int jb;
        const MemberGeom g = geom_of<T>(a, member_of(ql % a.nmem), jb);
        if (!(a.jflags[jb] & 4)) continue;
        if ((unsigned)(int(ql / a.nmem) - late(g)) >= (unsigned)g.swaths) continue;
        if (BAND && int(q / layer) >= member_band(g, a.nbands, 0).count) continue;
        break;
      }
      sm.task = q;
    }
    __syncthreads();
    const unsigned long long q = sm.task;
    if (q >= ntasks) break;
    const int b = BAND ? int(q / layer) : 0;
    const unsigned long long ql = q - (unsigned long long)b * layer;
    const int turn = int(ql / a.nmem);
    const int k = member_of(ql - (unsigned long long)turn * a.nmem);
    int jb;
    const MemberGeom g = geom_of<T>(a, k, jb);
    const int s = turn - late(g);
    const int flags = a.jflags[jb];
    const Band bd = member_band(g, BAND ? a.nbands : 1, b);
    const int os = flags & 1, oe = (flags >> 1) & 1;
    const T *seq = a.series + a.offsets[a.mseries[k]];
    const T *cen = a.centroids + a.coff[jb];
    T *b0 = a.edges + (unsigned long long)k * 2 * a.edge_stride;
    T *b1 = b0 + a.edge_stride;
    const int base = bd.rb - g.r0;  // even: bands keep the step layout
    const int c0 = s * kBlkCols;
    const bool last = s == g.swaths - 1;
    const unsigned long long ks = (unsigned long long)k * a.max_swaths + s;
    BlockJob<T> job;
    job.x = g.flip ? cen : seq;
    job.y = g.flip ? seq : cen;
    job.m = bd.re;
    job.n = g.n;
    job.c0 = c0;
    job.r0 = bd.rb;
    job.edge_in = s ? (((s - 1) & 1) ? b1 : b0) + base : nullptr;
    job.edge_out = last ? nullptr : ((s & 1) ? b1 : b0) + base;
    job.open_end = oe != 0;
    job.free_diag0 = c0 > 0;
    job.corner_init = c0 == 0 ? (g.r0 ? Num<T>::big() : T(0)) : (g.r0 ? T(0) : Num<T>::big());
    job.word_steps = g.steps;
    job.words = reinterpret_cast<unsigned *>(a.words + a.path_off[k] +
                                             (unsigned long long)s * g.steps * 64ull) +
                (size_t)(base / 2) * 32;
    if (BAND) {
      T *row = a.rowbuf + ks * (kBlkCols + 32);
      if (b > 0) {
        // the band below, complete: its last row, and its left edge's value there
        if (feeder && lane == 0)
          wait_word_at_least(a.bdone + ks, (unsigned long long)b, a.err, kWaitLimitNs);
        __syncthreads();
        (void)ld_acquire_gpu(a.bdone + ks);
        job.row_in = row;
        job.corner_init = s ? row[kBlkCols] : Num<T>::big();
      }
      job.top_band = b == bd.count - 1;
      if (b + 1 < bd.count) {
        job.row_out = row;
        job.corner_out = row + kBlkCols;
      }
    }
    T unused = T(0);
    EdgeStat<T> st;
    unsigned long long *words = a.prog + (unsigned long long)k * a.max_swaths;
    BandGate gate;
    gate.g.prog_in = words + (s ? s - 1 : 0);
    gate.g.prog_out = words + s;
    gate.g.err = a.err;
    gate.g.limit_ns = kWaitLimitNs;
    gate.g.avail = 0;
    gate.base = base;
    sweep_block<T, true, BAND, false, false>(job, sm, gate, CkptOut<T>{nullptr, 0, 1}, false, unused,
                                             st);
    if (feeder && lane == 0) {
      T *et = a.emtop + ((unsigned long long)b * layer + ks) * 2;
      et[0] = st.emin;
      et[1] = st.etop;
    }
    if (BAND && b + 1 < bd.count) {
      // the row buffer and corner of every thread, then the band word
      __threadfence();
      __syncthreads();
      if (feeder && lane == 0) st_release_gpu(a.bdone + ks, (unsigned long long)(b + 1));
    }
    if (a.walk_in_sweep) {
      // Member k's last task to finish resolves its shortcut and walks its
      // path (pass 1 of the backtrack) while other blocks sweep: every task
      // makes its moves and edge values visible before it is counted.
      __threadfence();
      __syncthreads();
      if (feeder) {
        unsigned long long n = 0;
        if (lane == 0) n = atomicAdd(a.mdone + k, 1ull) + 1;
        n = __shfl_sync(kFull, n, 0);
        if (n == (unsigned long long)g.swaths * bd.count) {
          __syncwarp();
          (void)ld_acquire_gpu(a.mdone + k);  // every lane: after all the member's tasks
          if (lane == 0) a.shortcut[k] = member_shortcut<T>(a, k, g, flags, kBlkCols);
          __syncwarp();
          walk_member_runs<T>(a, block_map<T>(a, g, k), g, k, os, oe, a.runs + a.runs_off[k]);
        }
      }
    }
    __syncthreads();  // the task word and the rings are free again
  }
}

// Path DTW, a warp per swath (sweep_warp; fills_with_warps): the same pipeline,
// tasks and turns, swaths of 512 columns in double.  Without PIPE (edge columns of
// all members too large) a task is a member, swath after swath, with two edge
// columns per warp.
//
// What bounds it is the issue port, with 12 warps per SM (8 in double): 2000 float
// members of 3000-8000 samples take 12.0 cycles per warp cell and scheduler, fill
// and padding included, against 11.1 in a loop of nothing but path cells (a block
// per swath 15.5).
constexpr int kRoundWarpBlocksF32 = 3, kRoundWarpBlocksF64 = 2;
template <typename T, int R, typename Gate>
__device__ __forceinline__ EdgeStat<T> path_warp_swath(const SwathJob<T> &job, WarpSmem<T> &sm,
                                                       Gate gate) {
  T unused = T(0);
  return sweep_warp<T, R, true, Gate>(job, sm, false, unused, gate);
}
template <typename T, typename Gate>
__device__ __forceinline__ EdgeStat<T> path_warp_any(const SwathJob<T> &job, WarpSmem<T> &sm,
                                                     Gate gate) {
  const int R = warp_regs<T>(job.n - job.c0);
  if (R == kWarpR<T>) return path_warp_swath<T, kWarpR<T>>(job, sm, gate);
  if (sizeof(T) == 4 && R == 16) return path_warp_swath<T, 16>(job, sm, gate);
  return path_warp_swath<T, 8>(job, sm, gate);
}
template <typename T, bool PIPE>
__global__ void
__launch_bounds__(kRoundWarps * 32, sizeof(T) == 4 ? kRoundWarpBlocksF32 : kRoundWarpBlocksF64)
    path_warp_kernel(RoundArgs<T> a) {
  __shared__ WarpSmem<T> s_warp[kRoundWarps];
  WarpSmem<T> &sm = s_warp[threadIdx.x >> 5];
  constexpr int W = 32 * kWarpR<T>;
  const int lane = threadIdx.x & 31;
  const unsigned long long ntasks =
      PIPE ? (unsigned long long)a.nmem * a.max_swaths : (unsigned long long)a.nmem;
  auto member_of = [&](unsigned long long qi) {
    return a.order ? a.order[qi] : a.nmem - 1 - int(qi);
  };
  auto swaths_of = [&](const MemberGeom &g) { return (g.n + W - 1) / W; };
  // the swath of a turn (negative or past the last one: none)
  auto swath_of = [&](const MemberGeom &g, int turn) {
    const int n = swaths_of(g);
    return turn - (n < a.max_swaths ? a.max_swaths - n : 0);
  };
  for (;;) {
    unsigned long long q = 0;
    if (lane == 0) {
      // the next task that exists
      for (;;) {
        q = atomicAdd(a.counter, 1ull);
        if (q >= ntasks) break;
        int jb;
        const MemberGeom g = geom_of<T>(a, member_of(PIPE ? q % a.nmem : q), jb);
        if (!(a.jflags[jb] & 4)) continue;
        if (PIPE && (unsigned)swath_of(g, int(q / a.nmem)) >= (unsigned)swaths_of(g)) continue;
        break;
      }
    }
    q = __shfl_sync(kFull, q, 0);
    if (q >= ntasks) break;
    const int k = member_of(PIPE ? q % a.nmem : q);
    int jb;
    const MemberGeom g = geom_of<T>(a, k, jb);
    const int flags = a.jflags[jb], os = flags & 1, oe = (flags >> 1) & 1;
    const int nsw = swaths_of(g), s0 = PIPE ? swath_of(g, int(q / a.nmem)) : 0;
    const T *seq = a.series + a.offsets[a.mseries[k]];
    const T *cen = a.centroids + a.coff[jb];
    const unsigned long long col =
        PIPE ? (unsigned long long)k
             : (unsigned long long)blockIdx.x * kRoundWarps + (threadIdx.x >> 5);
    T *b0 = a.edges + col * 2 * a.edge_stride;
    T *b1 = b0 + a.edge_stride;
    int shortcut = 0;
    for (int s = s0; s < (PIPE ? s0 + 1 : nsw); ++s) {
      const int c0 = s * W;
      const bool last = s == nsw - 1;
      SwathJob<T> job;
      job.x = g.flip ? cen : seq;
      job.y = g.flip ? seq : cen;
      job.m = g.m;
      job.n = g.n;
      job.c0 = c0;
      job.r0 = g.r0;
      job.edge_in = s ? (((s - 1) & 1) ? b1 : b0) : nullptr;
      job.edge_out = last ? nullptr : ((s & 1) ? b1 : b0);
      job.open_end = oe != 0;
      job.free_diag0 = c0 > 0 && c0 % kRefSwath == 0;
      job.track = oe && !os && !last;
      job.corner_init = c0 == 0 ? (g.r0 ? Num<T>::big() : T(0)) : (g.r0 ? T(0) : Num<T>::big());
      job.words = reinterpret_cast<unsigned *>(a.words + a.path_off[k]) +
                  (size_t)s * g.steps * 64 * WarpMoves<T>::kWords;
      if (PIPE) {
        unsigned long long *words = a.prog + (unsigned long long)k * a.max_swaths;
        PipeGate gate;
        gate.prog_in = words + (s ? s - 1 : 0);
        gate.prog_out = words + s;
        gate.err = a.err;
        gate.limit_ns = kWaitLimitNs;
        gate.avail = 0;
        const EdgeStat<T> st = path_warp_any<T>(job, sm, gate);
        if (lane == 0) {
          T *et = a.emtop + ((unsigned long long)k * a.max_swaths + s) * 2;
          et[0] = st.emin;
          et[1] = st.etop;
        }
      } else {
        const EdgeStat<T> st = path_warp_any<T>(job, sm, SoloGate());
        const int cnext = c0 + W;
        if (job.track && !shortcut && cnext % kRefSwath == 0 && cnext > g.m && st.etop == st.emin)
          shortcut = cnext;
        __syncwarp();  // the next swath reads what this one's lanes stored
      }
    }
    if (!PIPE && lane == 0) a.shortcut[k] = shortcut;
    if (PIPE && a.walk_in_sweep) {
      // as in path_block_kernel: the member's last task to finish walks its path
      __threadfence();
      __syncwarp();
      unsigned long long n = 0;
      if (lane == 0) n = atomicAdd(a.mdone + k, 1ull) + 1;
      n = __shfl_sync(kFull, n, 0);
      if (n == (unsigned long long)nsw) {
        __syncwarp();
        (void)ld_acquire_gpu(a.mdone + k);  // every lane: after all the member's tasks
        if (lane == 0) a.shortcut[k] = member_shortcut<T>(a, k, g, flags, W);
        __syncwarp();
        walk_member_runs<T>(a, warp_map<T>(a, g, k), g, k, os, oe, a.runs + a.runs_off[k]);
      }
    }
    __syncwarp();
  }
}

// The open-end shortcut of the swath pipeline's members (member_shortcut),
// when the row walk does not run inside the path DTW.
template <typename T>
__global__ void shortcut_kernel(RoundArgs<T> a) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= a.nmem) return;
  int jb;
  const MemberGeom g = geom_of<T>(a, k, jb);
  const int flags = a.jflags[jb];
  if (!(flags & 4)) return;
  a.shortcut[k] = member_shortcut<T>(a, k, g, flags, a.one_warp ? warp_cols<T>() : kBlkCols);
}

// Walks member k's path from its end cell toward (0, 0) with one warp and
// calls visit(move, r, c) for every cell; the last call has NIL or
// NIL_OPEN_RIGHT.  Returns false if the walk failed.  Every lane holds the
// moves of one of the 32 rows at and below the current cell in a block of 32
// columns, so the walk advances by shuffles and reloads only when it leaves
// those rows or columns -- about once per 32 steps instead of one dependent
// global load per step.  Every lane keeps the same walk state (visitors store
// from lane 0 only).  Moves are decoded as the reference defines them: the
// open-end shortcut overrides the top row first (with a single-row matrix that
// row is row 0, dtw.hpp:105-108 runs before the row-0 loop), then row 0
// (RIGHT or OPEN_RIGHT, NIL / NIL_OPEN_RIGHT at (0, 0)), then the recorded
// code with RIGHT on the open-end top row meaning OPEN_RIGHT.
template <typename T, typename Map, typename Visit>
__device__ __forceinline__ bool walk_member_path(const RoundArgs<T> &a, const Map &map,
                                                 const MemberGeom &g, int k, int os, int oe,
                                                 Visit &&visit) {
  const int lane = threadIdx.x & 31;
  const int shortcut = a.shortcut[k];
  // A path has at most m + n - 1 cells and never leaves the matrix; the checks
  // only keep a corrupt path buffer from turning into an endless or
  // out-of-bounds walk.
  const long long max_cells = (long long)g.m + g.n - 1;
  long long steps = 0;
  int r = g.m - 1, c = g.n - 1;
  for (;;) {
    const int top = r, cbeg = c & ~31;
    RowMoves mine{0u, 0u};
    if (top - lane >= 1) mine = map.load(map.at(top - lane, cbeg));
    for (;;) {
      const int src = (top - r) & 31;
      const unsigned rd = __shfl_sync(kFull, mine.d, src), ru = __shfl_sync(kFull, mine.u, src);
      int mv;
      if (shortcut && r == g.m - 1 && c >= shortcut) {
        mv = kMoveOpenRight;
      } else if (r == 0) {
        mv = c == 0 ? (os ? kMoveNilOpenRight : kMaxMoveNil) : (os ? kMoveOpenRight : kMoveRight);
      } else {
        const int j = c - cbeg;
        mv = ((rd >> j) & 1u) ? kMoveDiag : ((ru >> j) & 1u) ? kMoveUp : kMoveRight;
        if (mv == kMoveRight && oe && r == g.m - 1) mv = kMoveOpenRight;
      }
      if (mv == kMaxMoveNil || mv == kMoveNilOpenRight) {
        visit(mv, r, c);
        return true;
      }
      if (steps >= max_cells - 1) return false;
      visit(mv, r, c);
      ++steps;
      if (mv == kMoveDiag) {
        --r;
        --c;
      } else if (mv == kMoveUp) {
        --r;
      } else {
        --c;
      }
      if (r < 0 || c < 0) return false;
      if (top - r >= 32 || c < cbeg) break;  // reload the window
    }
  }
}

// The backtrack's ranges alone (no path listing), in two passes.  Pass 1 (one
// warp per member) walks the path a row at a time: in a row the backward walk
// moves left through RIGHT cells until the first cell whose D or U bit is set,
// one count-leading-zeros on the row's bits away, and the walk keeps the row's
// interval of contributing cells' columns for runs[r] ((1, 0) if none).  The
// contributing cells are those of walk_member_path with the backtrack's
// visitor: the top row's OPEN_RIGHT cells (from the open-end shortcut's column
// on, and RIGHT on the open-end top row) contribute nothing, so that row
// contributes only its last cell; row 0 is RIGHT (OPEN_RIGHT with open start)
// down to (0, 0), which contributes unless it is NIL_OPEN_RIGHT.  Pass 2
// (runs_to_ranges_kernel) turns the intervals into per-centroid-index ranges
// in parallel.  Returns false if the walk failed.
//
// The walk is one serial chain per member, so what counts is the latency per
// row: a row takes seven dependent instructions, unrolled eight rows at a time
// without a branch (a walk that has left the window keeps a negative column),
// and everything else -- the rows' bits, the intervals, the exit -- is off the
// chain.  A window is 32 rows (one per lane) by 32 columns; the windows below
// and to the left are loaded with it, and a lane keeps its row's interval in
// registers until the warp stores them together.
//
// The walk starts (or goes on) at st.r, st.c; st.entry is the column it
// entered row st.r at (-1 on the open-end top row, whose interval is its first
// cell alone).  map holds the moves of the columns from cmin (a multiple of the
// swath) on; the walk ends at the start cell (1), when it fails (2: NaN or
// infinite costs can lead it off column 0, in row st.r, whose interval is then
// not stored), or when it leaves cmin to the left (0).
struct RowWalk {
  int r, c, entry;
};
template <typename Map>
__device__ __forceinline__ int walk_runs(const Map &map, const MemberGeom &g, int cmin, RowWalk &st,
                                         int os, int2 *runs) {
  constexpr int G = 8;  // rows per group
  const int lane = threadIdx.x & 31;
  // every window advances the walk by a row or a block of columns: a bound on
  // windows
  const long long max_windows = (long long)g.m + g.n + 64;
  long long windows = 0;
  int r = st.r, c = st.c, entry = st.entry;
  // A window: rows top .. top - 31 of columns cb .. cb + 31; lane l holds row
  // top - l, its moves at `at`.
  int top = -1, cb = 0;
  RowMoves cur{0u, 0u}, down{0u, 0u}, left{0u, 0u};
  typename Map::At at{}, at_left{};
  int2 iv = make_int2(1, 0);
  bool have = false;
  for (;;) {
    const bool below = top >= 0 && r == top - 32;
    if ((below || r == 0 || c < cmin) && have) {
      runs[top - lane] = iv;
      have = false;
    }
    if (c < 0) {  // walked off column 0
      st = RowWalk{r, c, entry};
      return 2;
    }
    if (r == 0) {
      __syncwarp();
      if (lane == 0) runs[0] = os ? make_int2(1, 0) : make_int2(0, c);
      return 1;
    }
    if (c < cmin) {
      st = RowWalk{r, c, entry};
      return 0;
    }
    if (++windows > max_windows) return 2;
    if (below && c >= cb) {
      top -= 32;
      at = Map::below(at);
      cur = down;
    } else if (top >= 0 && !below) {
      cb -= 32;
      at = at_left;
      cur = left;
    } else {
      top = r;
      cb = c & ~31;
      at = map.at(top - lane, cb);
      if (top - lane >= 1) cur = map.load(at);
    }
    if (top - 32 - lane >= 1) down = map.load(Map::below(at));
    if (cb > cmin && top - lane >= 1) {
      at_left = map.left(at, top - lane, cb - 32);
      left = map.load(at_left);
    }
    // Rows that are not the walk's -- row 0 and below, and in the first group
    // those above the walk's row -- get moves that leave the walk where it is.
    const bool row_exists = top - lane >= 1;
    const unsigned dul = row_exists ? cur.d | cur.u : ~0u, dl = row_exists ? cur.d : 0u;
    const int rows = top < 32 ? top : 32;
    int i = top - r, j = c - cb;  // the walk: row top - i, column cb + j
    int i0 = i & ~(G - 1);        // the group: rows top - i0 - q, q < G
    unsigned du[G], d[G];
#pragma unroll
    for (int q = 0; q < G; ++q) {
      du[q] = __shfl_sync(kFull, dul, i0 + q);
      d[q] = __shfl_sync(kFull, dl, i0 + q);
      if (i0 + q < i) {
        du[q] = ~0u;
        d[q] = 0u;
      }
    }
    for (;;) {
      // The chain carries s = 31 - column: 32 or more once the walk has left
      // the window (shifts by more than 31 give 0, and s only grows).
      const int own = lane - i0;
      unsigned s = 31u - unsigned(j), mine = 0u;
#pragma unroll
      for (int q = 0; q < G; ++q) {
        if (own == q) mine = s;
        unsigned x, t;  // the row's moves, and its D bits, from the walk's column on
        asm("shl.b32 %0, %1, %2;" : "=r"(x) : "r"(du[q]), "r"(s));
        const unsigned stop = s + unsigned(__clz(x));
        asm("shl.b32 %0, %1, %2;" : "=r"(t) : "r"(d[q]), "r"(stop));
        s = stop + (t >> 31);
        du[q] = __shfl_sync(kFull, dul, (i0 + G + q) & 31);
        d[q] = __shfl_sync(kFull, dl, (i0 + G + q) & 31);
      }
      // the rows before `end` were entered and left inside the window's
      // columns; where the walk went out in row `end`, that row is complete if
      // it left it by DIAG in the first column, and still the walk's row if
      // its moves are all RIGHT
      const bool out = s >= 32u;
      int end = rows - i0 < G ? rows - i0 : G, after = 31 - int(s);
      unsigned x = 0u;
      if (mine < 32u) x = dul << mine;
      bool whole = false;
      if (out) {
        end = __popc(__ballot_sync(kFull, own >= 1 && own < G && mine < 32u));
        after = 31 - int(__shfl_sync(kFull, mine, i0 + end));
        whole = __any_sync(kFull, own == end && x != 0);
      }
      if (lane >= i && own < end + (whole ? 1 : 0)) {
        const int cp = cb + 31 - int(mine) - __clz(x);
        const int from = lane == i ? entry : cb + 31 - int(mine);
        iv = make_int2(cp, cp > from ? cp : from);
        have = true;
      }
      if (out) {
        if (whole)
          entry = cb - 1;
        else if (i0 + end > i)
          entry = cb + after;
        i = i0 + end + (whole ? 1 : 0);
        j = -1;
        break;
      }
      i = i0 + end;
      i0 = i;
      j = after;
      entry = cb + j;
      if (i >= rows) break;
    }
    r = top - i;
    c = cb + j;
  }
}

template <typename T, typename Map>
__device__ __forceinline__ bool walk_member_runs(const RoundArgs<T> &a, const Map &map,
                                                 const MemberGeom &g, int k, int os, int oe,
                                                 int2 *runs) {
  const int shortcut = a.shortcut[k];
  RowWalk st{g.m - 1, g.n - 1, 0};
  if (shortcut && st.c >= shortcut) st.c = shortcut - 1;  // OPEN_RIGHT from the shortcut's column on
  st.entry = oe ? -1 : st.c;
  return walk_runs(map, g, 0, st, os, runs) == 1;
}

// Pass 2: the contributing columns of row r are the interval runs[r] = [x, y].
// Member on the rows (centroid index t = column): column t's range is [lowest,
// highest] row holding t.  Consecutive rows' intervals share at most one
// column -- row r's first with row r - 1's last (an UP move) and row r's last
// with row r + 1's first -- so row r stores a column's high end unless row
// r + 1 also holds it and its low end unless row r - 1 also holds it; every
// other column of the interval is row r's alone.  Centroid on the rows (t =
// row): the interval is the range.
// lo, t_min: the lowest row walked and the first column taken (a failed walk).
__device__ __forceinline__ void runs_to_ranges(const int2 *runs, int2 *rg, int m, bool flip,
                                               int first, int stride, int lo = 0, int t_min = 0) {
  for (int r = lo + first; r < m; r += stride) {
    const int2 iv = runs[r];
    if (iv.x > iv.y) continue;
    if (flip) {
      rg[r] = iv;
      continue;
    }
    const int2 above = r + 1 < m ? runs[r + 1] : make_int2(1, 0);
    const int2 below = r > lo ? runs[r - 1] : make_int2(1, 0);
    const bool top_shared = above.x <= iv.y && iv.y <= above.y;
    const bool low_shared = below.x <= iv.x && iv.x <= below.y;
    for (int t = iv.x > t_min ? iv.x : t_min; t <= iv.y; ++t) {
      if (!(t == iv.y && top_shared)) rg[t].y = r;
      if (!(t == iv.x && low_shared)) rg[t].x = r;
    }
  }
}
template <typename T>
__global__ void runs_to_ranges_kernel(RoundArgs<T> a) {
  const int k = blockIdx.x;
  int jb;
  const MemberGeom g = geom_of<T>(a, k, jb);
  if (!(a.jflags[jb] & 4)) return;
  runs_to_ranges(a.runs + a.runs_off[k], a.ranges + a.rng_off[k], g.m, g.flip != 0, threadIdx.x,
                 blockDim.x);
}

// The backtrack (updateCentroid's loop, dba.hpp:374-423): per member the
// contiguous range of member samples each centroid index receives, and the
// path listing if asked.  One warp per member; without a listing it runs pass
// 1 of the two-pass ranges (walk_member_runs; launch_backtrack adds pass 2).
template <typename T>
__global__ void __launch_bounds__(kRoundWarps * 32) backtrack_kernel(RoundArgs<T> a) {
  const int lane = threadIdx.x & 31;
  const int k = blockIdx.x * kRoundWarps + (threadIdx.x >> 5);
  if (k >= a.nmem) return;
  int jb;
  const MemberGeom g = geom_of<T>(a, k, jb);
  const int flags = a.jflags[jb];
  if (!(flags & 4)) return;
  const int os = flags & 1, oe = (flags >> 1) & 1;
  int2 *rg = a.ranges + a.rng_off[k];
  if (!a.triples) {
    if (a.one_warp)
      walk_member_runs<T>(a, warp_map<T>(a, g, k), g, k, os, oe, a.runs + a.runs_off[k]);
    else
      walk_member_runs<T>(a, block_map<T>(a, g, k), g, k, os, oe, a.runs + a.runs_off[k]);
    return;
  }
  int32_t *tri = a.triples + 3ull * a.trip_off[k];
  const bool lead = lane == 0;
  long long nt = 0;
  int cur_t = -1, lo = 1, hi = 0;
  auto contribute = [&](int rr, int cc) {
    const int ti = g.flip ? rr : cc;  // centroid index
    const int mi = g.flip ? cc : rr;  // member sample index
    if (ti != cur_t) {
      if (lead && cur_t >= 0 && hi >= lo) rg[cur_t] = make_int2(lo, hi);
      cur_t = ti;
      lo = mi;
      hi = mi;
    } else {
      lo = mi;  // the walk only moves toward smaller indices
    }
  };
  auto visit = [&](int mv, int r, int c) {
    if (mv == kMaxMoveNil || mv == kMoveNilOpenRight) {
      // the start cell (dba.hpp:412-415)
      if (mv != kMoveNilOpenRight) contribute(0, 0);
      if (lead && cur_t >= 0 && hi >= lo) rg[cur_t] = make_int2(lo, hi);
    } else if (mv != kMoveOpenRight) {
      contribute(r, c);
    }
    if (lead && tri) {
      tri[3 * nt] = r;
      tri[3 * nt + 1] = c;
      tri[3 * nt + 2] = mv;
    }
    ++nt;
  };
  const bool ok = a.one_warp ? walk_member_path<T>(a, warp_map<T>(a, g, k), g, k, os, oe, visit)
                             : walk_member_path<T>(a, block_map<T>(a, g, k), g, k, os, oe, visit);
  if (lead && a.triple_counts) a.triple_counts[k] = ok ? nt : -1;
}

// Prefix chop (chopPrefixFromSequences' host walk, dba.hpp:1313-1336), on
// each series' open-end path against the leader (leader on the rows): skip
// the OPEN_RIGHT run along the top row from the end cell; the column reached
// is the chop position; then count, per leader row, the path cells from there
// to (0, 0) (the cell reached counts 1 on the top row).  One warp per series;
// rows are visited in one run each, so each count is stored once.
template <typename T>
__global__ void __launch_bounds__(kRoundWarps * 32) chop_walk_kernel(RoundArgs<T> a, long long *chop,
                                                                    int *hist, int P) {
  const int lane = threadIdx.x & 31;
  const int k = blockIdx.x * kRoundWarps + (threadIdx.x >> 5);
  if (k >= a.nmem) return;
  int jb;
  const MemberGeom g = geom_of<T>(a, k, jb);
  const int flags = a.jflags[jb];
  if (!(flags & 4)) return;
  const bool lead = lane == 0;
  int *h = hist + (unsigned long long)k * P;
  bool skipping = true;
  long long pos = -1;
  int row = -1, count = 0;
  auto visit = [&](int mv, int r, int c) {
    if (skipping) {
      if (mv == kMoveOpenRight) return;
      skipping = false;
      pos = c;
      row = r;
      count = 1;
      return;
    }
    if (r == row) {
      ++count;
    } else {
      if (lead) h[row] = count;
      row = r;
      count = 1;
    }
  };
  const int os = flags & 1, oe = (flags >> 1) & 1;
  const bool ok = a.one_warp ? walk_member_path<T>(a, warp_map<T>(a, g, k), g, k, os, oe, visit)
                             : walk_member_path<T>(a, block_map<T>(a, g, k), g, k, os, oe, visit);
  if (lead) {
    if (ok && row >= 0) h[row] = count;
    chop[k] = ok ? pos : -1;
  }
}

// The reference divides on the host (dba.hpp:820-822); a centroid index that
// received no sample gives 0/0, which x86 answers with its default NaN (sign
// bit set, printed "-nan").  The device's 0/0 NaN differs, so it is replaced.
template <typename T>
__device__ __forceinline__ T host_default_nan();
template <>
__device__ __forceinline__ float host_default_nan<float>() { return __int_as_float(0xffc00000); }
template <>
__device__ __forceinline__ double host_default_nan<double>() {
  return __longlong_as_double((long long)0xfff8000000000000ull);
}

template <typename T>
__device__ __forceinline__ T div_rn(T a, T b);
template <>
__device__ __forceinline__ float div_rn<float>(float a, float b) { return __fdiv_rn(a, b); }
template <>
__device__ __forceinline__ double div_rn<double>(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

// grid: (ceil(max centroid length / 256), jobs)
template <typename T>
__global__ void
__launch_bounds__(kReduceThreads, sizeof(T) == 4 ? kReduceBlocksF32 : kReduceBlocksF64)
    reduce_kernel(RoundArgs<T> a) {
  // One warp per centroid index: the index's sum is a chain of additions in
  // the reference's order (members in order, each member's samples from the
  // highest down, the stripe-mode extra sample last), so the warp's lanes
  // load the samples of consecutive members at once (lane l the l-th group
  // of mpl <= kMpl members of a chunk) and lay them out in that order in the
  // warp's shared-memory buffer; lane 0 then adds the buffer.  Many warps per
  // SM keep the loads and the chains of different indices in flight together.
  //
  // What bounds it is the chain of four dependent loads per member (offset,
  // range, series, sample).  The members of a chunk spread evenly over the
  // lanes, and each lane has its members' first samples in flight together.
  // 8 members per lane always, one load after the other, against this: 64
  // members of 512-1024 samples 33 -> 13 us, 690 in 24 jobs 79 -> 28, 400 of
  // 3000-8000 203 -> 112 (184 with kMpl = 8, four blocks per SM), 100 double of
  // 1000-4000 67 -> 57.
  constexpr int kCap = 8192 / int(sizeof(T));  // samples per warp's buffer
  constexpr int kMpl = 4;                      // members per lane per chunk
  __shared__ T s_buf[kReduceWarps][kCap];
  __shared__ double s_max[kReduceWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int jb = blockIdx.y;
  const int t = blockIdx.x * kReduceWarps + wid;
  const int Lc = a.clen[jb];
  const bool live = (a.jflags[jb] & 4) != 0;
  double dl = 0.0;
  if (live && t < Lc) {
    T sum = T(0);
    uint32_t cnt = 0;
    T *buf = s_buf[wid];
    const int kb = a.mbeg[jb], ke = a.mend[jb];
    for (int k0 = kb; k0 < ke; k0 += 32 * kMpl) {
      const int mpl = ke - k0 >= 32 * kMpl ? kMpl : (ke - k0 + 31) / 32;
      int2 r[kMpl];
      int e[kMpl];
      const T *sq[kMpl];
      T first[kMpl];
      int n_l = 0;
#pragma unroll
      for (int u = 0; u < kMpl; ++u) {
        const int m = k0 + lane * mpl + u;
        r[u] = make_int2(1, 0);
        e[u] = -1;
        sq[u] = a.series;
        if (u < mpl && m < ke) {
          const unsigned long long ro = a.rng_off[m];
          r[u] = a.ranges[ro + t];
          sq[u] = a.series + a.offsets[a.mseries[m]];
          if (a.extra) e[u] = a.extra[ro + t];
        }
      }
#pragma unroll
      for (int u = 0; u < kMpl; ++u) {
        first[u] = T(0);
        if (r[u].y < r[u].x) continue;
        n_l += r[u].y - r[u].x + 1 + (e[u] >= 0 ? 1 : 0);
        first[u] = __ldg(sq[u] + r[u].y);
      }
      int incl = n_l;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, off);
        if (lane >= off) incl += y;
      }
      const int total = __shfl_sync(kFull, incl, 31);
      cnt += uint32_t(total);
      if (total <= kCap) {
        int p = incl - n_l;
#pragma unroll
        for (int u = 0; u < kMpl; ++u) {
          if (r[u].y < r[u].x) continue;
          buf[p++] = first[u];
          for (int i = r[u].y - 1; i >= r[u].x; --i) buf[p++] = __ldg(sq[u] + i);
          if (e[u] >= 0) buf[p++] = __ldg(sq[u] + e[u]);
        }
        __syncwarp();
        if (lane == 0)
          for (int q = 0; q < total; ++q) sum = add_rn(sum, buf[q]);
        __syncwarp();
      } else {
        // more samples than the buffer holds: the lanes add theirs in turn,
        // each starting from the previous lane's sum
        for (int L = 0; L < 32; ++L) {
          if (lane == L) {
#pragma unroll
            for (int u = 0; u < kMpl; ++u) {
              if (r[u].y < r[u].x) continue;
              for (int i = r[u].y; i >= r[u].x; --i) sum = add_rn(sum, sq[u][i]);
              if (e[u] >= 0) sum = add_rn(sum, sq[u][e[u]]);
            }
          }
          sum = __shfl_sync(kFull, sum, L);
        }
      }
    }
    if (lane == 0) {
      const T mean = cnt ? div_rn<T>(sum, T(cnt)) : host_default_nan<T>();
      a.means[a.coff[jb] + t] = mean;
      a.counts[a.coff[jb] + t] = cnt;
      const double d = fabs(double(a.centroids[a.coff[jb] + t] - mean));
      dl = d > 0.0 ? d : 0.0;  // NaN never raises the maximum (dba.hpp:833)
    }
  }
  if (lane == 0) s_max[wid] = dl;
  __syncthreads();
  if (threadIdx.x == 0 && live) {
    double m = s_max[0];
    for (int q = 1; q < kReduceWarps; ++q) m = s_max[q] > m ? s_max[q] : m;
    // non-negative doubles order like their bit patterns
    atomicMax(reinterpret_cast<unsigned long long *>(a.deltas + jb), (unsigned long long)__double_as_longlong(m));
  }
}

// One job, members 0..n-1 in order (the single-cluster DBAUpdate call).
__global__ void single_job_kernel(int *mseries, int *mjob, int n, int *clen, int Lc, int *jflags,
                                  int flags, int *mbeg, int *mend, unsigned long long *coff) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    mseries[k] = k;
    mjob[k] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    clen[0] = Lc;
    jflags[0] = flags;
    mbeg[0] = 0;
    mend[0] = n;
    coff[0] = 0;
  }
}

// Resident blocks of the path kernel on the current device, cached per device
// index (host threads may race; both compute the same value).
template <typename T>
int round_grid() {
  static std::atomic<int> cached[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    const int c = cached[dev].load(std::memory_order_relaxed);
    if (c) return c;
  }
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, path_block_kernel<T, false>, kBlkThreads, 0);
  constexpr int want = sizeof(T) == 4 ? kRoundBlocksF32 : kRoundBlocksF64;
  if (per_sm > want) per_sm = want;
  if (per_sm < 1) per_sm = 1;
  const int g = sms * per_sm;
  if (dev >= 0 && dev < 64) cached[dev].store(g, std::memory_order_relaxed);
  return g;
}

// Resident blocks of the one-warp path kernel (cached like round_grid).
template <typename T>
int round_warp_grid() {
  static std::atomic<int> cached[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    const int c = cached[dev].load(std::memory_order_relaxed);
    if (c) return c;
  }
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, path_warp_kernel<T, true>, kRoundWarps * 32, 0);
  constexpr int want = sizeof(T) == 4 ? kRoundWarpBlocksF32 : kRoundWarpBlocksF64;
  if (per_sm > want) per_sm = want;
  if (per_sm < 1) per_sm = 1;
  const int g = sms * per_sm;
  if (dev >= 0 && dev < 64) cached[dev].store(g, std::memory_order_relaxed);
  return g;
}

struct RoundLayout {
  size_t off_counter, off_path, off_trip, off_rng, off_runoff, off_short, off_single, off_ranges,
      off_runs, off_edges, off_words, off_prog, off_bdone, off_mdone, off_order, off_emtop,
      off_rowbuf, total;
  unsigned long long edge_stride;
  int max_swaths;
  int nbands;  // row bands of the swath pipeline
  bool pipe;   // path DTW as the swath pipeline (two edge columns per member)
  bool one_warp;  // a warp per swath, not a block
};

constexpr size_t kPipeEdgeBytes = size_t(8) << 30;  // per-member edge columns up to 8 GB
constexpr int kMaxBands = 8;
constexpr size_t kMaxRowBufBytes = size_t(256) << 20;
std::atomic<int> g_round_bands{0};  // odba_round_set_bands (0: chosen per launch)

// Row bands of the swath pipeline: those pinned, else none.
int pipe_bands() {
  const int forced = g_round_bands.load(std::memory_order_relaxed);
  return forced > 0 ? (forced < kMaxBands ? forced : kMaxBands) : 1;
}

// Whether a round fills the GPU with one warp per swath.  units: its work, the
// rows of all (member, 1024-column swath) pairs over the most rows of a member;
// max_swaths: the most swaths of a member.  At full load the one-warp sweep
// takes three quarters of the block sweep's issue slots per cell; the block sweep
// ends a chain of swaths in a quarter of the steps, and the longer the chains the
// more of them it takes to hide their ends.  One B200, block time / one-warp time
// of a round (lengths even over the range, centroid of a middling member):
//   float, 1 swath   100-400 samples    630 / 940 / 1250 / 1560 units    0.99 / 1.03 / 1.10 / 1.10
//                    400-800            750 / 1500 / 1880                0.93 / 0.94 / 1.07
//          2         1000-2000          900 / 1200 / 1500 / 1800         0.97 / 1.01 / 1.11 / 1.28
//          3         2000-4000          900 / 1350 / 1580 / 2030         0.81 / 0.99 / 1.03 / 1.04
//          5-6       3000-8000          1240 / 1860 / 2060 / 2480        0.92 / 1.02 / 0.98 / 1.07
//          12-13     8000-16000         1800 / 2250 / 2930               0.92 / 0.96 / 1.04
//   double, 1        100-400            310 / 440 / 560                  0.99 / 1.11 / 1.24
//                    400-800            230 / 380 / 530                  0.79 / 1.01 / 1.23
//          2         1000-2000          300 / 450 / 600                  0.82 / 1.03 / 1.15
//          3-4       2000-4000          450 / 900                        0.86 / 1.13
//          5-6       3000-8000          830 / 1040 / 1240                0.96 / 1.02 / 1.03
//          11-12     8000-16000         900 / 1240                       0.96 / 0.99
// Few long members among short ones leave the long chains alone at the end (float,
// 300 members of 200-20000, log-even, 3600 pairs in 611 units: 7.6 ms by blocks,
// 11.0 by warps), so the rule counts work, not pairs.  Larger rounds: 2000 float
// members of 3000-8000 25.2 ms (block) and 20.0, 1000 double ones 28.2 and 21.7.
template <typename T>
bool fills_with_warps(unsigned long long units, int max_swaths) {
  const unsigned long long slots = (unsigned long long)round_warp_grid<T>() * kRoundWarps;
  // percent of the resident warps
  const unsigned pc = sizeof(T) == 4 ? (max_swaths <= 4 ? 85 : max_swaths <= 8 ? 150 : 160)
                                     : (max_swaths <= 2   ? 38
                                        : max_swaths <= 4 ? 63
                                        : max_swaths <= 8 ? 90
                                                          : 110);
  return units * 100 >= slots * pc;
}

// Workspace layout for nmem members / njobs jobs with the given totals; units:
// the active members' work (fills_with_warps).
template <typename T>
RoundLayout round_layout(int nmem, int njobs, unsigned long long words,
                         unsigned long long ranges, unsigned long long maxm, int max_swaths = 0,
                         unsigned long long rows = 0, unsigned long long units = 0) {
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  RoundLayout L;
  L.edge_stride = (maxm + 32 + 31) / 32 * 32;
  L.pipe = max_swaths > 0 && size_t(nmem) * 2 * L.edge_stride * sizeof(T) <= kPipeEdgeBytes;
  L.nbands = L.pipe ? pipe_bands() : 1;
  L.one_warp = max_swaths > 0 && (!L.pipe || (L.nbands == 1 && fills_with_warps<T>(units, max_swaths)));
  L.max_swaths = L.one_warp ? max_swaths * (kBlkCols / warp_cols<T>()) : max_swaths;
  const size_t edge_cols = L.pipe ? size_t(nmem)
                           : L.one_warp ? size_t(round_warp_grid<T>()) * kRoundWarps : 0;
  size_t o = 0;
  L.off_counter = o; o += 256;
  L.off_path = o; o += up(size_t(nmem) * 8);
  L.off_trip = o; o += up(size_t(nmem) * 8);
  L.off_rng = o; o += up(size_t(nmem) * 8);
  L.off_runoff = o; o += up(size_t(nmem) * 8);
  L.off_short = o; o += up(size_t(nmem) * 4);
  // single-job descriptors: mseries, mjob (nmem ints each), clen, jflags, mbeg, mend, coff
  L.off_single = o; o += up(size_t(nmem) * 8 + 64);
  L.off_ranges = o; o += up(size_t(ranges) * sizeof(int2));
  L.off_runs = o; o += up(size_t(rows) * sizeof(int2));  // cleared with the ranges
  L.off_edges = o; o += up(edge_cols * 2 * L.edge_stride * sizeof(T));
  L.off_words = o; o += up(words * 8);
  const size_t ps = L.pipe ? size_t(nmem) * size_t(L.max_swaths) : 0;
  // row buffers for at most kMaxRowBufBytes (many inactive members: no bands)
  if (L.nbands > 1 && ps * (kBlkCols + 32) * sizeof(T) > kMaxRowBufBytes) L.nbands = 1;
  L.off_prog = o; o += up(ps * 8);
  L.off_bdone = o; o += up(ps * 8);  // cleared with the progress words
  L.off_mdone = o; o += L.pipe ? up(size_t(nmem) * 8) : 0;  // likewise
  L.off_order = o; o += L.pipe ? up(size_t(nmem) * 4) : 0;
  L.off_emtop = o; o += up(ps * L.nbands * 2 * sizeof(T));
  L.off_rowbuf = o; o += L.nbands > 1 ? up(ps * (kBlkCols + 32) * sizeof(T)) : 0;
  L.total = o;
  (void)njobs;
  return L;
}

template <typename T>
void host_totals(const uint64_t *h_lens, const int *h_mjob, int nmem, const uint64_t *h_clen,
                 const int *h_flags, unsigned long long &words, unsigned long long &ranges,
                 unsigned long long &maxm, int *max_swaths = nullptr,
                 unsigned long long *rows = nullptr, unsigned long long *units = nullptr) {
  words = ranges = 0;
  maxm = 1;
  if (max_swaths) *max_swaths = 1;
  if (rows) *rows = 0;
  unsigned long long work = 0;
  for (int k = 0; k < nmem; ++k) {
    const int j = h_mjob ? h_mjob[k] : 0;
    const int f = h_flags[j];
    if (!(f & 4)) continue;
    const MemberGeom g = member_geom<T>(h_lens[k], h_clen[j], f & 1, (f >> 1) & 1, (f >> 3) & 1);
    words += g.words;
    ranges += h_clen[j];
    if ((unsigned long long)g.m > maxm) maxm = g.m;
    if (max_swaths && g.swaths > *max_swaths) *max_swaths = g.swaths;
    if (rows) *rows += (unsigned long long)g.m;
    work += (unsigned long long)g.m * g.swaths;
  }
  if (units) *units = work / maxm;
}

// Planning, range clearing and the path DTW of a round (everything before
// the backtrack).
template <typename T>
void launch_paths(RoundArgs<T> &a, const RoundLayout &L, char *base, cudaStream_t stream,
                  bool walk_runs = false) {
  a.counter = reinterpret_cast<unsigned long long *>(base + L.off_counter);
  a.path_off = reinterpret_cast<unsigned long long *>(base + L.off_path);
  a.trip_off = reinterpret_cast<unsigned long long *>(base + L.off_trip);
  a.rng_off = reinterpret_cast<unsigned long long *>(base + L.off_rng);
  a.runs_off = reinterpret_cast<unsigned long long *>(base + L.off_runoff);
  a.shortcut = reinterpret_cast<int *>(base + L.off_short);
  a.ranges = reinterpret_cast<int2 *>(base + L.off_ranges);
  a.runs = reinterpret_cast<int2 *>(base + L.off_runs);
  a.edges = reinterpret_cast<T *>(base + L.off_edges);
  a.edge_stride = L.edge_stride;
  a.words = reinterpret_cast<unsigned long long *>(base + L.off_words);
  a.prog = reinterpret_cast<unsigned long long *>(base + L.off_prog);
  a.emtop = reinterpret_cast<T *>(base + L.off_emtop);
  a.bdone = reinterpret_cast<unsigned long long *>(base + L.off_bdone);
  a.rowbuf = L.nbands > 1 ? reinterpret_cast<T *>(base + L.off_rowbuf) : nullptr;
  a.nbands = L.nbands;
  a.mdone = reinterpret_cast<unsigned long long *>(base + L.off_mdone);
  a.walk_in_sweep = (L.pipe && walk_runs) ? 1 : 0;
  a.err = reinterpret_cast<unsigned *>(base + L.off_counter + 8);
  a.max_swaths = L.max_swaths;
  const unsigned long long nr = (L.off_edges - L.off_ranges) / sizeof(int2);
  cudaMemsetAsync(a.counter, 0, 16, stream);  // work counter and error word
  plan_kernel<T><<<1, kPlanThreads, 0, stream>>>(a);
  fill_ranges_kernel<<<int(nr / 256 + 1 < 4096 ? nr / 256 + 1 : 4096), 256, 0, stream>>>(a.ranges, nr);
  a.one_warp = L.one_warp ? 1 : 0;
  const unsigned long long tasks =
      L.pipe ? (unsigned long long)a.nmem * L.max_swaths * L.nbands : (unsigned long long)a.nmem;
  const unsigned long long wgrid = L.one_warp ? round_warp_grid<T>() : round_grid<T>(),
                           wblocks = L.one_warp ? (tasks + kRoundWarps - 1) / kRoundWarps : tasks;
  const int grid = int(wblocks < wgrid ? wblocks : wgrid);
  if (!L.pipe) {
    path_warp_kernel<T, false><<<grid, kRoundWarps * 32, 0, stream>>>(a);
    return;
  }
  cudaMemsetAsync(a.prog, 0, L.off_order - L.off_prog, stream);  // progress, band, member words
  if (!a.order && a.nmem <= kRankMembers) {
    int *ord = reinterpret_cast<int *>(base + L.off_order);
    rank_members_kernel<T><<<(a.nmem + 255) / 256, 256, 0, stream>>>(a, ord);
    a.order = ord;
  }
  if (L.one_warp)
    path_warp_kernel<T, true><<<grid, kRoundWarps * 32, 0, stream>>>(a);
  else if (L.nbands > 1)
    path_block_kernel<T, true><<<grid, kBlkThreads, 0, stream>>>(a);
  else
    path_block_kernel<T, false><<<grid, kBlkThreads, 0, stream>>>(a);
  if (!a.walk_in_sweep) shortcut_kernel<T><<<(a.nmem + 127) / 128, 128, 0, stream>>>(a);
}

// The backtrack: with a path listing one kernel walking cell by cell; without,
// the row walk (pass 1, inside the swath pipeline's path DTW when it ran
// there) and the parallel conversion of its row intervals into ranges
// (pass 2).
template <typename T>
void launch_backtrack(const RoundArgs<T> &a, cudaStream_t stream) {
  if (!a.walk_in_sweep)
    backtrack_kernel<T><<<(a.nmem + kRoundWarps - 1) / kRoundWarps, kRoundWarps * 32, 0, stream>>>(a);
  if (!a.triples) runs_to_ranges_kernel<T><<<a.nmem, 256, 0, stream>>>(a);
}

template <typename T>
int launch_round(RoundArgs<T> &a, const RoundLayout &L, char *base, int max_clen,
                 cudaStream_t stream) {
  launch_paths<T>(a, L, base, stream, !a.triples);
  launch_backtrack<T>(a, stream);
  dim3 rg((max_clen + kReduceWarps - 1) / kReduceWarps, a.njobs);
  reduce_kernel<T><<<rg, kReduceThreads, 0, stream>>>(a);
  return check_launch("DBA round kernels");
}

}  // namespace

int dba_round_bands(int n) { return g_round_bands.exchange(n); }

template <typename T>
size_t dba_round_workspace_bytes(const uint64_t *h_lens, int n, uint64_t Lc, int os, int oe) {
  unsigned long long words, ranges, maxm;
  const uint64_t clen = Lc;
  const int flags = (os ? 1 : 0) | (oe ? 2 : 0) | 4;
  int ms = 1;
  unsigned long long rows = 0, units = 0;
  host_totals<T>(h_lens, nullptr, n, &clen, &flags, words, ranges, maxm, &ms, &rows, &units);
  if (Lc > maxm) maxm = Lc;
  return round_layout<T>(n, 1, words, ranges, maxm, ms, rows, units).total;
}

namespace {

// The descriptors of a one-job round (members 0..n-1 in order, all active)
// in the workspace, and round arguments pointing at them; outputs unset.
template <typename T>
RoundArgs<T> single_job_round(const T *centroid, uint64_t Lc, const T *series,
                              const uint64_t *offsets, const uint64_t *lens, int n, int flags,
                              const RoundLayout &L, char *base, cudaStream_t stream) {
  int *single = reinterpret_cast<int *>(base + L.off_single);
  int *mseries = single, *mjob = single + n, *d_clen = single + 2 * n, *d_flags = single + 2 * n + 1,
      *d_mbeg = single + 2 * n + 2, *d_mend = single + 2 * n + 3;
  unsigned long long *d_coff =
      reinterpret_cast<unsigned long long *>(base + L.off_single + ((size_t(2 * n + 4) * 4 + 7) / 8) * 8);
  single_job_kernel<<<(n + 255) / 256, 256, 0, stream>>>(mseries, mjob, n, d_clen, int(Lc), d_flags,
                                                        flags, d_mbeg, d_mend, d_coff);
  RoundArgs<T> a;
  a.centroids = centroid;
  a.coff = d_coff;
  a.clen = d_clen;
  a.jflags = d_flags;
  a.mbeg = d_mbeg;
  a.mend = d_mend;
  a.njobs = 1;
  a.series = series;
  a.offsets = offsets;
  a.lens = lens;
  a.mseries = mseries;
  a.mjob = mjob;
  a.order = nullptr;
  a.nmem = n;
  a.means = nullptr;
  a.counts = nullptr;
  a.deltas = nullptr;
  a.triples = nullptr;
  a.triple_counts = nullptr;
  return a;
}

template <typename T>
RoundLayout single_job_layout(const uint64_t *h_lens, int n, uint64_t Lc, int flags) {
  unsigned long long words, ranges, maxm;
  const uint64_t clen = Lc;
  int ms = 1;
  unsigned long long rows = 0, units = 0;
  host_totals<T>(h_lens, nullptr, n, &clen, &flags, words, ranges, maxm, &ms, &rows, &units);
  if (Lc > maxm) maxm = Lc;
  return round_layout<T>(n, 1, words, ranges, maxm, ms, rows, units);
}

}  // namespace

template <typename T>
int dba_round_launch(const T *centroid, uint64_t Lc, const T *series, const uint64_t *offsets,
                     const uint64_t *lens, const uint64_t *h_lens, int n, int os, int oe, T *mean,
                     uint32_t *counts, double *delta, int32_t *triples, int64_t *triple_counts,
                     void *ws, size_t ws_bytes, cudaStream_t stream) {
  const int flags = (os ? 1 : 0) | (oe ? 2 : 0) | 4;
  const RoundLayout L = single_job_layout<T>(h_lens, n, Lc, flags);
  if (ws_bytes < L.total) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "DBA round workspace too small");
  char *base = static_cast<char *>(ws);
  RoundArgs<T> a = single_job_round<T>(centroid, Lc, series, offsets, lens, n, flags, L, base, stream);
  a.means = mean;
  a.counts = counts;
  a.deltas = delta;
  a.triples = triples;
  a.triple_counts = triple_counts;
  return launch_round<T>(a, L, base, int(Lc), stream);
}

// The first half of a round for a share of the members (a multi-GPU round
// deals members to ranks): path DTW and backtrack, then every member's
// per-centroid-index sample ranges copied to ranges_out (member k's at
// k * Lc; (1, 0) where a centroid index receives nothing).  Same workspace as
// dba_round_launch.
template <typename T>
int dba_round_ranges_launch(const T *centroid, uint64_t Lc, const T *series,
                            const uint64_t *offsets, const uint64_t *lens, const uint64_t *h_lens,
                            int n, int os, int oe, int2 *ranges_out, void *ws, size_t ws_bytes,
                            cudaStream_t stream) {
  const int flags = (os ? 1 : 0) | (oe ? 2 : 0) | 4;
  const RoundLayout L = single_job_layout<T>(h_lens, n, Lc, flags);
  if (ws_bytes < L.total) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "DBA round workspace too small");
  char *base = static_cast<char *>(ws);
  RoundArgs<T> a = single_job_round<T>(centroid, Lc, series, offsets, lens, n, flags, L, base, stream);
  // the plan clears the job's delta: point it at a spare word of the header
  a.deltas = reinterpret_cast<double *>(base + L.off_counter + 16);
  launch_paths<T>(a, L, base, stream, true);
  launch_backtrack<T>(a, stream);
  cudaMemcpyAsync(ranges_out, a.ranges, size_t(n) * Lc * sizeof(int2), cudaMemcpyDeviceToDevice, stream);
  return check_launch("DBA round path and backtrack kernels");
}

template <typename T>
size_t dba_reduce_workspace_bytes(int n) {
  return round_layout<T>(n, 1, 0, 0, 1, 0).total;
}

// The second half: the ordered reducer over all n members' sample ranges
// (from dba_round_ranges_launch, members in the round's order), giving the
// new centroid, the pile-up counts and the delta exactly as the whole round
// does.
template <typename T>
int dba_reduce_ranges_launch(const T *centroid, uint64_t Lc, const T *series,
                             const uint64_t *offsets, const uint64_t *lens, int n, int os, int oe,
                             const int2 *ranges, T *mean, uint32_t *counts, double *delta, void *ws,
                             size_t ws_bytes, cudaStream_t stream) {
  const int flags = (os ? 1 : 0) | (oe ? 2 : 0) | 4;
  const RoundLayout L = round_layout<T>(n, 1, 0, 0, 1, 0);
  if (ws_bytes < L.total) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "reducer workspace too small");
  char *base = static_cast<char *>(ws);
  RoundArgs<T> a = single_job_round<T>(centroid, Lc, series, offsets, lens, n, flags, L, base, stream);
  a.path_off = reinterpret_cast<unsigned long long *>(base + L.off_path);
  a.trip_off = reinterpret_cast<unsigned long long *>(base + L.off_trip);
  a.rng_off = reinterpret_cast<unsigned long long *>(base + L.off_rng);
  a.ranges = const_cast<int2 *>(ranges);
  a.means = mean;
  a.counts = counts;
  a.deltas = delta;
  plan_kernel<T><<<1, kPlanThreads, 0, stream>>>(a);
  reduce_kernel<T><<<dim3(unsigned((Lc + kReduceWarps - 1) / kReduceWarps), 1), kReduceThreads, 0, stream>>>(a);
  return check_launch("DBA reducer kernels");
}

template <typename T>
size_t dba_batch_workspace_bytes(const uint64_t *h_mlens, const int *h_mjob, int nmem,
                                 const uint64_t *h_clen, const int *h_flags, int njobs) {
  unsigned long long words, ranges, maxm;
  int ms = 1;
  unsigned long long rows = 0, units = 0;
  host_totals<T>(h_mlens, h_mjob, nmem, h_clen, h_flags, words, ranges, maxm, &ms, &rows, &units);
  for (int j = 0; j < njobs; ++j)
    if (h_clen[j] > maxm) maxm = h_clen[j];
  return round_layout<T>(nmem, njobs, words, ranges, maxm, ms, rows, units).total;
}

template <typename T>
bool dba_batch_by_warp(const uint64_t *h_mlens, const int *h_mjob, int nmem, const uint64_t *h_clen,
                       const int *h_flags, int njobs) {
  unsigned long long words, ranges, maxm;
  int ms = 1;
  unsigned long long rows = 0, units = 0;
  host_totals<T>(h_mlens, h_mjob, nmem, h_clen, h_flags, words, ranges, maxm, &ms, &rows, &units);
  for (int j = 0; j < njobs; ++j)
    if (h_clen[j] > maxm) maxm = h_clen[j];
  return round_layout<T>(nmem, njobs, words, ranges, maxm, ms, rows, units).one_warp;
}
template bool dba_batch_by_warp<float>(const uint64_t *, const int *, int, const uint64_t *,
                                       const int *, int);
template bool dba_batch_by_warp<double>(const uint64_t *, const int *, int, const uint64_t *,
                                        const int *, int);

template <typename T>
int dba_batch_launch(const T *centroids, const unsigned long long *coff, const int *clen,
                     const int *jflags, const int *mbeg, const int *mend, int njobs, int max_clen,
                     const T *series, const uint64_t *offsets, const uint64_t *lens,
                     const int *mseries, const int *mjob, const int *order, int nmem,
                     const uint64_t *h_mlens, const int *h_mjob, const uint64_t *h_clen,
                     const int *h_flags, T *means, uint32_t *counts, double *deltas,
                     int32_t *triples, int64_t *triple_counts, void *ws, size_t ws_bytes,
                     cudaStream_t stream) {
  unsigned long long words, ranges, maxm;
  int ms = 1;
  unsigned long long rows = 0, units = 0;
  host_totals<T>(h_mlens, h_mjob, nmem, h_clen, h_flags, words, ranges, maxm, &ms, &rows, &units);
  for (int j = 0; j < njobs; ++j)
    if (h_clen[j] > maxm) maxm = h_clen[j];
  const RoundLayout L = round_layout<T>(nmem, njobs, words, ranges, maxm, ms, rows, units);
  if (ws_bytes < L.total) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "DBA batch workspace too small");
  RoundArgs<T> a;
  a.centroids = centroids;
  a.coff = coff;
  a.clen = clen;
  a.jflags = jflags;
  a.mbeg = mbeg;
  a.mend = mend;
  a.njobs = njobs;
  a.series = series;
  a.offsets = offsets;
  a.lens = lens;
  a.mseries = mseries;
  a.mjob = mjob;
  a.order = order;
  a.nmem = nmem;
  a.means = means;
  a.counts = counts;
  a.deltas = deltas;
  a.triples = triples;
  a.triple_counts = triple_counts;
  return launch_round<T>(a, L, static_cast<char *>(ws), max_clen, stream);
}

// ---------------------------------------------------------------------------
// Stripe mode: one DBA round for members whose 2-bit path does not fit in
// memory (the reference's stripe mode, dba.hpp:515-763).  Per member, in the
// orientation of the full-path round (centroid on the rows when an open end
// flips the member, dba.hpp:497-501):
//   1. forward: the swath pipeline (a block per 1024-column swath, bounded
//      hand-off waits); every swath's right edge is kept (E, one column of
//      rows per swath) and every K-th cost row is kept across all columns (Q);
//   2. backtrack, from the right: the K-row tiles of a group of reference
//      stripes (1024 columns each) below the current backtrack height H are
//      recomputed with their moves in parallel (one block per tile: its row
//      below comes from Q, its left edge from E), then one warp continues the
//      walk through the group;
//   3. the ordered reducer of the full-path round.
// The reference re-runs each stripe with the first sequence's length set to H
// (dba.hpp:700-721), so with an open end its top-row rule acts on row H-1 and
// its shortcut (dtw.hpp:74-129, open end only) is checked on the stored left
// edge's rows below H whenever the stripe starts past column H: if it fires,
// the stripe's row H-1 is all OPEN_RIGHT.  Stripes from the first one whose
// shortcut fired in the forward pass on take that branch too (the reference's
// forward pass stopped there and left those edges unwritten).  The recompute
// here does the same: rows below H-1 are the forward pass's, row H-1 follows
// the open-end rules.  A group is then one stripe.  Without an open end the
// round equals the full-path round bit for bit.
//
// What the shapes are for: one member's forward pass is a chain of swaths and
// its walk a chain of rows, so members run side by side (kStripeSlots, as many
// as it takes to fill the GPU with swaths), and a group has as many stripes as
// it takes to fill it with tiles.  3 members of 40k-80k samples against a 70k
// centroid, 1024-row tiles: 203 ms a round with one member at a time, one warp
// per swath and per tile and one stripe per launch (forward 60 ms, tiles 67,
// walks 76).
namespace {

constexpr int kStripeSlots = 8;       // members side by side, at most
constexpr int kStripeGroup = 4;       // stripes per group, at most
// at most, of a workspace of any size: move words of all slots' groups, and edges
// and checkpoint rows of all slots (one stripe and one slot whatever they take)
constexpr size_t kStripeGroupBytes = size_t(1) << 30;
constexpr size_t kStripeSlotBytes = size_t(4) << 30;
constexpr int kStripeFill = 512;      // swaths side by side that fill the GPU

struct StripeWalk {
  int r, c, h, cur_t, lo, hi, state;  // state: 0 walking, 1 done, 2 failed
  int s_fwd;                          // first stripe whose forward shortcut fired, or INT_MAX
  int entry;                          // row walk: the column row r was entered at
  long long nt;
};

// One member in a batch: its matrix in the round's orientation.
struct StripeMember {
  int member, flip, m, n, swaths;
  unsigned long long trip;  // offset of its path listing, in triples
};

template <typename T>
struct StripeArgs {
  const T *series;
  const uint64_t *offsets;
  const T *centroid;
  int Lc, r0, oe, shift;        // tile height K = 1 << shift
  int count;                    // members in the batch
  StripeMember mem[kStripeSlots];
  // per slot (member of the batch): strides between slots
  T *E;
  unsigned long long e_stride, e_slot;
  T *Q;
  unsigned long long q_stride, q_slot;
  unsigned long long *prog;     // one progress word per swath
  unsigned long long prog_slot;
  unsigned *words;              // move words of a group, the stripes in column order
  unsigned long long words_slot;
  unsigned long long words_all; // of all slots: the second buffer's offset
  int odd_words;                // 1: groups take two buffers in turn, 0: one buffer
  int2 *runs;                   // row walk: the column interval of every row
  unsigned long long runs_slot;
  typename CostBits<T>::U *fmin, *cmin;  // per stripe: shortcut minima (forward, below H)
  unsigned long long min_slot;
  StripeWalk *walk;
  unsigned *err;
  unsigned long long *counter;
  int2 *ranges;                 // all members' ranges, Lc per member
  int *extra;                   // all members' extra samples, or null
  int32_t *triples;             // path listings, or null
  int64_t *triple_counts;       // or null
  unsigned long long limit_ns;
};

template <typename T>
__device__ __forceinline__ const T *stripe_member_ptr(const StripeArgs<T> &a, int slot) {
  return a.series + a.offsets[a.mem[slot].member];
}

template <typename T>
__device__ __forceinline__ T stripe_corner(int c0, int r0) {
  return c0 == 0 ? (r0 ? Num<T>::big() : T(0)) : (r0 ? T(0) : Num<T>::big());
}

// The stored left edge of stripe t >= 1.
template <typename T>
__device__ __forceinline__ const T *stripe_edge(const StripeArgs<T> &a, int slot, int t) {
  return a.E + (unsigned long long)slot * a.e_slot + (unsigned long long)(t - 1) * a.e_stride;
}

// The lowest stripe of group gi, counted from the right, of `group` stripes;
// [lo, hi) with hi <= lo: none.
__host__ __device__ inline void stripe_group(int stripes, int group, int gi, int &lo, int &hi) {
  hi = stripes - gi * group;
  lo = hi - group > 0 ? hi - group : 0;
}

// Group gi's move words: with two buffers, groups take them in turn.
template <typename T>
__device__ __forceinline__ unsigned *stripe_words(const StripeArgs<T> &a, int slot, int gi) {
  return a.words + (unsigned long long)(gi & a.odd_words) * a.words_all + slot * a.words_slot;
}

// Whether the reference's re-run of stripe t at height H takes its shortcut
// branch (the whole of row H-1 OPEN_RIGHT).
template <typename T>
__device__ __forceinline__ bool stripe_fires(const StripeArgs<T> &a, int slot, int t, int H,
                                             const StripeWalk &w) {
  if (!a.oe || a.r0) return false;
  const long long L = (long long)t * kRefSwath;
  if (L <= H) return false;
  if (t >= w.s_fwd) return true;
  return CostBits<T>::of(stripe_edge(a, slot, t)[H - 1]) == a.cmin[slot * a.min_slot + t];
}

template <typename T>
__global__ void
__launch_bounds__(kBlkThreads, sizeof(T) == 4 ? kRoundBlocksF32 : kRoundBlocksF64)
    stripe_forward_kernel(StripeArgs<T> a, int max_swaths) {
  __shared__ BlockSmem<T> sm;
  const unsigned long long ntasks = (unsigned long long)a.count * max_swaths;
  for (;;) {
    if (threadIdx.x == 0) {
      unsigned long long q;
      do {
        q = atomicAdd(a.counter, 1ull);
      } while (q < ntasks && int(q / a.count) >= a.mem[q % a.count].swaths);
      sm.task = q;
    }
    __syncthreads();
    const unsigned long long q = sm.task;
    if (q >= ntasks) break;
    const int sw = int(q / a.count), slot = int(q - (unsigned long long)sw * a.count);
    const StripeMember &mem = a.mem[slot];
    const int c0 = sw * kBlkCols;
    T *E = a.E + slot * a.e_slot;
    BlockJob<T> job;
    job.x = mem.flip ? a.centroid : stripe_member_ptr(a, slot);
    job.y = mem.flip ? stripe_member_ptr(a, slot) : a.centroid;
    job.m = mem.m;
    job.n = mem.n;
    job.c0 = c0;
    job.r0 = a.r0;
    job.edge_in = sw ? E + (unsigned long long)(sw - 1) * a.e_stride : nullptr;
    job.edge_out = sw + 1 < mem.swaths ? E + (unsigned long long)sw * a.e_stride : nullptr;
    job.open_end = a.oe != 0;
    job.free_diag0 = c0 > 0;
    job.corner_init = stripe_corner<T>(c0, a.r0);
    job.words = nullptr;
    job.word_steps = 0;
    PipeGate gate;
    unsigned long long *prog = a.prog + slot * a.prog_slot;
    gate.prog_in = prog + (sw ? sw - 1 : 0);
    gate.prog_out = prog + sw;
    gate.err = a.err;
    gate.limit_ns = a.limit_ns;
    gate.avail = 0;
    T unused = T(0);
    EdgeStat<T> st;
    sweep_block<T, false, false, true, false>(
        job, sm, gate, CkptOut<T>{a.Q + slot * a.q_slot + c0, a.q_stride, a.shift}, false, unused,
        st);
    __syncthreads();
  }
}

// Shortcut minimum of the stored edge before stripe t over rows [0, H)
// (ShortcutRows), reduced into the slot's minima.  Forward pass (fwd): every
// stripe t in [tlo, thi] (stripes past the last row), H = m.  Backtrack: the
// one stripe tlo, H the walk's height, skipped where the stripe's branch is
// already decided.
template <typename T>
__global__ void stripe_min_kernel(StripeArgs<T> a, int slot, int tlo, int thi, int fwd) {
  using U = typename CostBits<T>::U;
  __shared__ U smin[256];
  const StripeWalk *wp = a.walk + slot;
  int H = a.mem[slot].m;
  if (!fwd) {
    if (wp->state != 0) return;
    H = wp->h;
    if ((long long)tlo * kRefSwath <= H || tlo >= wp->s_fwd) return;
  }
  U *out = (fwd ? a.fmin : a.cmin) + slot * a.min_slot;
  for (int t = tlo + int(blockIdx.y); t <= thi; t += int(gridDim.y)) {
    const T *e = stripe_edge(a, slot, t);
    U best = ~U(0);
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < H;
         r += (long long)gridDim.x * blockDim.x) {
      if (!shortcut_row<T>(int(r))) continue;
      const U b = CostBits<T>::of(e[r]);
      best = b < best ? b : best;
    }
    smin[threadIdx.x] = best;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s && smin[threadIdx.x + s] < smin[threadIdx.x])
        smin[threadIdx.x] = smin[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0 && smin[0] != ~U(0)) atomicMin(out + t, smin[0]);
    __syncthreads();
  }
}

// The first stripe in [tlo, thi] whose forward shortcut fires (one warp).
template <typename T>
__global__ void stripe_sfwd_kernel(StripeArgs<T> a, int slot, int tlo, int thi) {
  const int lane = threadIdx.x & 31;
  for (int t0 = tlo; t0 <= thi; t0 += 32) {
    const int t = t0 + lane;
    bool f = false;
    if (t <= thi)
      f = CostBits<T>::of(stripe_edge(a, slot, t)[a.mem[slot].m - 1]) == a.fmin[slot * a.min_slot + t];
    const unsigned ballot = __ballot_sync(kFull, f);
    if (ballot) {
      if (lane == 0) a.walk[slot].s_fwd = t0 + __ffs(ballot) - 1;
      return;
    }
  }
}

// The K-row tile kt of group gi's b-th stripe, where it lies below the
// backtrack height in w, for one block.
template <typename T>
__device__ __forceinline__ void stripe_tile(const StripeArgs<T> &a, BlockSmem<T> &sm, int group,
                                            int gi, int kt, int b, int slot, const StripeWalk &w) {
  const StripeMember &mem = a.mem[slot];
  int lo, hi;
  stripe_group(mem.swaths, group, gi, lo, hi);
  const int t = lo + b;
  if (t >= hi) return;
  const int H = w.h, K = 1 << a.shift;
  const long long rb_l = (long long)a.r0 + (long long)kt * K;
  if (w.state != 0 || rb_l >= H || stripe_fires(a, slot, t, H, w)) return;
  const int rb = int(rb_l), re = rb + K < H ? rb + K : H;
  const int c0 = t * kBlkCols;
  BlockJob<T> job;
  job.x = mem.flip ? a.centroid : stripe_member_ptr(a, slot);
  job.y = mem.flip ? stripe_member_ptr(a, slot) : a.centroid;
  job.m = re;
  job.n = mem.n;
  job.c0 = c0;
  job.r0 = rb;
  const T *left = t ? stripe_edge(a, slot, t) : nullptr;
  job.edge_in = left ? left + (unsigned long long)kt * K : nullptr;
  job.edge_out = nullptr;
  job.open_end = a.oe != 0;
  job.free_diag0 = c0 > 0;
  job.corner_init = kt == 0 ? stripe_corner<T>(c0, a.r0)
                            : (left ? left[(unsigned long long)kt * K - 1] : Num<T>::big());
  // the re-run's top row is the backtrack height's (open end)
  job.top_band = re == H;
  job.row_in = kt ? a.Q + slot * a.q_slot + (unsigned long long)(kt - 1) * a.q_stride + c0 : nullptr;
  const int steps = block_steps(mem.m - a.r0);
  job.word_steps = steps;
  job.words = stripe_words(a, slot, gi) + (size_t)(t - lo) * kBlkWarps * steps * 32 +
              (size_t)kt * (K / 2) * 32;
  T unused = T(0);
  EdgeStat<T> st;
  sweep_block<T, true, true, false, false>(job, sm, NoGate(a.err, a.limit_ns),
                                           CkptOut<T>{nullptr, 0, 1}, false, unused, st);
}

// Block (kt, b, slot): one tile of the group.
template <typename T>
__global__ void
__launch_bounds__(kBlkThreads, sizeof(T) == 4 ? kRoundBlocksF32 : kRoundBlocksF64)
    stripe_tile_kernel(StripeArgs<T> a, int group, int gi) {
  __shared__ BlockSmem<T> sm;
  const StripeWalk w = a.walk[blockIdx.z];
  stripe_tile(a, sm, group, gi, int(blockIdx.x), int(blockIdx.y), int(blockIdx.z), w);
}

template <typename T>
__global__ void stripe_walk_init_kernel(StripeArgs<T> a) {
  const int slot = threadIdx.x;
  if (slot >= a.count || blockIdx.x) return;
  StripeWalk *w = a.walk + slot;
  w->r = a.mem[slot].m - 1;
  w->c = a.mem[slot].n - 1;
  w->h = a.mem[slot].m;
  w->cur_t = -1;
  w->lo = 1;
  w->hi = 0;
  w->state = 0;
  w->s_fwd = INT_MAX;
  w->entry = a.mem[slot].n - 1;
  w->nt = 0;
}

// The row walk (walk_runs) through a group, one warp per member: without an
// open end and without a path listing.
template <typename T>
__device__ __forceinline__ void stripe_walk_runs(const StripeArgs<T> &a, int group, int gi, int slot) {
  const int lane = threadIdx.x & 31;
  const StripeMember &mem = a.mem[slot];
  int lo, hi;
  stripe_group(mem.swaths, group, gi, lo, hi);
  StripeWalk w = a.walk[slot];
  if (w.state || hi <= lo) return;
  MemberGeom g;
  g.m = mem.m;
  g.n = mem.n;
  g.r0 = a.r0;
  g.steps = block_steps(mem.m - a.r0);
  RowWalk rw{w.r, w.c, w.entry};
  const BlockMap map{reinterpret_cast<const unsigned short *>(stripe_words(a, slot, gi)), g.r0, g.steps,
                     lo * kBlkCols};
  const int got = walk_runs(map, g, lo * kBlkCols, rw, a.r0, a.runs + slot * a.runs_slot);
  if (lane == 0) {
    if (got == 2 && rw.entry >= 0) a.runs[slot * a.runs_slot + rw.r] = make_int2(0, rw.entry);
    w.r = rw.r;
    w.c = rw.c;
    w.entry = rw.entry;
    w.h = rw.r + 1;
    w.state = got;
    a.walk[slot] = w;
  }
}

template <typename T>
__global__ void __launch_bounds__(32) stripe_walk_runs_kernel(StripeArgs<T> a, int group, int gi) {
  stripe_walk_runs(a, group, gi, int(blockIdx.x));
}

// The row walk through group gi by the first blocks, one per member, and the
// tiles of group gi + 1 by the others (two word buffers, no open end).  A tile
// of group gi + 1 takes part or not by the height before or after the walk
// through group gi, whichever its block finds: the rows above the later height
// are computed for nothing, those below are the same.
//
// 3 members of 40k-80k samples against a 70k centroid: a group of 4 stripes takes
// 0.33 ms on three warps and its tiles 0.25 on the whole GPU; one after the
// other a round took 20.7 ms, beside each other 17.7 (groups of 8 stripes 18.2,
// of 2 18.3).
template <typename T>
__global__ void
__launch_bounds__(kBlkThreads, sizeof(T) == 4 ? kRoundBlocksF32 : kRoundBlocksF64)
    stripe_walk_tile_kernel(StripeArgs<T> a, int group, int gi, int tiles) {
  __shared__ BlockSmem<T> sm;
  __shared__ StripeWalk s_walk;
  if (int(blockIdx.x) < a.count) {
    if (threadIdx.x < 32) stripe_walk_runs(a, group, gi, int(blockIdx.x));
    return;
  }
  const unsigned q = blockIdx.x - a.count, per_slot = unsigned(tiles) * group;
  const int slot = int(q / per_slot), u = int(q - slot * per_slot), b = u / tiles;
  if (threadIdx.x == 0) {
    const volatile StripeWalk *w = a.walk + slot;
    s_walk.h = w->h;
    s_walk.state = w->state;
    s_walk.s_fwd = INT_MAX;
  }
  __syncthreads();
  const StripeWalk w = s_walk;
  stripe_tile(a, sm, group, gi + 1, u - b * tiles, b, slot, w);
}

// The rows' intervals as ranges (runs_to_ranges; the member on the rows).  A
// walk that failed has what it passed, as the walk by cells leaves it: all but
// the column it was in, the first.
template <typename T>
__global__ void stripe_ranges_kernel(StripeArgs<T> a) {
  const int slot = blockIdx.y;
  const StripeWalk &w = a.walk[slot];
  const bool failed = w.state == 2;
  if (w.state != 1 && !failed) return;
  runs_to_ranges(a.runs + slot * a.runs_slot,
                 a.ranges + (unsigned long long)a.mem[slot].member * a.Lc, a.mem[slot].m, false,
                 blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x,
                 failed ? (w.entry >= 0 ? w.r : w.r + 1) : 0, failed ? 1 : 0);
}

// Continues the backtrack cell by cell through a group (updateCentroid's loop,
// dba.hpp:393-421, with the stripe branch's height, dba.hpp:384-386) until it
// leaves the group to the left or reaches the start cell.  One warp per
// member: every lane holds the moves of one of the 32 rows at and below the
// current cell in a block of 32 columns, so the walk advances by shuffles and
// reloads the window only when it leaves those rows or columns.  Every lane
// keeps the same walk state; lane 0 does the stores.  The height moves to the
// walk's row when it leaves a reference stripe.
template <typename T>
__global__ void __launch_bounds__(32) stripe_walk_kernel(StripeArgs<T> a, int group, int gi) {
  const int lane = threadIdx.x, slot = blockIdx.x;
  const StripeMember &mem = a.mem[slot];
  int t_lo, t_hi;
  stripe_group(mem.swaths, group, gi, t_lo, t_hi);
  StripeWalk w = a.walk[slot];
  if (w.state || t_hi <= t_lo) return;
  const int os = a.r0, flip = mem.flip;
  const long long max_cells = (long long)mem.m + mem.n - 1;
  const BlockMap map{reinterpret_cast<const unsigned short *>(stripe_words(a, slot, gi)), a.r0,
                     block_steps(mem.m - a.r0), t_lo * kBlkCols};
  int2 *rg = a.ranges + (unsigned long long)mem.member * a.Lc;
  int *extra = a.extra ? a.extra + (unsigned long long)mem.member * a.Lc : nullptr;
  int32_t *tri = a.triples ? a.triples + 3ull * mem.trip : nullptr;
  int64_t *tri_count = a.triple_counts ? a.triple_counts + mem.member : nullptr;
  const bool lead = lane == 0;
  // rr: the member's sample index, cc: the centroid index
  auto contribute = [&](int rr, int cc) {
    if (cc != w.cur_t) {
      if (lead && w.cur_t >= 0 && w.hi >= w.lo) rg[w.cur_t] = make_int2(w.lo, w.hi);
      w.cur_t = cc;
      w.lo = rr;
      w.hi = rr;
    } else if (rr == w.lo - 1) {
      w.lo = rr;
    } else if (lead && extra) {
      // past an OPEN_RIGHT run on a re-run's top row (centroid on the rows)
      extra[cc] = rr;
    }
  };
  auto contribute_cell = [&](int r, int c) {
    if (flip)
      contribute(c, r);
    else
      contribute(r, c);
  };
  auto emit = [&](int mv) {
    if (lead && tri) {
      tri[3 * w.nt] = w.r;
      tri[3 * w.nt + 1] = w.c;
      tri[3 * w.nt + 2] = mv;
    }
    ++w.nt;
  };
  for (int t = t_hi - 1; t >= t_lo && w.state == 0; --t) {
    const int H = w.h, c0 = t * kBlkCols;
    if (stripe_fires(a, slot, t, H, w)) {
      // the re-run's shortcut: row H-1 of the stripe is OPEN_RIGHT throughout
      for (; w.c >= c0; --w.c) {
        if (w.nt >= max_cells - 1) {
          w.state = 2;
          break;
        }
        emit(kMoveOpenRight);
      }
    }
    bool stripe_done = w.c < c0 || w.state != 0;
    while (!stripe_done && w.state == 0) {
      // window: rows w.r - lane, columns cbeg .. cbeg + 31
      const int top = w.r, cbeg = w.c & ~31;
      RowMoves mine{0u, 0u};
      if (top - lane >= 1) mine = map.load(map.at(top - lane, cbeg));
      for (;;) {
        int mv;
        const unsigned rd = __shfl_sync(kFull, mine.d, (top - w.r) & 31);
        const unsigned ru = __shfl_sync(kFull, mine.u, (top - w.r) & 31);
        if (w.r == 0) {
          mv = w.c == 0 ? (os ? kMoveNilOpenRight : kMaxMoveNil) : (os ? kMoveOpenRight : kMoveRight);
        } else {
          const int j = w.c - cbeg;
          mv = ((rd >> j) & 1u) ? kMoveDiag : ((ru >> j) & 1u) ? kMoveUp : kMoveRight;
          if (mv == kMoveRight && a.oe && w.r == H - 1) mv = kMoveOpenRight;
        }
        if (mv == kMaxMoveNil || mv == kMoveNilOpenRight) {
          // the start cell (dba.hpp:412-415)
          if (mv != kMoveNilOpenRight) contribute(0, 0);
          if (lead && w.cur_t >= 0 && w.hi >= w.lo) rg[w.cur_t] = make_int2(w.lo, w.hi);
          emit(mv);
          if (lead && tri_count) *tri_count = w.nt;
          w.state = 1;
          break;
        }
        if (w.nt >= max_cells - 1) {
          w.state = 2;
          break;
        }
        emit(mv);
        if (mv != kMoveOpenRight) contribute_cell(w.r, w.c);
        if (mv == kMoveDiag) {
          --w.r;
          --w.c;
        } else if (mv == kMoveUp) {
          --w.r;
        } else {
          --w.c;
        }
        if (w.r < 0 || w.c < 0) {
          w.state = 2;
          break;
        }
        if (w.c < c0) {
          stripe_done = true;
          break;
        }
        if (top - w.r >= 32 || w.c < cbeg) break;  // reload the window
      }
    }
    if (w.state == 0 && w.c < c0) w.h = w.r + 1;
  }
  if (lead) {
    if (w.state == 2 && tri_count) *tri_count = -1;
    a.walk[slot] = w;
  }
}

// One member's matrix: rows x columns in the round's orientation.
struct StripeDims {
  int flip;
  uint64_t rows, cols;
};
inline StripeDims stripe_dims(uint64_t len, uint64_t Lc, int oe) {
  StripeDims d;
  d.flip = (oe && Lc < len) ? 1 : 0;
  d.rows = d.flip ? Lc : len;
  d.cols = d.flip ? len : Lc;
  return d;
}

struct StripeLayout {
  RoundLayout round;
  size_t off_head, off_prog, off_E, off_Q, off_W, off_runs, off_min, off_extra, total;
  unsigned long long e_stride, q_stride, words_slot, e_slot, q_slot, runs_slot, min_slot;
  int swaths_max;
  int slots, group;
  bool two;  // two word buffers (row walks beside the next group's tiles)
};

// The layout with the most members and stripes side by side whose total is at
// most `limit` bytes; the smallest layout if none is.
template <typename T>
StripeLayout stripe_layout(const uint64_t *h_lens, int n, uint64_t Lc, int os, int oe, int shift,
                           size_t limit) {
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  uint64_t max_rows = 1, max_cols = 1;
  for (int k = 0; k < n; ++k) {
    const StripeDims d = stripe_dims(h_lens[k], Lc, oe);
    max_rows = d.rows > max_rows ? d.rows : max_rows;
    max_cols = d.cols > max_cols ? d.cols : max_cols;
  }
  StripeLayout S;
  S.round = round_layout<T>(n, 1, 0, (unsigned long long)n * Lc, 1);
  S.swaths_max = int((max_cols + kBlkCols - 1) / kBlkCols);
  S.e_stride = (max_rows + 64 + 31) / 32 * 32;
  S.q_stride = (unsigned long long)S.swaths_max * kBlkCols;
  const unsigned long long K = 1ull << shift;
  const unsigned long long nq = (max_rows - (os ? 1 : 0)) / K + 1;
  S.e_slot = (unsigned long long)(S.swaths_max > 1 ? S.swaths_max - 1 : 1) * S.e_stride;
  S.q_slot = nq * S.q_stride;
  S.min_slot = (unsigned long long)S.swaths_max + 1;
  const size_t stripe_bytes = size_t(kBlkWarps) * block_steps(int(max_rows)) * 32 * 4;
  // the offsets of one choice of slots, stripes per group, word buffers and
  // row intervals
  auto place = [&](int slots, int group, bool two, bool by_runs) {
    S.slots = slots;
    S.group = group;
    S.two = two;
    S.words_slot = stripe_bytes / 4 * group;
    S.runs_slot = by_runs ? max_rows : 0;
    size_t o = S.round.total;
    S.off_head = o; o += 1024;
    S.off_prog = o; o += up(size_t(slots) * S.swaths_max * 8);
    S.off_E = o; o += up(size_t(slots) * S.e_slot * sizeof(T));
    S.off_Q = o; o += up(size_t(slots) * S.q_slot * sizeof(T));
    S.off_W = o; o += up(size_t(slots) * S.words_slot * 4 * (two ? 2 : 1));
    S.off_runs = o; o += up(size_t(slots) * S.runs_slot * sizeof(int2));
    // with an open end: the extra samples, and the shortcut minima of every stripe
    S.off_extra = o; o += oe ? up(size_t(n) * Lc * 4) : 0;
    S.off_min = o; o += oe ? (size_t(2) * slots * S.min_slot * sizeof(T) + 63) / 64 * 64 : 0;
    S.total = o;
    return S.total <= limit;
  };
  const size_t slot_bytes = size_t(S.e_slot + S.q_slot) * sizeof(T);
  int slots = (kStripeFill + S.swaths_max - 1) / S.swaths_max;
  if (slots > kStripeSlots) slots = kStripeSlots;
  if (slots > n) slots = n;
  while (slots > 1 && slot_bytes * slots > kStripeSlotBytes) --slots;
  // the most side by side that fits: first without the second word buffer,
  // then with fewer stripes per group, then fewer members; last one member,
  // one stripe and no row intervals (the walk goes cell by cell)
  for (; slots >= 1; --slots) {
    int group = S.swaths_max < kStripeGroup ? S.swaths_max : kStripeGroup;
    while (group > 1 && stripe_bytes * group * slots > kStripeGroupBytes) --group;
    if (S.swaths_max > group && 2 * stripe_bytes * group * slots <= kStripeGroupBytes &&
        place(slots, group, true, true))
      return S;
    for (; group >= 1; --group)
      if (place(slots, group, false, true)) return S;
  }
  place(1, 1, false, false);
  return S;
}

// What a workspace may take: 95 % of the device memory that is free, or no
// limit where there is no device to ask.
size_t stripe_memory_limit() {
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) == cudaSuccess) return fr / 20 * 19;
  cudaGetLastError();
  return SIZE_MAX;
}

int stripe_shift(int ckpt_rows) {
  if (ckpt_rows == 0) return 12;  // 4096 rows per tile
  if (ckpt_rows < 2 || (ckpt_rows & (ckpt_rows - 1))) return -1;
  int sh = 0;
  while ((1 << sh) < ckpt_rows) ++sh;
  return sh;
}

}  // namespace

template <typename T>
size_t dba_round_stripe_workspace_bytes(const uint64_t *h_lens, int n, uint64_t Lc, int os, int oe,
                                        int ckpt_rows) {
  const int sh = stripe_shift(ckpt_rows);
  if (sh < 0 || n < 1 || Lc == 0) return 0;
  return stripe_layout<T>(h_lens, n, Lc, os, oe, sh, stripe_memory_limit()).total;
}

template <typename T>
int dba_round_stripe_launch(const T *centroid, uint64_t Lc, const T *series,
                            const uint64_t *offsets, const uint64_t *lens, const uint64_t *h_lens,
                            int n, int os, int oe, int ckpt_rows, T *mean, uint32_t *counts,
                            double *delta, int32_t *triples, int64_t *triple_counts, void *ws,
                            size_t ws_bytes, cudaStream_t stream) {
  const int sh = stripe_shift(ckpt_rows);
  if (sh < 0) return fail(ODBA_ERR_INVALID_ARGUMENT, "checkpoint rows must be a power of two >= 2 (0: default)");
  const StripeLayout S = stripe_layout<T>(h_lens, n, Lc, os, oe, sh, ws_bytes);
  if (ws_bytes < S.total) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "stripe DBA round workspace too small");
  const RoundLayout &L = S.round;
  char *base = static_cast<char *>(ws);
  const int flags = (os ? 1 : 0) | (oe ? 2 : 0) | 4;
  int *extra = oe ? reinterpret_cast<int *>(base + S.off_extra) : nullptr;
  RoundArgs<T> a = single_job_round<T>(centroid, Lc, series, offsets, lens, n, flags, L, base, stream);
  a.means = mean;
  a.counts = counts;
  a.deltas = delta;
  a.triples = triples;
  a.triple_counts = triple_counts;
  a.extra = extra;
  a.counter = reinterpret_cast<unsigned long long *>(base + L.off_counter);
  a.path_off = reinterpret_cast<unsigned long long *>(base + L.off_path);
  a.trip_off = reinterpret_cast<unsigned long long *>(base + L.off_trip);
  a.rng_off = reinterpret_cast<unsigned long long *>(base + L.off_rng);
  a.shortcut = reinterpret_cast<int *>(base + L.off_short);
  a.ranges = reinterpret_cast<int2 *>(base + L.off_ranges);
  a.edges = reinterpret_cast<T *>(base + L.off_edges);
  a.edge_stride = L.edge_stride;
  a.words = reinterpret_cast<unsigned long long *>(base + L.off_words);
  const unsigned long long nr = (unsigned long long)n * Lc;
  plan_kernel<T><<<1, kPlanThreads, 0, stream>>>(a);
  fill_ranges_kernel<<<int(nr / 256 + 1 < 4096 ? nr / 256 + 1 : 4096), 256, 0, stream>>>(a.ranges, nr);
  if (extra) cudaMemsetAsync(extra, 0xff, size_t(nr) * 4, stream);
  if (int rc = check_launch("stripe DBA round set-up")) return rc;

  char *head = base + S.off_head;
  StripeArgs<T> sa;
  sa.series = series;
  sa.offsets = offsets;
  sa.centroid = centroid;
  sa.Lc = int(Lc);
  sa.r0 = os ? 1 : 0;
  sa.oe = oe ? 1 : 0;
  sa.shift = sh;
  sa.E = reinterpret_cast<T *>(base + S.off_E);
  sa.e_stride = S.e_stride;
  sa.e_slot = S.e_slot;
  sa.Q = reinterpret_cast<T *>(base + S.off_Q);
  sa.q_stride = S.q_stride;
  sa.q_slot = S.q_slot;
  sa.prog = reinterpret_cast<unsigned long long *>(base + S.off_prog);
  sa.prog_slot = (unsigned long long)S.swaths_max;
  sa.words = reinterpret_cast<unsigned *>(base + S.off_W);
  sa.words_slot = S.words_slot;
  sa.words_all = (unsigned long long)S.slots * S.words_slot;
  sa.runs = reinterpret_cast<int2 *>(base + S.off_runs);
  sa.runs_slot = S.runs_slot;
  sa.fmin = oe ? reinterpret_cast<typename CostBits<T>::U *>(base + S.off_min) : nullptr;
  sa.min_slot = S.min_slot;
  sa.cmin = oe ? sa.fmin + S.slots * S.min_slot : nullptr;
  sa.counter = reinterpret_cast<unsigned long long *>(head);
  sa.walk = reinterpret_cast<StripeWalk *>(head + 64);
  // the wait error word is byte 8 of the workspace, as in the full-path round
  sa.err = reinterpret_cast<unsigned *>(base + L.off_counter + 8);
  cudaMemsetAsync(base + L.off_counter, 0, 16, stream);
  sa.ranges = a.ranges;
  sa.extra = extra;
  sa.triples = triples;
  sa.triple_counts = triple_counts;
  sa.limit_ns = kWaitLimitNs;
  static_assert(64 + kStripeSlots * sizeof(StripeWalk) <= 1024, "walk states fit the header");
  const bool check_short = oe && !os;
  const bool by_rows = !oe && !triples && S.runs_slot;
  const int K = 1 << sh;
  const int group = oe ? 1 : S.group;
  const bool beside = by_rows && S.two;
  sa.odd_words = beside ? 1 : 0;
  unsigned long long trip = 0;
  for (int k0 = 0; k0 < n; k0 += S.slots) {
    sa.count = n - k0 < S.slots ? n - k0 : S.slots;
    int max_swaths = 0, max_m = 0;
    unsigned long long all_swaths = 0;
    for (int i = 0; i < sa.count; ++i) {
      const StripeDims d = stripe_dims(h_lens[k0 + i], Lc, oe);
      StripeMember &mem = sa.mem[i];
      mem.member = k0 + i;
      mem.flip = d.flip;
      mem.m = int(d.rows);
      mem.n = int(d.cols);
      mem.swaths = (mem.n + kBlkCols - 1) / kBlkCols;
      mem.trip = trip;
      trip += h_lens[k0 + i] + Lc + 1;
      max_swaths = mem.swaths > max_swaths ? mem.swaths : max_swaths;
      max_m = mem.m > max_m ? mem.m : max_m;
      all_swaths += mem.swaths;
    }
    cudaMemsetAsync(head, 0, 64, stream);
    cudaMemsetAsync(sa.prog, 0, size_t(S.slots) * S.swaths_max * 8, stream);
    if (check_short)
      cudaMemsetAsync(sa.fmin, 0xff, size_t(2) * S.slots * S.min_slot * sizeof(T), stream);
    stripe_walk_init_kernel<T><<<1, 32, 0, stream>>>(sa);
    const int resident = round_grid<T>();
    const int fgrid = all_swaths < (unsigned long long)resident ? int(all_swaths) : resident;
    stripe_forward_kernel<T><<<fgrid, kBlkThreads, 0, stream>>>(sa, max_swaths);
    auto min_blocks = [](int m) { return (m + 2047) / 2048 < 64 ? (m + 2047) / 2048 : 64; };
    if (check_short) {
      // stripes past the last row: where the forward pass's shortcut fired first
      for (int i = 0; i < sa.count; ++i) {
        const int tlo = sa.mem[i].m / kRefSwath + 1, thi = sa.mem[i].swaths - 1;
        if (tlo > thi) continue;
        const int gy = thi - tlo + 1 < 1024 ? thi - tlo + 1 : 1024;
        stripe_min_kernel<T><<<dim3(min_blocks(sa.mem[i].m), gy), 256, 0, stream>>>(sa, i, tlo, thi, 1);
        stripe_sfwd_kernel<T><<<1, 32, 0, stream>>>(sa, i, tlo, thi);
      }
    }
    const int tiles = (max_m - sa.r0 + K - 1) / K > 0 ? (max_m - sa.r0 + K - 1) / K : 1;
    for (int gi = 0; gi * group < max_swaths; ++gi) {
      if (check_short)
        for (int i = 0; i < sa.count; ++i) {
          const int t = sa.mem[i].swaths - 1 - gi;
          // (rows below H reach a stripe's shortcut only past column H)
          if (t >= 1) stripe_min_kernel<T><<<dim3(min_blocks(sa.mem[i].m), 1), 256, 0, stream>>>(sa, i, t, t, 0);
        }
      if (!beside || gi == 0)
        stripe_tile_kernel<T><<<dim3(tiles, group, sa.count), kBlkThreads, 0, stream>>>(sa, group, gi);
      if (beside && (gi + 1) * group < max_swaths)
        stripe_walk_tile_kernel<T><<<sa.count + tiles * group * sa.count, kBlkThreads, 0, stream>>>(
            sa, group, gi, tiles);
      else if (by_rows)
        stripe_walk_runs_kernel<T><<<sa.count, 32, 0, stream>>>(sa, group, gi);
      else
        stripe_walk_kernel<T><<<sa.count, 32, 0, stream>>>(sa, group, gi);
    }
    if (by_rows)
      stripe_ranges_kernel<T><<<dim3((max_m + 255) / 256 < 256 ? (max_m + 255) / 256 : 256, sa.count), 256,
                                0, stream>>>(sa);
    if (int rc = check_launch("stripe DBA round member kernels")) return rc;
  }
  dim3 rg((unsigned(Lc) + kReduceWarps - 1) / kReduceWarps, 1);
  reduce_kernel<T><<<rg, kReduceThreads, 0, stream>>>(a);
  return check_launch("stripe DBA round reduce");
}

template size_t dba_round_stripe_workspace_bytes<float>(const uint64_t *, int, uint64_t, int, int, int);
template size_t dba_round_stripe_workspace_bytes<double>(const uint64_t *, int, uint64_t, int, int, int);
template int dba_round_stripe_launch<float>(const float *, uint64_t, const float *, const uint64_t *,
                                            const uint64_t *, const uint64_t *, int, int, int, int,
                                            float *, uint32_t *, double *, int32_t *, int64_t *,
                                            void *, size_t, cudaStream_t);
template int dba_round_stripe_launch<double>(const double *, uint64_t, const double *,
                                             const uint64_t *, const uint64_t *, const uint64_t *,
                                             int, int, int, int, double *, uint32_t *, double *,
                                             int32_t *, int64_t *, void *, size_t, cudaStream_t);

// ---------------------------------------------------------------------------
// Prefix chop (chopPrefixFromSequences, dba.hpp:1191-1395): every series is
// aligned to the leader with open-end DTW and a recorded path (leader on the
// rows, whatever the lengths), by the DBA round's path kernels; then one warp
// per series walks its path (chop_walk_kernel).
namespace {
constexpr int kChopFlags = 2 | 4 | 8;  // open end, active, centroid (the leader) on the rows
}  // namespace

template <typename T>
size_t prefix_chop_workspace_bytes(const uint64_t *h_lens, int n, uint64_t P) {
  unsigned long long words, ranges, maxm;
  const uint64_t clen = P;
  const int flags = kChopFlags;
  int ms = 1;
  unsigned long long units = 0;
  host_totals<T>(h_lens, nullptr, n, &clen, &flags, words, ranges, maxm, &ms, nullptr, &units);
  if (P > maxm) maxm = P;
  return round_layout<T>(n, 1, words, ranges, maxm, ms, 0, units).total;
}

template <typename T>
int prefix_chop_launch(const T *prefix, uint64_t P, const T *series, const uint64_t *offsets,
                       const uint64_t *lens, const uint64_t *h_lens, int n, long long *chop,
                       int *hist, void *ws, size_t ws_bytes, cudaStream_t stream) {
  unsigned long long words, ranges, maxm;
  const uint64_t clen = P;
  const int flags = kChopFlags;
  int ms = 1;
  unsigned long long units = 0;
  host_totals<T>(h_lens, nullptr, n, &clen, &flags, words, ranges, maxm, &ms, nullptr, &units);
  if (P > maxm) maxm = P;
  const RoundLayout L = round_layout<T>(n, 1, words, ranges, maxm, ms, 0, units);
  if (ws_bytes < L.total) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "prefix chop workspace too small");
  char *base = static_cast<char *>(ws);
  int *single = reinterpret_cast<int *>(base + L.off_single);
  int *mseries = single, *mjob = single + n, *d_clen = single + 2 * n, *d_flags = single + 2 * n + 1,
      *d_mbeg = single + 2 * n + 2, *d_mend = single + 2 * n + 3;
  unsigned long long *d_coff =
      reinterpret_cast<unsigned long long *>(base + L.off_single + ((size_t(2 * n + 4) * 4 + 7) / 8) * 8);
  single_job_kernel<<<(n + 255) / 256, 256, 0, stream>>>(mseries, mjob, n, d_clen, int(P), d_flags,
                                                        flags, d_mbeg, d_mend, d_coff);
  RoundArgs<T> a;
  a.centroids = prefix;
  a.coff = d_coff;
  a.clen = d_clen;
  a.jflags = d_flags;
  a.mbeg = d_mbeg;
  a.mend = d_mend;
  a.njobs = 1;
  a.series = series;
  a.offsets = offsets;
  a.lens = lens;
  a.mseries = mseries;
  a.mjob = mjob;
  a.order = nullptr;
  a.nmem = n;
  a.means = nullptr;
  a.counts = nullptr;
  // the planner clears the job's delta: a spare word of the counter block
  a.deltas = reinterpret_cast<double *>(base + L.off_counter + 16);
  a.triples = nullptr;
  a.triple_counts = nullptr;
  cudaMemsetAsync(hist, 0, size_t(n) * P * sizeof(int), stream);
  launch_paths<T>(a, L, base, stream);
  chop_walk_kernel<T><<<(n + kRoundWarps - 1) / kRoundWarps, kRoundWarps * 32, 0, stream>>>(a, chop, hist,
                                                                                          int(P));
  return check_launch("prefix chop kernels");
}

template size_t prefix_chop_workspace_bytes<float>(const uint64_t *, int, uint64_t);
template size_t prefix_chop_workspace_bytes<double>(const uint64_t *, int, uint64_t);
template int prefix_chop_launch<float>(const float *, uint64_t, const float *, const uint64_t *,
                                       const uint64_t *, const uint64_t *, int, long long *, int *,
                                       void *, size_t, cudaStream_t);
template int prefix_chop_launch<double>(const double *, uint64_t, const double *, const uint64_t *,
                                        const uint64_t *, const uint64_t *, int, long long *, int *,
                                        void *, size_t, cudaStream_t);

template size_t dba_round_workspace_bytes<float>(const uint64_t *, int, uint64_t, int, int);
template size_t dba_round_workspace_bytes<double>(const uint64_t *, int, uint64_t, int, int);
template int dba_round_launch<float>(const float *, uint64_t, const float *, const uint64_t *,
                                     const uint64_t *, const uint64_t *, int, int, int, float *,
                                     uint32_t *, double *, int32_t *, int64_t *, void *, size_t,
                                     cudaStream_t);
template int dba_round_launch<double>(const double *, uint64_t, const double *, const uint64_t *,
                                      const uint64_t *, const uint64_t *, int, int, int, double *,
                                      uint32_t *, double *, int32_t *, int64_t *, void *, size_t,
                                      cudaStream_t);
template int dba_round_ranges_launch<float>(const float *, uint64_t, const float *, const uint64_t *,
                                            const uint64_t *, const uint64_t *, int, int, int, int2 *,
                                            void *, size_t, cudaStream_t);
template int dba_round_ranges_launch<double>(const double *, uint64_t, const double *,
                                             const uint64_t *, const uint64_t *, const uint64_t *, int,
                                             int, int, int2 *, void *, size_t, cudaStream_t);
template size_t dba_reduce_workspace_bytes<float>(int);
template size_t dba_reduce_workspace_bytes<double>(int);
template int dba_reduce_ranges_launch<float>(const float *, uint64_t, const float *, const uint64_t *,
                                             const uint64_t *, int, int, int, const int2 *, float *,
                                             uint32_t *, double *, void *, size_t, cudaStream_t);
template int dba_reduce_ranges_launch<double>(const double *, uint64_t, const double *,
                                              const uint64_t *, const uint64_t *, int, int, int,
                                              const int2 *, double *, uint32_t *, double *, void *,
                                              size_t, cudaStream_t);
template size_t dba_batch_workspace_bytes<float>(const uint64_t *, const int *, int,
                                                 const uint64_t *, const int *, int);
template size_t dba_batch_workspace_bytes<double>(const uint64_t *, const int *, int,
                                                  const uint64_t *, const int *, int);
template int dba_batch_launch<float>(const float *, const unsigned long long *, const int *,
                                     const int *, const int *, const int *, int, int,
                                     const float *, const uint64_t *, const uint64_t *,
                                     const int *, const int *, const int *, int, const uint64_t *,
                                     const int *, const uint64_t *, const int *, float *,
                                     uint32_t *, double *, int32_t *, int64_t *, void *, size_t,
                                     cudaStream_t);
template int dba_batch_launch<double>(const double *, const unsigned long long *, const int *,
                                      const int *, const int *, const int *, int, int,
                                      const double *, const uint64_t *, const uint64_t *,
                                      const int *, const int *, const int *, int,
                                      const uint64_t *, const int *, const uint64_t *, const int *,
                                      double *, uint32_t *, double *, int32_t *, int64_t *, void *,
                                      size_t, cudaStream_t);

}  // namespace odba
