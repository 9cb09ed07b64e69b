// One warp sweeps one swath of a cost matrix: the form that fills the GPU with
// many matrices at the least cost per cell.
//
// Rows come in chunks of 32 pairs.  The warp stages a chunk's samples and
// left-edge values in shared memory while it sweeps the chunk before, collects
// the right edge there and stores it 32 pairs at a time, so that a step is the
// cells, two shuffles, two shared loads and one shared store and no lane
// branches.  Lanes outside the matrix compute values nobody reads: above the
// first row a lane is re-set when it reaches it (the first 31 steps), below the
// last row nothing is stored; only the steps that need the open-end top row or
// the last cell run a slower form, and a last swath ends with the last cell.
//
// What bounds it: the issue port.  A float cell is half a packed subtraction, a
// three-input minimum and a multiply-add, 3.9 cycles per warp cell and scheduler
// in a loop of nothing else; a double one two compare-and-selects, 13.6.  300
// float series of 2000-8000 samples (all pairs): 4.5 cycles per cell, padding
// and fill included, 141 ms (a form that shuffled and packed the samples and
// stored the edge from one lane by branch: 147).
//
// PATH records moves (dtw_path.cuh), for rounds large enough to fill the GPU
// with one warp per swath: per step and lane 2 * WarpMoves<T>::kWords words, row
// a's then row b's (float: D and U plane of 32 bits; double: one word, D in its
// low half): word of (step t, lane l, row) of a swath at
// ((t * 32 + l) * 2 + row) * kWords.
#pragma once

#include <type_traits>

#include "dtw_path.cuh"

namespace odba {

constexpr int kWarpChunk = 32;  // row pairs (steps) per chunk

template <typename T>
struct WarpSmem {
  // the pairs of two chunks, twice: a chunk's reads (pair t - lane) never wrap
  alignas(16) XPair<T> x[4 * kWarpChunk];
  alignas(16) T ein[2 * kWarpChunk];   // left edge of the chunk
  alignas(16) T eout[2 * kWarpChunk];  // right edge, pair t - 31 at step t
  alignas(16) T sink[2 * kWarpChunk];  // where the lanes without a right edge store
};

// Words of a row's moves per step and lane.
template <typename T>
struct WarpMoves;
template <>
struct WarpMoves<float> {
  static constexpr int kBits = 32, kWords = 2;
  using V = uint4;
  static __device__ __forceinline__ V pack(const unsigned (&w)[4]) {
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
};
template <>
struct WarpMoves<double> {
  static constexpr int kBits = 16, kWords = 1;
  using V = uint2;
  static __device__ __forceinline__ V pack(const unsigned (&w)[4]) { return make_uint2(w[0], w[1]); }
};

// The gate of a warp that sweeps a matrix's swaths in turn: nothing to wait for.
struct SoloGate {
  static constexpr bool kActive = false;
  __device__ __forceinline__ void wait(int) {}
  __device__ __forceinline__ void publish(int) {}
};

// One swath for one warp.
template <typename T>
struct SwathJob {
  const T *x;         // first series (rows), length m
  const T *y;         // second series (columns), length n
  int m, n;
  int c0;             // first column of this swath
  int r0;             // first computed row: 0, or 1 with open start (row 0 is all zeros)
  const T *edge_in;   // C[r][c0-1] by r - r0, or nullptr for the first swath
  T *edge_out;        // receives C[r][c_last] by r - r0, or nullptr
  bool open_end;
  bool free_diag0;    // column c0 is a reference swath-left column (c0 % 1024 == 0, c0 > 0)
  bool track = false; // keep the right edge's EdgeStat (needs edge_out)
  T corner_init;      // diagonal input of lane 0 at its first row
  unsigned *words = nullptr;  // move words of this swath (PATH)
};

// Sweeps one swath.  last: the swath holds column n - 1; corner then receives
// cell (m - 1, n - 1) in every lane (not with PATH).  Returns the right edge's
// EdgeStat in every lane (the big value unless job.track).  Gate: the left edge
// is another warp's, which publishes its rows, and the right edge is published.
template <typename T, int R, bool PATH = false, typename Gate = SoloGate>
__device__ __forceinline__ EdgeStat<T> sweep_warp(const SwathJob<T> &job, WarpSmem<T> &sm, bool last,
                                                  T &corner, Gate gate = Gate()) {
  using V2 = typename Pair2<T>::V;
  const int lane = threadIdx.x & 31;
  const int r0 = job.r0, rows = job.m - r0;
  const T init = r0 ? T(0) : Num<T>::big();
  EdgeStat<T> st{Num<T>::big(), Num<T>::big()};
  if (rows <= 0) {  // open start over a single row: all zeros
    if (last && !PATH) corner = init;
    return st;
  }
  const int pairs = (rows + 1) / 2;
  YCols<T, R> yv;
  yv.load(job.y, job.c0 + lane * R, job.n);
  T col[R];
#pragma unroll
  for (int j = 0; j < R; ++j) col[j] = init;
  T a_last = init, dg = init;
  const bool lane0 = lane == 0, lane31 = lane == 31;
  const T dinit = lane0 ? job.corner_init : init;
  const bool fd0 = job.free_diag0 && lane0;
  const bool has_in = job.edge_in != nullptr, has_out = job.edge_out != nullptr;
  const int last_pair = (rows - 1) >> 1;
  const bool last_is_b = ((rows - 1) & 1) != 0;
  const bool oe_top = job.open_end && job.m >= 2;  // a single-row matrix has no open-end rule
  // the lane and register of column n - 1, and the step that computes the last
  // cell: the last one of a last swath, which has no right edge
  const bool cap_last = last && !PATH;
  const int cap_lane = cap_last ? (job.n - 1 - job.c0) / R : 0;
  const int capj = cap_last ? job.n - 1 - job.c0 - cap_lane * R : -1;
  const int steps = cap_last ? last_pair + cap_lane + 1 : pairs + 31;
  // the steps from slow0 on run the slow form
  const int slow0 = oe_top ? last_pair : cap_last ? steps - 1 : steps;
  using Moves = typename WarpMoves<T>::V;
  Moves *wp = PATH ? reinterpret_cast<Moves *>(job.words) + lane : nullptr;

  // the left edge's rows of pairs [0, k)
  auto await = [&](int k) {
    if (Gate::kActive && has_in) {
      if (lane == 0) gate.wait(2 * k < rows ? 2 * k : rows);
      __syncwarp();
    }
  };

  // this lane's row pair of the next chunk
  T nx0 = T(0), nx1 = T(0), ne0 = T(0), ne1 = T(0);
  auto load = [&](int k) {
    if (k >= pairs) return;
    const int row = 2 * k;
    nx0 = job.x[r0 + row];
    nx1 = job.x[r0 + (row + 1 < rows ? row + 1 : row)];
    if (has_in) {
      const V2 e = __ldcg(reinterpret_cast<const V2 *>(job.edge_in + row));
      ne0 = e.x;
      ne1 = e.y;
    }
  };
  auto put = [&](int k) {
    if (k >= pairs) return;
    XPair<T> *p = &sm.x[k & (2 * kWarpChunk - 1)];
    XPair<T>::put(p, 0, nx0);
    XPair<T>::put(p, 1, nx1);
    p[2 * kWarpChunk] = p[0];
    if (has_in) {
      sm.ein[2 * lane] = ne0;
      sm.ein[2 * lane + 1] = ne1;
    }
  };
  if (!has_in) sm.ein[2 * lane] = sm.ein[2 * lane + 1] = Num<T>::big();
  await(kWarpChunk);
  load(lane);
  put(lane);
  __syncwarp();

  V2 *os = reinterpret_cast<V2 *>(lane31 ? sm.eout : sm.sink);
  const V2 *es = reinterpret_cast<const V2 *>(sm.ein);
  // One copy of each form of the step: what runs next to other swath widths has
  // to share the instruction cache with them.  Double has a loop of its own for
  // the chunks without a slow step all the same (kApart): beside the slow form its
  // two rows' chains were scheduled one after the other (one pair of 1000 x 1000
  // 0.62 ms so, 0.37 apart; 100 series of 1000-4000 13.6 and 12.6); float 147 us
  // and 142 ms either way.
  constexpr bool kApart = sizeof(T) == 8;
  auto chunk = [&](auto mixed_c, int t0, int lim) {
    constexpr bool MIXED = decltype(mixed_c)::value;
    await(t0 + 2 * kWarpChunk);
    load(t0 + kWarpChunk + lane);
    const XPair<T> *xs = sm.x + ((t0 - lane) & (2 * kWarpChunk - 1));
    auto step = [&](auto slow_c, int s) {
      constexpr bool SLOW = decltype(slow_c)::value;
      const XPair<T> xv = xs[s];
      const V2 ev = es[s];
      T la = __shfl_up_sync(kFull, a_last, 1);
      T lb = __shfl_up_sync(kFull, col[R - 1], 1);
      la = lane0 ? ev.x : la;
      lb = lane0 ? ev.y : lb;
      const T diag = dg;
      dg = lb;
      unsigned word[4] = {0u, 0u, 0u, 0u};
      const int k = t0 + s - lane;
      const bool top = SLOW && oe_top && k == last_pair;
      a_last = step_row_pair<T, R, PATH, SLOW, SLOW && !PATH, PATH ? WarpMoves<T>::kBits : 8>(
          col, yv, xv, la, lb, diag, top && !last_is_b, top && last_is_b, fd0, word,
          SLOW && k == last_pair && !last_is_b);
      if (PATH) wp[(size_t)(t0 + s) * 32] = WarpMoves<T>::pack(word);
      V2 v;
      v.x = a_last;
      v.y = col[R - 1];
      os[s] = v;
    };
    for (int s = 0; s < lim;) {
      if (t0 == 0 && s == lane) {  // the lane's first row pair
        dg = dinit;
#pragma unroll
        for (int j = 0; j < R; ++j) col[j] = init;
      }
      int s1 = t0 == 0 ? s + 1 : lim;
      if (!MIXED || t0 + s < slow0) {
        if (MIXED && s1 > slow0 - t0) s1 = slow0 - t0;
#pragma unroll 1
        for (; s < s1; ++s) step(std::false_type{}, s);
      } else {
        step(std::true_type{}, s);
        ++s;
      }
    }
    __syncwarp();
    if (has_out) {
      const int k = t0 - 31 + lane, row = 2 * k;
      if (lane < lim && k >= 0 && row < rows) {
        const V2 v = reinterpret_cast<const V2 *>(sm.eout)[lane];
        __stcg(reinterpret_cast<V2 *>(job.edge_out + row), v);
        if (job.track) {
          if (shortcut_row<T>(r0 + row)) st.emin = Num<T>::min2(st.emin, v.x);
          if (row == rows - 1) st.etop = v.x;
          if (row + 1 < rows) {
            if (shortcut_row<T>(r0 + row + 1)) st.emin = Num<T>::min2(st.emin, v.y);
            if (row + 1 == rows - 1) st.etop = v.y;
          }
        }
      }
    }
    put(t0 + kWarpChunk + lane);
    __syncwarp();
    if (Gate::kActive && has_out && lane == 0) {
      const int stored = 2 * (t0 - 31 + lim);
      if (stored > 0) gate.publish(stored < rows ? stored : rows);
    }
  };
  int t0 = 0;
  if (kApart)
    for (; t0 < steps; t0 += kWarpChunk) {
      const int lim = steps - t0 < kWarpChunk ? steps - t0 : kWarpChunk;
      if (t0 + lim > slow0) break;
      chunk(std::false_type{}, t0, lim);
    }
  for (; t0 < steps; t0 += kWarpChunk)
    chunk(std::true_type{}, t0, steps - t0 < kWarpChunk ? steps - t0 : kWarpChunk);
  if (job.track) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      st.emin = Num<T>::min2(st.emin, __shfl_xor_sync(kFull, st.emin, off));
    // every lane the same figures, whatever the values: the warp goes on or
    // stops by them.  The last row's value is the one of the lane that stored
    // it (a minimum with the other lanes' big would lose a NaN or an infinity).
    st.emin = __shfl_sync(kFull, st.emin, 0);
    st.etop = __shfl_sync(kFull, st.etop, (last_pair + 31) & 31);
  }
  if (cap_last) {
    T cap = T(0);
#pragma unroll
    for (int j = 0; j < R; ++j) cap = capj == j ? col[j] : cap;
    corner = __shfl_sync(kFull, cap, cap_lane);
  }
  return st;
}

}  // namespace odba
