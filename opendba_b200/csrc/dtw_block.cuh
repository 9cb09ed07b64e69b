// A thread block sweeps one 1024-column swath of a cost matrix: four compute
// warps in a row and a fifth warp feeding them.
//
// Why a block per swath: a one-warp swath (dtw_warp.cuh) is the cheapest
// way to fill the GPU with many matrices, but a matrix is then a chain of
// long steps -- 64 cells per lane, about 800 cycles for a warp that records
// moves and has the scheduler to itself -- and few matrices leave most
// schedulers idle.  Four warps of 8 columns per lane take a step in about a
// quarter of that and need a third of the registers.
//
// Warp w owns columns c0 + 256 w .. + 255, lane l of it the 8 columns from
// 8 (32 w + l).  A step takes a lane two rows down (row pair k = rows
// r0 + 2k, r0 + 2k + 1); lane l works on pair t - l at its warp's step t.
// Steps run in chunks of kBlkChunk.  A warp starts a chunk when its left
// neighbour has written the edge pairs the chunk reads (or the feeder has
// staged them) and its own edge ring has room; every warp counts the steps it
// has done in shared memory.  (A barrier per chunk instead makes every block
// wait for its slowest scheduler: half of all warp time at full load.)
//
// The fifth warp owns everything that touches global memory at the edges: it
// stages the rows' samples and the left edge ahead, stores the right edge,
// publishes it to the block that sweeps the next swath (PipeGate) and keeps
// the edge's open-end shortcut figures.  Its waits and fences overlap the
// compute warps' steps.
//
// Lanes outside the matrix compute values nobody reads: above the first row a
// lane is re-set when it reaches it (the FILL steps), below the last row its
// edge values are not stored and its move words have slots of their own.
//
// Moves: per step a lane stores one 32-bit word, row a in the low half, row b
// in the high half, each half D bits 0-7 and U bits 8-15 (register j's bit j;
// dtw_path.cuh says what D and U are): a warp writes 128 contiguous bytes.
// Word of (warp w, step t, lane l) of a swath: (w * steps + t) * 32 + l with
// steps of block_steps.
//
// Waits inside the block are on counters that warps of the same block raise
// without waiting on the waiter (a warp waits for its left neighbour's steps,
// or for room its right neighbour frees; the feeder never blocks on one of
// its duties while another could go on); they are bounded like the waits
// between blocks (dtw_pipe.cuh).
#pragma once

#include <type_traits>

#include "dtw_path.cuh"
#include "dtw_pipe.cuh"

namespace odba {

constexpr int kBlkWarps = 4;                          // compute warps
constexpr int kBlkR = 8;                              // columns per lane
constexpr int kBlkWarpCols = 32 * kBlkR;
constexpr int kBlkCols = kBlkWarps * kBlkWarpCols;    // one reference swath
constexpr int kBlkThreads = 32 * (kBlkWarps + 1);
constexpr int kBlkChunk = 8;                          // steps between counter checks
constexpr int kBlkSlack = 8;                          // extra steps a waiting warp waits for
constexpr int kBlkStage = 16;                         // row pairs the feeder moves at once
constexpr int kBlkRing = 128;                         // row pairs per edge ring
constexpr int kBlkXPairs = 512;                       // row pairs of staged samples
static_assert(kBlkCols == kRefSwath, "the open-end rules act on 1024-column swaths");
static_assert(kBlkXPairs >= kBlkWarps * (31 + kBlkChunk) + 2 * kBlkStage, "sample ring");
static_assert(kBlkRing >= 31 + 2 * kBlkChunk + kBlkStage, "edge ring");

// Steps of a swath of `rows` rows, in whole chunks.
__host__ __device__ inline int block_steps(int rows) {
  return ((rows + 1) / 2 + 31 + kBlkChunk - 1) / kBlkChunk * kBlkChunk;
}

template <typename T>
struct BlockSmem {
  // the first kBlkChunk pairs again past the end: a chunk's reads never wrap
  alignas(16) XPair<T> x[kBlkXPairs + kBlkChunk];
  alignas(16) T ring[kBlkWarps + 1][2 * kBlkRing];  // [0]: left edge, [w + 1]: warp w's right edge
  alignas(16) T sink[2 * kBlkRing];
  int done[kBlkWarps];                // steps done by each compute warp
  int staged, drained;                // row pairs staged / stored by the feeder
  unsigned *err;                      // the launch's error word, and the limit of the
  unsigned long long limit_ns;        // compute warps' waits (read only when one is long)
  unsigned long long task;
};

__device__ __forceinline__ int smem_count(const int *p) {
  return *reinterpret_cast<const volatile int *>(p);
}

// What lane 0 reads, in every lane of the calling warp: a warp whose lanes decide
// by a word that changes under them must decide by one read of it (lanes need
// not run in step).
__device__ __forceinline__ int warp_count(const int *p) {
  return __shfl_sync(kFull, smem_count(p), 0);
}
__device__ __forceinline__ unsigned long long warp_timer_ns() {
  return __shfl_sync(kFull, global_timer_ns(), 0);
}

// Waits until the counter is at least v (every lane of the calling warp);
// one that has to wait waits for `more` instead, so that a neighbour of nearly
// the same pace is not waited for again at every chunk.  Bounded: past the
// block's limit the launch's error word is raised; a word already up ends the
// wait.
template <typename T>
__device__ __forceinline__ void wait_count(const int *p, int v, int more, const BlockSmem<T> &sm) {
  if (smem_count(p) < v) {
    unsigned long long t0 = 0;
    for (unsigned it = 0; smem_count(p) < more; ++it) {
      __nanosleep(it < 4 ? 64u << it : 1000u);
      if ((it & 63u) == 63u) {
        if (*reinterpret_cast<volatile unsigned *>(sm.err)) break;
        const unsigned long long now = global_timer_ns();
        if (t0 == 0) {
          t0 = now;
        } else if (now - t0 > sm.limit_ns) {
          atomicExch(sm.err, 1u);
          break;
        }
      }
    }
  }
  __threadfence_block();
  __syncwarp();
}

// Row checkpoints (the stripe-mode forward pass): the full cost row
// r = r0 + k*K - 1 (k >= 1, K = 2^shift >= 2) of this swath's columns is
// stored at q + (k - 1) * stride + (c - c0) -- q points at this swath's first
// column.  K is even, so these rows are always the second row of a lane's
// step pair.
template <typename T>
struct CkptOut {
  T *q;
  unsigned long long stride;
  int shift;
};

// One swath for one block.
template <typename T>
struct BlockJob {
  const T *x, *y;
  int m, n, c0, r0;
  const T *edge_in;     // C[r][c0 - 1] by r - r0, or null for the first swath
  T *edge_out;          // C[r][c0 + 1023] by r - r0, or null
  bool open_end;
  bool free_diag0;
  T corner_init;
  unsigned *words;      // move words of this swath (PATH)
  int word_steps;       // steps of the whole swath in the words' layout
  bool top_band = true; // row m - 1 is the matrix's last row
  // a band of a swath's rows: the row below (this block's columns) or null for
  // the boundary, and where the band leaves its last row and its left edge's
  // value there (null: nowhere)
  const T *row_in = nullptr;
  T *row_out = nullptr, *corner_out = nullptr;
};

// The sweep.  All kBlkThreads threads call it with the same job.  PATH
// records moves; BAND: the job may be a band of a swath's rows (rows counted
// from the band's first; an even number of rows below the top band); CKPT
// stores row checkpoints (CkptOut); CAP gives `corner` the cost of
// cell (m - 1, n - 1) in the thread that owns it (and returns true there) --
// the caller passes cap_last for the swath that holds column n - 1.  The
// returned EdgeStat is valid in the feeding warp's lane 0 when the job has an
// edge_out.
template <typename T, bool PATH, bool BAND, bool CKPT, bool CAP, typename Gate>
__device__ __forceinline__ bool sweep_block(const BlockJob<T> &job, BlockSmem<T> &sm, Gate gate,
                                            CkptOut<T> ckpt, bool cap_last, T &corner,
                                            EdgeStat<T> &st) {
  using V2 = typename Pair2<T>::V;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int rows = job.m - job.r0, r0 = job.r0;
  const T init = r0 ? T(0) : Num<T>::big();
  st.emin = st.etop = Num<T>::big();
  if (rows <= 0) return false;
  const int pairs = (rows + 1) / 2, steps = block_steps(rows);
  const int left_cols = job.n - job.c0;
  const int wact = left_cols >= kBlkCols ? kBlkWarps : (left_cols + kBlkWarpCols - 1) / kBlkWarpCols;
  if (threadIdx.x < kBlkWarps) sm.done[threadIdx.x] = 0;
  if (threadIdx.x == kBlkWarps) sm.staged = 0;
  if (threadIdx.x == kBlkWarps + 1) sm.drained = 0;
  if (threadIdx.x == kBlkWarps + 2) {
    sm.err = gate.error();
    sm.limit_ns = 4 * gate.limit();  // past every wait of a feeder
  }
  __syncthreads();

  if (w == kBlkWarps) {
    // ---- the feeder: one row per lane
    const bool has_in = job.edge_in != nullptr, has_out = job.edge_out != nullptr;
    if (!has_in)
      for (int i = lane; i < 2 * kBlkRing; i += 32) sm.ring[0][i] = Num<T>::big();
    T emin = Num<T>::big(), etop = Num<T>::big();
    int staged = 0, drained = has_out ? 0 : pairs;
    int published = 0, top_lane = 0;  // top_lane: the lane that stores the top row
    const int *last_done = &sm.done[wact - 1];
    unsigned long long t0 = 0;
    for (unsigned idle = 0; staged < pairs || drained < pairs;) {
      const int ld = warp_count(last_done), d0 = warp_count(&sm.done[0]);
      __threadfence_block();
      __syncwarp();
      bool moved = false;
      if (drained < pairs) {
        // whole chunks of the right edge, up to kBlkStage pairs
        int avail = ld - 31 < pairs ? ld - 31 : pairs;
        if (avail - drained > kBlkStage) avail = drained + kBlkStage;
        if (avail > drained && (avail - drained >= kBlkChunk || avail == pairs)) {
          const int row = 2 * drained + lane;
          if (row < 2 * avail && row < rows) {
            const T v = sm.ring[wact][row & (2 * kBlkRing - 1)];
            __stcg(job.edge_out + row, v);
            if (shortcut_row<T>(r0 + row)) emin = Num<T>::min2(emin, v);
            if (row == rows - 1 && job.top_band) etop = v;
          }
          top_lane = (rows - 1 - 2 * drained) & 31;  // (the last time through)
          __syncwarp();
          drained = avail;
          if (lane == 0) *reinterpret_cast<volatile int *>(&sm.drained) = drained;
          if (Gate::kActive) {
            published = 2 * drained < rows ? 2 * drained : rows;
            if (lane == 0) gate.publish(published);
          }
          moved = true;
        }
      }
      if (staged < pairs) {
        // room in the sample ring (the last warp's lane 31 reads the oldest
        // pair) and in the left-edge ring, and the left edge published
        const int k1 = staged + kBlkStage < pairs ? staged + kBlkStage : pairs;
        bool ok = k1 + 31 - ld <= kBlkXPairs && k1 - d0 <= kBlkRing;
        if (ok && has_in && Gate::kActive) {
          int have = 0;
          if (lane == 0) have = gate.ready(2 * k1 < rows ? 2 * k1 : rows) ? 1 : 0;
          ok = __shfl_sync(kFull, have, 0) != 0;
        }
        if (ok) {
          __threadfence_block();
          __syncwarp();  // lane 0 has acquired the rows for all
          // (past pair k1 the slots still hold older pairs)
          const int k = staged + (lane >> 1);
          if (k < k1) {
            const int row = 2 * staged + lane < rows ? 2 * staged + lane : rows - 1;
            const T xv = job.x[r0 + row];
            T ev = T(0);
            if (has_in) ev = __ldcg(job.edge_in + row);
            const int slot = k & (kBlkXPairs - 1);
            XPair<T>::put(&sm.x[slot], lane, xv);
            if (slot < kBlkChunk) XPair<T>::put(&sm.x[slot + kBlkXPairs], lane, xv);
            if (has_in) {
              sm.ring[0][(2 * staged + lane) & (2 * kBlkRing - 1)] = ev;
              if (BAND && job.corner_out && 2 * staged + lane == rows - 1) *job.corner_out = ev;
            }
          }
          __threadfence_block();
          __syncwarp();
          staged = k1;
          if (lane == 0) *reinterpret_cast<volatile int *>(&sm.staged) = staged;
          moved = true;
        }
      }
      if (moved) {
        idle = 0;
        t0 = 0;
      } else {
        __nanosleep(idle < 4 ? 128u << idle : 2000u);
        if ((++idle & 15u) == 0) {
          // bounded, before the compute warps' waits are
          const unsigned long long now = warp_timer_ns();
          if (t0 == 0) {
            t0 = now;
          } else if (now - t0 > gate.limit()) {
            if (lane == 0) gate.fail();
            staged = drained = pairs;
            if (lane == 0) {
              *reinterpret_cast<volatile int *>(&sm.staged) = staged;
              *reinterpret_cast<volatile int *>(&sm.drained) = drained;
            }
          }
        }
      }
    }
    if (Gate::kActive && has_out && published < rows && lane == 0) gate.publish(rows);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      emin = Num<T>::min2(emin, __shfl_xor_sync(kFull, emin, off));
    etop = __shfl_sync(kFull, etop, top_lane);  // (no minimum: it may be NaN or infinite)
    st.emin = emin;
    st.etop = etop;
    return false;
  }
  if (w >= wact) return false;

  // ---- the compute warps
  T col[kBlkR];
  YCols<T, kBlkR> yv;
  const int c_lane = job.c0 + w * kBlkWarpCols + lane * kBlkR;
  yv.load(job.y, c_lane, job.n);
#pragma unroll
  for (int j = 0; j < kBlkR; ++j) col[j] = init;
  T a_last = init, dg = init, cap = T(0);
  T dinit = (w == 0 && lane == 0) ? job.corner_init : init;
  const bool band_in = BAND && job.row_in != nullptr;
  if (band_in && !(w == 0 && lane == 0)) dinit = job.row_in[c_lane - 1 - job.c0];
  const bool lane0 = lane == 0, lane31 = lane == 31;
  const bool fd0 = job.free_diag0 && w == 0 && lane0;
  const int last_pair = (rows - 1) >> 1;        // the pair that holds row m - 1
  const bool last_is_b = ((rows - 1) & 1) != 0;
  const bool oe_top = job.open_end && job.m >= 2 && job.top_band;
  const int cap_c = job.n - 1 - c_lane;         // 0 .. 7 in the lane that owns column n - 1
  const int capj = (CAP && cap_last) ? cap_c : -1;
  // the step at which the lane that owns column n - 1 is on the last row
  const int cap_step = (CAP && cap_last) ? last_pair + (((job.n - 1 - job.c0) / kBlkR) & 31) : -1;
  unsigned *wp = PATH ? job.words + (size_t)w * job.word_steps * 32 + lane : nullptr;
  const bool has_next = w + 1 < wact || job.edge_out != nullptr;  // somebody reads the edge ring
  const int *from = w ? &sm.done[w - 1] : &sm.staged;
  const int *to = w + 1 < wact ? &sm.done[w + 1] : &sm.drained;

  // steps t0 .. t0 + kBlkChunk - 1
  auto chunk = [&](auto fill_c, auto slow_c, int t0) {
    constexpr bool FILL = decltype(fill_c)::value, SLOW = decltype(slow_c)::value;
    const XPair<T> *xs = sm.x + ((t0 - lane) & (kBlkXPairs - 1));
    const V2 *es = reinterpret_cast<const V2 *>(sm.ring[w]) + (t0 & (kBlkRing - 1));
    // lane 31's last column; the other lanes store to a ring nobody reads, so
    // that no lane branches
    V2 *os = reinterpret_cast<V2 *>(lane31 ? sm.ring[w + 1] : sm.sink);
#pragma unroll SLOW ? 1 : 4
    for (int s = 0; s < kBlkChunk; ++s) {
      const XPair<T> xv = xs[s];
      const V2 ev = es[s];
      T la = __shfl_up_sync(kFull, a_last, 1);
      T lb = __shfl_up_sync(kFull, col[kBlkR - 1], 1);
      la = lane0 ? ev.x : la;
      lb = lane0 ? ev.y : lb;
      T diag = dg;
      dg = lb;
      const int k = t0 + s - lane;
      if (FILL && k == 0) {
        diag = dinit;
#pragma unroll
        for (int j = 0; j < kBlkR; ++j) col[j] = init;
        if (band_in) {
#pragma unroll
          for (int j = 0; j < kBlkR; ++j) col[j] = job.row_in[c_lane - job.c0 + j];
        }
      }
      unsigned word[4] = {0u, 0u, 0u, 0u};
      const bool top = SLOW && oe_top && k == last_pair;
      a_last = step_row_pair<T, kBlkR, PATH, SLOW, SLOW && CAP>(
          col, yv, xv, la, lb, diag, top && !last_is_b, top && last_is_b, fd0, word,
          SLOW && CAP && k == last_pair && !last_is_b);
      if (SLOW && CAP && t0 + s == cap_step) {  // (the last row in every lane's col)
#pragma unroll
        for (int j = 0; j < kBlkR; ++j) cap = capj == j ? col[j] : cap;
      }
      V2 v;
      v.x = a_last;
      v.y = col[kBlkR - 1];
      os[(t0 + s - 31) & (kBlkRing - 1)] = v;
      // (a band's idle lanes would hit its neighbours' slots)
      if (PATH && (!BAND || (k >= 0 && k <= last_pair))) wp[(size_t)(t0 + s) * 32] = word[0];
      if (BAND && k == last_pair && job.row_out) {
#pragma unroll
        for (int j = 0; j < kBlkR; ++j) job.row_out[c_lane - job.c0 + j] = col[j];
      }
      if (CKPT) {
        const int kk = 2 * k + 2;
        if (k >= 0 && kk <= rows && (kk & ((1 << ckpt.shift) - 1)) == 0) {
          T *dst = ckpt.q + (unsigned long long)((kk >> ckpt.shift) - 1) * ckpt.stride +
                   (c_lane - job.c0);
#pragma unroll
          for (int j = 0; j < kBlkR; ++j) dst[j] = col[j];
        }
      }
    }
  };
  // the steps at which some lane is on row m - 1 are slow where that row has
  // rules of its own (open end) or its value is wanted
  const bool slow_end = oe_top || (CAP && cap_last);
  // a chunk with its waits before and its count after
  auto turn = [&](auto fill_c, auto slow_c, int t0) {
    // this chunk's left-edge pairs, and room in the right-edge ring
    int need = t0 + kBlkChunk;
    need = need < pairs ? need : pairs;
    if (w) need = need + 31 < steps ? need + 31 : steps;
    const int most = w ? steps : pairs;
    wait_count(from, need, need + kBlkSlack < most ? need + kBlkSlack : most, sm);
    if (has_next) {
      const int room = t0 + kBlkChunk - 31 - kBlkRing;
      if (room > 0) {
        // (the right neighbour can go on to step t0 - 39 whatever this warp does)
        const int v = room < pairs ? room : pairs, more = room + 4 * kBlkChunk;
        wait_count(to, v, more < pairs ? more : pairs, sm);
      }
    }
    chunk(fill_c, slow_c, t0);
    __syncwarp();
    if (lane31) {
      __threadfence_block();
      *reinterpret_cast<volatile int *>(&sm.done[w]) = t0 + kBlkChunk;
    }
  };
  // Each form of the chunk in a loop of its own: beside one another in one loop
  // they spoil each other's schedule (double, a round of 100 members of 1000-4000,
  // open end: 1.41 ms in one loop, 1.32 so).
  const int slow_from = !slow_end ? steps : last_pair >= kBlkChunk ? last_pair + 1 - kBlkChunk : 0;
  int t0 = 0;
#pragma unroll 1
  for (; t0 < 32 && t0 < slow_from; t0 += kBlkChunk) turn(std::true_type{}, std::false_type{}, t0);
#pragma unroll 1
  for (; t0 < slow_from; t0 += kBlkChunk) turn(std::false_type{}, std::false_type{}, t0);
#pragma unroll 1
  for (; t0 < steps; t0 += kBlkChunk) turn(std::true_type{}, std::true_type{}, t0);
  corner = cap;
  return CAP && cap_last && capj >= 0 && capj < kBlkR;
}

}  // namespace odba
