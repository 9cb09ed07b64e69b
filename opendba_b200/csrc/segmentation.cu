// Adaptive k-segmentation (adaptive_device_segmentation, segmentation.hpp:48-337).
//
// One CTA per block of 256*dw raw samples (dw = ceil(minseg/3)):
// down-average by dw, 8-bit quantise against the block's range, then the
// Bellman k-segment DP on integer squared errors, with a binary search on k
// for the largest k whose segments are all at least minseg/dw long, and the
// segment medians of the raw samples.
//
// Differences in structure, not in results:
//  * DP row p depends only on row p-1, so all n of a row are computed at once
//    (one thread per n, each scanning its <= e candidates in increasing order,
//    first strict minimum wins) -- the reference runs every n through thread 0
//    with two barriers per n.
//  * The sum / square tables are prefix sums (the reference's 16-bit sums never
//    wrap for <= 256 samples of at most 255), and the whole backtrack table
//    stays in shared memory instead of a global working buffer.
//  * The DP extent e is computed from the reference's shared-memory layout and
//    the device's opt-in shared memory per block (segmentation.hpp:162, 458-461).
// Kept as the reference computes them: the down-averaging loop bound (which
// averages zero samples -- NaN -- for the upper part of a block), the
// FLT_MIN/partial-warp rules of the min/max reduction, the block minimum that
// only thread 0 sees, the 8-bit conversion (seg_byte), the wrapping int product
// in DIST, and the even-span median pick (segmentation.hpp:327-332).  Where the
// reference races (a 2-sample segment's median reads the first sample of the
// next segment while that one is being sorted) the sorted value is used.
#include <cuda_runtime.h>

#include <cfloat>
#include <climits>
#include <cstdint>

#include "dtw_device.cuh"
#include "odba_internal.h"

namespace odba {

namespace {

template <typename T>
struct SegLim;
template <>
struct SegLim<float> {
  static __device__ __forceinline__ float lo() { return FLT_MIN; }
  static __device__ __forceinline__ float hi() { return FLT_MAX; }
};
template <>
struct SegLim<double> {
  static __device__ __forceinline__ double lo() { return DBL_MIN; }
  static __device__ __forceinline__ double hi() { return DBL_MAX; }
};

// warpReduceMin / warpReduceMax of cuda_utils.hpp:20-40
template <typename T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const T o = __shfl_down_sync(kFull, v, off);
    if (o < v) v = o;
  }
  return v;
}
template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const T o = __shfl_down_sync(kFull, v, off);
    if (o > v) v = o;
  }
  return v;
}

// The conversion to 8 bits as the device compiles the reference's cast
// (segmentation.hpp:168): truncated to an unsigned 32-bit value, which saturates
// (negative and NaN give a low byte of 0), and of that the low byte.  Points past
// the last whole group of 32 are not part of the block's range and can lie
// outside it: 256 gives 0, 300 gives 44.
__device__ __forceinline__ unsigned char seg_byte(double v) {
  return (unsigned char)(__double2uint_rz(v) & 255u);
}

struct SegParams {
  int spb, k_max, minseg, dw, smem_optin;
  int fast;  // the shared memory holds the fast form's rows
  int smem;  // bytes of dynamic shared memory
};

// DP extent from the reference's dynamic shared-memory layout.
template <typename T>
__device__ __forceinline__ int dp_extent(int k_max, int N_ds, int smem) {
  if (N_ds <= 0) return 1;
  const long off_opt = ((long)(k_max + 1) * 2 + 3) / 4 * 4;
  const long off_ksd = off_opt + (long)(N_ds + 1) * 4;
  const long off_ds = (off_ksd + 2L * (N_ds + 1) * 4 + (long)sizeof(T) - 1) / (long)sizeof(T) * (long)sizeof(T);
  const long off_sq = (off_ds + (long)(N_ds + 2) * (long)sizeof(T) + 3) / 4 * 4;
  return int((smem - off_sq) / ((long)N_ds * 6));
}

// ---- the DP of one block --------------------------------------------------------
// Row p of the DP holds, for every prefix of n points, the least cost of p
// segments; it depends on row p - 1 only, never on the k being tried, so the
// binary search on k keeps the rows it has and adds the missing ones (the
// rows of one block: at most the largest k tried instead of the sum of all).
//
// Fast form (kSegThreads threads): four threads share a prefix length n and
// thread g of them holds the costs of the last segments of 4i + g + 1 points
// ending at n in registers, one 32-bit word each, cost << 8 | (n - length).  A
// candidate is then one shared-memory read of row p - 1 and one fused
// add-and-minimum: the word's low byte carries the first point of the last
// segment, so the least word is the least cost and, among equal costs, the
// smallest index -- the reference's first strict minimum.  What bounds it is
// the shared-memory read per candidate.  One thread per prefix, an integer
// division per candidate, all rows again for every k tried and one thread
// per segment sorting it took 46.0 ms for 2.3 M float samples with a minimum
// segment of 4 (one B200); this form with the rank sort takes 2.73 ms.
// Conditions (else the general form): no product of the reference's int
// arithmetic wraps (the block's sum is at most 46340), every cost fits the
// word (sum of squares below 2^23 - 1), the extent e covers half the block
// (then every row has a candidate inside it and the reference's out-of-extent
// sentinel never wins), and no segment is longer than kSegLens points.
constexpr int kSegThreads = 1024;
constexpr int kSegGroups = 4;                         // threads per prefix length
constexpr int kSegRegs = 49;                          // segment costs per thread
constexpr int kSegLens = kSegGroups * kSegRegs;       // 196
constexpr int kSegChunk = 7;                          // costs per skip test
constexpr unsigned kSegBadRow = 0x7fffff00u;          // no such prefix in row p - 1
constexpr unsigned kSegBadCost = 0x80000000u;         // no such segment
constexpr int kSegRowWords = kSegLens + 257;          // one padded DP row

__device__ __forceinline__ int seg_cost_div(unsigned sm, int len) {
  return int(unsigned(sm * sm)) / len;
}

// Rows from + 1 .. to of the DP, fast form.  rows: two padded rows (row r at
// rows + (r & 1) * kSegRowWords + kSegLens + n).
template <int REGS>
__device__ __forceinline__ void seg_rows_fast(const unsigned (&cost)[kSegRegs], unsigned *rows,
                                              unsigned short *kpath, int W, int N_ds, int from,
                                              int to) {
  static_assert(REGS <= kSegRegs, "costs held per thread");
  const int t = threadIdx.x, n = t / kSegGroups + 1, g = t % kSegGroups;
  const int nmax = (t | 31) / kSegGroups + 1;  // the warp's longest prefix
  const unsigned live = __ballot_sync(kFull, n <= N_ds);  // whole groups of kSegGroups lanes
  for (int p = from + 1; p <= to; ++p) {
    const unsigned *prev = rows + ((p - 1) & 1) * kSegRowWords + kSegLens;
    unsigned *cur = rows + (p & 1) * kSegRowWords + kSegLens;
    if (n <= N_ds) {
      unsigned best = 0xffffffffu;
      const unsigned *q = prev + (n - 1 - g);
#pragma unroll
      for (int c = 0; c < REGS; c += kSegChunk) {
        // segments of more than n - p + 1 points start before row p - 1's
        // first prefix
        if (c * kSegGroups + 1 <= nmax - p + 1) {
#pragma unroll
          for (int i = c; i < c + kSegChunk && i < REGS; ++i)
            best = __viaddmin_u32(q[-i * kSegGroups], cost[i], best);
        }
      }
#pragma unroll
      for (int off = 1; off < kSegGroups; off <<= 1) {
        const unsigned o = __shfl_xor_sync(live, best, off);
        best = o < best ? o : best;
      }
      if (g == 0) {
        cur[n] = n >= p ? (best & ~255u) : kSegBadRow;
        if (n >= p) kpath[(p - 1) * W + (n - 1)] = (unsigned short)(best & 255u);
      }
    }
    __syncthreads();
  }
}

// The general form (any block): one thread per prefix, two rows ksd0 / ksd1.
__device__ __forceinline__ void seg_rows_general(const unsigned *P, const unsigned *Q,
                                                 unsigned *ksd0, unsigned *ksd1,
                                                 unsigned short *kpath, int W, int N_ds, int e,
                                                 int from, int to) {
  for (int p = from + 1; p <= to; ++p) {
    const unsigned *prev = (p & 1) ? ksd0 : ksd1;
    unsigned *cur = (p & 1) ? ksd1 : ksd0;
    for (int n = p + int(threadIdx.x); n <= N_ds; n += blockDim.x) {
      const int lo = (n - e + 1 > p) ? n - e + 1 : p;
      int minval = INT_MAX, minidx = -1;
      const unsigned Pn = P[n], Qn = Q[n];
      for (int idx = lo; idx <= n; ++idx) {
        const unsigned sm = Pn - P[idx - 1];
        const unsigned sq = Qn - Q[idx - 1];
        const unsigned opt = prev[idx - 1] + (sq - unsigned(seg_cost_div(sm, n - idx + 1)));
        if (opt < unsigned(minval)) {
          minval = int(opt);
          minidx = idx;
        }
      }
      cur[n] = unsigned(minval);
      kpath[(p - 1) * W + (n - 1)] = (unsigned short)((unsigned short)minidx - 1);
    }
    __syncthreads();
  }
}

// A total order of the raw samples exists and sorting them by rank gives what
// the exchange sort gives: no NaN, and no negative zero (equal to zero, told
// apart by its bits only).
__device__ __forceinline__ bool seg_plain_value(float v) {
  return v == v && __float_as_uint(v) != 0x80000000u;
}
__device__ __forceinline__ bool seg_plain_value(double v) {
  return v == v && (unsigned long long)__double_as_longlong(v) != 0x8000000000000000ull;
}

// The segment bounds of a block whose medians the exchange sort has to give
// (segment_sort_kernel), left in the place of its medians: NaNs whose payload no
// arithmetic gives, with the bound in the low 16 bits.
template <typename T>
struct SegPending;
template <>
struct SegPending<float> {
  static constexpr unsigned kTag = 0x7fdb0000u;
  static __device__ __forceinline__ float put(unsigned short b) { return __uint_as_float(kTag | b); }
  static __device__ __forceinline__ bool is(float v) {
    return (__float_as_uint(v) & 0xffff0000u) == kTag;
  }
  static __device__ __forceinline__ unsigned short get(float v) {
    return (unsigned short)__float_as_uint(v);
  }
};
template <>
struct SegPending<double> {
  static constexpr unsigned long long kTag = 0x7ffdba0000000000ull;
  static __device__ __forceinline__ double put(unsigned short b) {
    return __longlong_as_double((long long)(kTag | b));
  }
  static __device__ __forceinline__ bool is(double v) {
    return ((unsigned long long)__double_as_longlong(v) & ~0xffffull) == kTag;
  }
  static __device__ __forceinline__ unsigned short get(double v) {
    return (unsigned short)__double_as_longlong(v);
  }
};

// The median of samples lb .. rb-1 of a block sorted within its segments
// (segmentation.hpp:327-332).
template <typename T>
__device__ __forceinline__ T seg_median(const T *sorted, int lb, int rb) {
  const int mid = (lb + rb) / 2;
  return ((lb - rb) % 2) ? sorted[mid] : (sorted[mid] + sorted[mid + 1]) / 2;
}

template <typename T>
__global__ void __launch_bounds__(kSegThreads) segment_kernel(const T *series,
                                                              const uint64_t *offsets,
                                                              const uint64_t *lens,
                                                              const unsigned long long *seg_base,
                                                              SegParams sp, T *medians) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int s = blockIdx.x, by = blockIdx.y;
  const long orig_N = long(lens[s]);
  const int spb = sp.spb, dw = sp.dw, k_max = sp.k_max;
  if ((long)by * spb >= orig_N) return;
  const T *x = series + offsets[s] + (long)by * spb;
  T *out = medians + seg_base[s] + (unsigned long long)by * k_max;

  const bool partial = (long)(by + 1) * spb > orig_N;
  const int N = partial ? int(orig_N % spb) : spb;
  int expected_k = k_max;
  if (partial) {
    const int per = (spb + k_max - 1) / k_max;
    expected_k = (int(orig_N % spb) + per - 1) / per;
  }
  const int N_ds = N / dw;
  const int e = dp_extent<T>(k_max, N_ds, sp.smem_optin);

  // shared memory carve-up (segment_smem_bytes)
  const int W = N_ds + 2;
  T *od = reinterpret_cast<T *>(smem_raw);                                // spb raw samples + 2
  unsigned *P = reinterpret_cast<unsigned *>(od + spb + 2);                // 257 prefix sums
  unsigned *Q = P + 257;                                                   // 257 prefix squares
  unsigned *ksd0 = Q + 257;                                                // two DP rows
  unsigned *ksd1 = ksd0 + W;
  unsigned *rows = ksd0;  // the fast form's two padded rows
  unsigned char *after = reinterpret_cast<unsigned char *>(
      ksd0 + (sp.fast ? 2 * kSegRowWords : 2 * W));
  unsigned short *bp = reinterpret_cast<unsigned short *>(after);          // k_max + 2
  unsigned short *kpath = bp + (k_max + 2);                                // (k_max + 1) * W
  __shared__ T wmaxs[8], wmins[8];
  __shared__ T gstat[2];
  __shared__ unsigned char q[256];
  __shared__ unsigned wp[8], wq[8];
  __shared__ int ctrl[4];

  // 1. down-average, with the reference's loop bound (segmentation.hpp:111-120)
  T dsv = T(0);
  if (t < 256) {
    if (t * dw <= N - dw) {
      T acc = T(0);
      int num = 0;
      for (int i = 0; i < dw && dw * t + t + i < N; i++) {
        acc = acc + x[dw * t + i];
        num++;
      }
      dsv = acc / T(num);
    }
  }
  // 2. block range (segmentation.hpp:124-150)
  const int nw = N_ds / 32;
  if (t < 256) {
    T vmax = t < N_ds ? dsv : SegLim<T>::lo();
    T vmin = t < N_ds ? dsv : SegLim<T>::hi();
    vmin = warp_min(vmin);
    vmax = warp_max(vmax);
    if (lane == 0 && wid < nw) {
      wmaxs[wid] = vmax;
      wmins[wid] = vmin;
    }
  }
  __syncthreads();
  if (wid == 0) {
    T a = lane < nw ? wmaxs[lane] : SegLim<T>::lo();
    a = warp_max(a);
    T b = lane < nw ? wmins[lane] : SegLim<T>::hi();
    b = warp_min(b);
    if (lane == 0) {
      gstat[0] = a;
      gstat[1] = b;
    }
  }
  __syncthreads();
  const T gmax = gstat[0];
  // thread 0 sees the block minimum; the others read slot nw of the max array
  const T others_min = nw >= 2 ? wmins[0] : (nw == 1 ? gstat[1] : gmax);
  const T mn = t == 0 ? gstat[1] : others_min;
  // 3. quantise (segmentation.hpp:168), and prefix sums of the values and
  // their squares
  unsigned pv = 0, pq = 0;
  if (t < 256) {
    if (t < N_ds) {
      q[t] = seg_byte(256.0 * ((dsv - mn) / (gmax - mn + 1)));
      pv = q[t];
      pq = pv * pv;
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned a = __shfl_up_sync(kFull, pv, off), b = __shfl_up_sync(kFull, pq, off);
      if (lane >= off) {
        pv += a;
        pq += b;
      }
    }
    if (lane == 31) {
      wp[wid] = pv;
      wq[wid] = pq;
    }
  }
  __syncthreads();
  if (t < 256) {
    for (int w = 0; w < wid; ++w) {
      pv += wp[w];
      pq += wq[w];
    }
    if (t < N_ds) {
      P[t + 1] = pv;
      Q[t + 1] = pq;
    }
  }
  if (t == 0) {
    P[0] = 0;
    Q[0] = 0;
    ctrl[0] = (expected_k + 1) / 2;      // test_k
    ctrl[1] = ctrl[0] / 2;               // delta
    ctrl[2] = expected_k + 1;            // smallest noisy k found
    ctrl[3] = 0;                         // exit
  }
  __syncthreads();

  // 4. DP with the binary search on k (segmentation.hpp:190-336)
  const int longest = e < N_ds ? e : N_ds;
  const bool fast = sp.fast && N_ds >= 1 && 2 * e >= N_ds && longest <= kSegLens &&
                    P[N_ds] <= 46340u && Q[N_ds] < (1u << 23) - 1;
  unsigned cost[kSegRegs];
  if (fast) {
    const int n = t / kSegGroups + 1, g = t % kSegGroups;
#pragma unroll
    for (int i = 0; i < kSegRegs; ++i) {
      const int len = i * kSegGroups + g + 1;
      cost[i] = kSegBadCost;
      if (n <= N_ds && len <= n && len <= e) {
        const unsigned sm = P[n] - P[n - len], sq = Q[n] - Q[n - len];
        cost[i] = ((sq - (sm * sm) / unsigned(len)) << 8) | unsigned(n - len);
      }
    }
    for (int i = t; i < 2 * kSegRowWords; i += kSegThreads) rows[i] = kSegBadRow;
    __syncthreads();
    unsigned *row1 = rows + kSegRowWords + kSegLens;
    if (t >= 1 && t <= N_ds && t <= e)
      row1[t] = (Q[t] - (P[t] * P[t]) / unsigned(t)) << 8;
  } else {
    for (int n1 = t + 1; n1 <= N_ds; n1 += blockDim.x)
      ksd1[n1] = n1 <= e ? Q[n1] - unsigned(seg_cost_div(P[n1], n1)) : unsigned(INT_MAX / 2);
  }
  __syncthreads();
  int rows_done = 1;
  while (!ctrl[3]) {
    const int test_k = ctrl[0];
    __syncthreads();  // every thread has read the control words
    if (test_k > rows_done) {
      if (!fast)
        seg_rows_general(P, Q, ksd0, ksd1, kpath, W, N_ds, e, rows_done, test_k);
      else if (longest <= 37 * kSegGroups)
        seg_rows_fast<37>(cost, rows, kpath, W, N_ds, rows_done, test_k);
      else
        seg_rows_fast<kSegRegs>(cost, rows, kpath, W, N_ds, rows_done, test_k);
      rows_done = test_k;
    }
    if (t == 0) {
      bp[test_k] = (unsigned short)N_ds;
      bool noisy = false;
      int right = N_ds;
      const int least = sp.minseg / dw;
      for (int p = test_k - 1; p >= 1; p--) {
        const int col = right - 1;
        const int left = (col >= 0 && col < W) ? kpath[p * W + col] : 0;
        bp[p] = (unsigned short)left;
        noisy |= right - left < least;
        right = left;
      }
      bp[0] = 0;
      noisy |= right < least;
      int delta = ctrl[1];
      int tk = test_k;
      if (delta == 0 || tk + delta > k_max) {
        ctrl[3] = 1;
      } else if (tk != 1 && noisy) {
        ctrl[2] = tk;
        tk -= delta;
      } else {
        if (tk == 1 || ctrl[2] == tk + 1)
          ctrl[3] = 1;
        else
          tk += delta;
      }
      ctrl[1] = (delta + 1) / 2;
      if (!ctrl[3]) ctrl[0] = tk;
    }
    __syncthreads();
  }
  const int test_k = ctrl[0];

  // 5. medians of the raw samples (segmentation.hpp:287-333)
  // samples past the block read as 0 (the reference reads whatever its shared
  // memory holds there, which only an even-span last segment can reach)
  bool plain = true;
  for (int i = t; i < spb + 2; i += blockDim.x) {
    const T v = (i < spb && (long)by * spb + i < orig_N) ? x[i] : T(0);
    od[i] = v;
    plain &= seg_plain_value(v);
  }
  for (int seg = t + 1; seg <= test_k; seg += blockDim.x) plain &= bp[seg - 1] <= bp[seg];
  for (int seg = t + 1; seg <= k_max; seg += blockDim.x)
    if (seg > test_k) out[seg - 1] = SegLim<T>::hi();
  // the move table is dead: its space takes the sorted samples where they fit
  T *sorted = reinterpret_cast<T *>((reinterpret_cast<uintptr_t>(kpath) + 15) & ~uintptr_t(15));
  const bool room = smem_raw + sp.smem >= reinterpret_cast<unsigned char *>(sorted + spb + 2);
  if (!__syncthreads_and(plain) || !room) {
    for (int seg = t + 1; seg <= test_k; seg += blockDim.x) out[seg - 1] = SegPending<T>::put(bp[seg]);
    return;
  }
  // every sample to its rank within its segment (equal samples by index).
  // One thread per segment with an exchange sort is serial in the longest
  // segment, and the reference's down-averaging makes the upper third of
  // each block one such segment (170 of 512 samples with minseg 4).
  for (int i = t; i < spb + 2; i += blockDim.x) {
    int lo = 0, hi = test_k;  // bp[lo] * dw <= i < bp[hi] * dw
    const int last = bp[test_k] * dw < N ? bp[test_k] * dw : N;
    const T v = od[i];
    if (i >= last) {
      sorted[i] = v;
      continue;
    }
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (bp[mid] * dw <= i) lo = mid; else hi = mid;
    }
    const int lb = bp[lo] * dw;
    const int rb = bp[hi] * dw < N ? bp[hi] * dw : N;
    int rank = 0;  // (no NaN: equal samples before this one come first)
    for (int j = lb; j < i; ++j) rank += int(od[j] <= v);
    for (int j = i + 1; j < rb; ++j) rank += int(od[j] < v);
    sorted[lb + rank] = v;
  }
  __syncthreads();
  for (int seg = t + 1; seg <= test_k; seg += blockDim.x) {
    int rb = bp[seg] * dw;
    if (rb > N) rb = N;
    out[seg - 1] = seg_median(sorted, bp[seg - 1] * dw, rb);
  }
}

// The medians of the blocks segment_kernel left bounds for: those with a NaN or
// a negative zero, whose order is the exchange sort's own, and those too long
// for the rank sort's copy.  One thread per segment, as the reference has it; a
// kernel of its own, since the serial sort of a long segment beside the DP's
// 1024 threads keeps a whole SM waiting (1 M samples with negative zeros, minimum
// segment 9: 37 ms in one kernel, 22 in blocks of 256 threads).
constexpr int kSegSortThreads = 256;
template <typename T>
__global__ void __launch_bounds__(kSegSortThreads) segment_sort_kernel(const T *series,
                                                                       const uint64_t *offsets,
                                                                       const uint64_t *lens,
                                                                       const unsigned long long *seg_base,
                                                                       SegParams sp, T *medians) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int t = threadIdx.x, s = blockIdx.x, by = blockIdx.y;
  const long orig_N = long(lens[s]);
  const int spb = sp.spb, dw = sp.dw, k_max = sp.k_max;
  if ((long)by * spb >= orig_N) return;
  T *out = medians + seg_base[s] + (unsigned long long)by * k_max;
  if (!SegPending<T>::is(out[0])) return;
  const T *x = series + offsets[s] + (long)by * spb;
  const int N = (long)(by + 1) * spb > orig_N ? int(orig_N % spb) : spb;
  T *od = reinterpret_cast<T *>(smem_raw);                                // spb samples + 2
  unsigned short *bp = reinterpret_cast<unsigned short *>(od + spb + 2);  // k_max + 1
  __shared__ int segs;
  if (t == 0) {
    segs = 0;
    bp[0] = 0;
  }
  __syncthreads();
  for (int i = t; i < spb + 2; i += blockDim.x)
    od[i] = (i < spb && (long)by * spb + i < orig_N) ? x[i] : T(0);
  for (int seg = t + 1; seg <= k_max; seg += blockDim.x)
    if (SegPending<T>::is(out[seg - 1])) {
      bp[seg] = SegPending<T>::get(out[seg - 1]);
      atomicMax(&segs, seg);
    }
  __syncthreads();
  const int test_k = segs;
  for (int seg = t + 1; seg <= test_k; seg += blockDim.x) {
    int rb = bp[seg] * dw;
    if (rb > N) rb = N;
    const int lb = bp[seg - 1] * dw;
    for (int i = lb; i < rb - 1; ++i)
      for (int j = i + 1; j < rb; ++j)
        if (od[i] > od[j]) {
          const T tmp = od[i];
          od[i] = od[j];
          od[j] = tmp;
        }
  }
  __syncthreads();
  for (int seg = t + 1; seg <= test_k; seg += blockDim.x) {
    int rb = bp[seg] * dw;
    if (rb > N) rb = N;
    const int lb = bp[seg - 1] * dw < N ? bp[seg - 1] * dw : N;
    out[seg - 1] = seg_median(od, lb, rb);
  }
}

// Shared memory of one block; fast: with the fast form's padded rows.
template <typename T>
size_t segment_smem_bytes(int spb, int k_max, bool fast) {
  const int W = 256 + 2;
  return size_t(spb + 2) * sizeof(T) + 2 * 257 * 4 +
         size_t(fast ? 2 * kSegRowWords : 2 * W) * 4 + size_t(k_max + 2) * 2 +
         size_t(k_max + 1) * W * 2 + 64;
}

}  // namespace

void segment_params(int minseg, int *dw, int *spb, int *k_max) {
  *dw = (minseg + 2) / 3;
  *spb = 256 * *dw;
  const float per = float(minseg) / float(*dw);
  *k_max = int((256 + per - 1) / per);
}

template <typename T>
int segment_launch(const T *series, const uint64_t *offsets, const uint64_t *lens,
                   const unsigned long long *seg_base, int n, int max_blocks, int minseg,
                   T *medians, cudaStream_t stream) {
  SegParams sp;
  segment_params(minseg, &sp.dw, &sp.spb, &sp.k_max);
  sp.minseg = minseg;
  int dev = 0;
  cudaGetDevice(&dev);
  sp.smem_optin = 48 * 1024;
  cudaDeviceGetAttribute(&sp.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  // the fast form's padded rows take 1.6 KB more: at the longest minimum
  // segment lengths the general form alone fits
  sp.fast = segment_smem_bytes<T>(sp.spb, sp.k_max, true) <= size_t(sp.smem_optin);
  const size_t smem = segment_smem_bytes<T>(sp.spb, sp.k_max, sp.fast != 0);
  sp.smem = int(smem);
  if (smem > size_t(sp.smem_optin))
    return fail(ODBA_ERR_INVALID_ARGUMENT, "minimum segment length needs more shared memory than the device has");
  cudaFuncSetAttribute(segment_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (n < 1 || max_blocks < 1) return ODBA_OK;
  dim3 grid(n, max_blocks);
  segment_kernel<T><<<grid, kSegThreads, smem, stream>>>(series, offsets, lens, seg_base, sp, medians);
  const size_t sort_smem = size_t(sp.spb + 2) * sizeof(T) + size_t(sp.k_max + 2) * 2;
  cudaFuncSetAttribute(segment_sort_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sort_smem));
  segment_sort_kernel<T><<<grid, kSegSortThreads, sort_smem, stream>>>(series, offsets, lens, seg_base,
                                                                       sp, medians);
  return check_launch("segmentation kernel");
}

__global__ void seg_base_kernel(const uint64_t *lens, int n, int spb, int k_max,
                                unsigned long long *base) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  unsigned long long acc = 0;
  for (int i = 0; i < n; ++i) {
    base[i] = acc;
    acc += (unsigned long long)((lens[i] + spb - 1) / spb) * k_max;
  }
}

template <typename T>
int segment_blocks(const T *series, const uint64_t *offsets, const uint64_t *lens,
                   const uint64_t *h_lens, int n, int minseg, T *medians, void *ws,
                   size_t ws_bytes, cudaStream_t stream) {
  if (n < 1) return ODBA_OK;
  if (ws_bytes < size_t(n) * 8) return fail(ODBA_ERR_WORKSPACE_TOO_SMALL, "segmentation workspace too small");
  int dw, spb, k_max;
  segment_params(minseg, &dw, &spb, &k_max);
  int max_blocks = 0;
  for (int i = 0; i < n; ++i) {
    const long nb = long((h_lens[i] + spb - 1) / spb);
    if (nb > 65535) return fail(ODBA_ERR_INVALID_ARGUMENT, "series too long for one segmentation grid");
    if (nb > max_blocks) max_blocks = int(nb);
  }
  auto *base = static_cast<unsigned long long *>(ws);
  seg_base_kernel<<<1, 32, 0, stream>>>(lens, n, spb, k_max, base);
  return segment_launch<T>(series, offsets, lens, base, n, max_blocks, minseg, medians, stream);
}

template int segment_blocks<float>(const float *, const uint64_t *, const uint64_t *,
                                   const uint64_t *, int, int, float *, void *, size_t,
                                   cudaStream_t);
template int segment_blocks<double>(const double *, const uint64_t *, const uint64_t *,
                                    const uint64_t *, int, int, double *, void *, size_t,
                                    cudaStream_t);

template int segment_launch<float>(const float *, const uint64_t *, const uint64_t *,
                                   const unsigned long long *, int, int, int, float *, cudaStream_t);
template int segment_launch<double>(const double *, const uint64_t *, const uint64_t *,
                                    const unsigned long long *, int, int, int, double *,
                                    cudaStream_t);

}  // namespace odba
