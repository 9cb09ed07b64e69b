// Device-side DTW engine for sm_100a: what the sweeps of a cost matrix share.
//
// Matrix convention (the reference's, dtw.hpp:35-42): rows r in [0, m) walk
// the FIRST series x (the Y axis), columns c in [0, n) walk the SECOND series y
// (the X axis).  Cell rule (dtw.hpp:158-239), with d = x[r] - y[c]:
//     C[r][c] = fma(d, d, min(C[r-1][c], C[r][c-1], C[r-1][c-1]))
// The reference's nvcc build fuses "cost + diff*diff" into one fma on sm_100a;
// that choice is pinned against the reference's own GPU outputs.
//
// A warp sweeps a vertical swath with an anti-diagonal wavefront: lane l owns
// the R consecutive columns c0 + l*R + j (j < R), holding y[c] and the running
// column costs in registers.  At step t lane l works on row pair t - l (rows
// r0 + 2(t - l) and the next, two interleaved dependency chains), so it needs
// from lane l-1 the costs of the same two rows one column to the left, produced
// one step earlier: shuffles carry them.  The rows' samples come from shared
// memory.  The swath's left edge is the previous swath's right-edge column.
// Swaths of 1024 columns are the reference's, so its swath-dependent open-end
// rule (a free diagonal at columns c % 1024 == 0, dtw.hpp:172-186) lands on
// lane 0 / register 0.  One warp per swath: dtw_warp.cuh; a block per swath:
// dtw_block.cuh.
#pragma once

#include <cfloat>
#include <cstdint>

namespace odba {

constexpr int kRefSwath = 1024;  // blockDim.x of every reference DTWDistance launch
constexpr unsigned kFull = 0xffffffffu;

// The reference's open-end shortcut (dtw.hpp:74-129) compares the swath's
// left-edge value on the last row with a minimum that warp 0 reduces and all
// 32 of its lanes store to one shared word (dtw.hpp:97-105); lane l's partial
// minimum covers the rows r with r % 1024 >= 32*l.  On the B200 the float
// build's check reads lane 0's store (all rows), the double build's lane 16's
// (rows with r % 1024 >= 512), as its own open-end and stripe-mode runs show.
template <typename T>
struct ShortcutRows;
template <>
struct ShortcutRows<float> {
  static constexpr int floor = 0;
};
template <>
struct ShortcutRows<double> {
  static constexpr int floor = 512;
};
template <typename T>
__host__ __device__ inline bool shortcut_row(int r) {
  return (r & (kRefSwath - 1)) >= ShortcutRows<T>::floor;
}

template <typename T>
struct Num;
template <>
struct Num<float> {
  // "max" sentinel of the reference (limits.hpp:40-43) for absent predecessors
  static __device__ __forceinline__ float big() { return FLT_MAX; }
  static __device__ __forceinline__ float quiet_nan() { return __int_as_float(0x7fc00000); }
  static __device__ __forceinline__ float cell(float d, float m) { return __fmaf_rn(d, d, m); }
  static __device__ __forceinline__ float min2(float a, float b) { return fminf(a, b); }
  static __device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
  }
};
// Costs of finite samples are never NaN and never -0 (they start at +0 or d*d and
// only grow), so a compare-and-select minimum gives the same bits as fmin
// without fmin's NaN handling, which costs several extra instructions per call
// in double.  With a NaN cost the order of the arguments decides (b wins only if
// it compares less).
template <>
struct Num<double> {
  static __device__ __forceinline__ double big() { return DBL_MAX; }
  static __device__ __forceinline__ double quiet_nan() {
    return __longlong_as_double(0x7ff8000000000000ll);
  }
  static __device__ __forceinline__ double cell(double d, double m) { return __fma_rn(d, d, m); }
  static __device__ __forceinline__ double min2(double a, double b) { return b < a ? b : a; }
  static __device__ __forceinline__ double min3(double a, double b, double c) {
    return min2(min2(a, b), c);
  }
};

// The right-edge column's open-end shortcut figures: the minimum over the rows
// ShortcutRows selects and the value on the last row.
template <typename T>
struct EdgeStat {
  T emin, etop;
};

// A lane's column values y[c] of the swath, and the differences x - y[c] of
// a step's two rows.  For float the values are kept as packed pairs of
// adjacent columns, and one sub.rn.f32x2 gives the differences of two
// columns (each half rounds as sub.rn.f32, so the bits are those of x - y).
// The differences of a row must be asked for in increasing column order, in
// fully unrolled code (the column index is then a constant).
template <typename T, int R>
struct YCols {
  T v[R];
  __device__ __forceinline__ void load(const T *y, int c, int n) {
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = (c + j < n) ? y[c + j] : T(0);
  }
  __device__ __forceinline__ T get(int j) const { return v[j]; }
};
__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
template <int H>
__device__ __forceinline__ float half_f32x2(unsigned long long p) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
  return H ? hi : lo;
}
__device__ __forceinline__ unsigned long long sub_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
template <int R>
struct YCols<float, R> {
  static_assert(R % 2 == 0, "columns come in pairs");
  unsigned long long p[R / 2];
  __device__ __forceinline__ void load(const float *y, int c, int n) {
#pragma unroll
    for (int i = 0; i < R / 2; ++i) {
      const int j = c + 2 * i;
      p[i] = pack_f32x2(j < n ? y[j] : 0.f, j + 1 < n ? y[j + 1] : 0.f);
    }
  }
  __device__ __forceinline__ float get(int j) const {
    return (j & 1) ? half_f32x2<1>(p[j / 2]) : half_f32x2<0>(p[j / 2]);
  }
};

// The samples of a row pair as they are staged in shared memory: float twice
// each, so that a step reads the two operand pairs of its packed differences.
template <typename T>
struct XPair;
template <>
struct XPair<float> {
  float4 v;
  static __device__ __forceinline__ void put(XPair *p, int row, float x) {
    reinterpret_cast<float2 *>(p)[row & 1] = make_float2(x, x);
  }
};
template <>
struct XPair<double> {
  double2 v;
  static __device__ __forceinline__ void put(XPair *p, int row, double x) {
    reinterpret_cast<double *>(p)[row & 1] = x;
  }
};

// The differences of a step's two rows (a, b) from every column.
template <typename T, int R>
struct RowDiffs {
  T xa, xb;
  __device__ __forceinline__ explicit RowDiffs(const XPair<T> &x) : xa(x.v.x), xb(x.v.y) {}
  __device__ __forceinline__ T a(const YCols<T, R> &y, int j) const { return xa - y.get(j); }
  __device__ __forceinline__ T b(const YCols<T, R> &y, int j) const { return xb - y.get(j); }
};
template <int R>
struct RowDiffs<float, R> {
  unsigned long long xa2, xb2, pa = 0, pb = 0;  // pa, pb: the row's current column pair
  __device__ __forceinline__ explicit RowDiffs(const XPair<float> &x)
      : xa2(pack_f32x2(x.v.x, x.v.y)), xb2(pack_f32x2(x.v.z, x.v.w)) {}
  __device__ __forceinline__ float a(const YCols<float, R> &y, int j) {
    if ((j & 1) == 0) pa = sub_f32x2(xa2, y.p[j / 2]);
    return (j & 1) ? half_f32x2<1>(pa) : half_f32x2<0>(pa);
  }
  __device__ __forceinline__ float b(const YCols<float, R> &y, int j) {
    if ((j & 1) == 0) pb = sub_f32x2(xb2, y.p[j / 2]);
    return (j & 1) ? half_f32x2<1>(pb) : half_f32x2<0>(pb);
  }
};

// One cell: the open-end top-row rule when TOP (the right move is free,
// dtw.hpp:196-200; at a reference swath-left column the diagonal is free too,
// dtw.hpp:179-185), the White-Neely cost otherwise.
template <typename T>
__device__ __forceinline__ T cell_rule(T d, T up, T diag, T left, bool top, bool fd) {
  const T v = Num<T>::cell(d, Num<T>::min3(up, diag, left));
  const T vt = fd ? Num<T>::min3(Num<T>::cell(d, up), diag, left)
                  : Num<T>::min2(Num<T>::cell(d, Num<T>::min2(up, diag)), left);
  return top ? vt : v;
}

template <typename T>
struct Pair2;
template <>
struct Pair2<float> {
  using V = float2;
};
template <>
struct Pair2<double> {
  using V = double2;
};

// Hand-off of swath-edge rows.  NoGate: the edge buffer is complete or the
// sweep's own, no other block to wait for (PipeGate in dtw_pipe.cuh is the
// other).  The block's warps still wait for one another, and such a wait that
// runs out raises the launch's error word as any other.
constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // 2 s
struct NoGate {
  static constexpr bool kActive = false;
  unsigned *err;
  unsigned long long limit_ns;
  __device__ __forceinline__ explicit NoGate(unsigned *e, unsigned long long limit = kWaitLimitNs)
      : err(e), limit_ns(limit) {}
  __device__ __forceinline__ void publish(int) {}
  __device__ __forceinline__ bool ready(int) { return true; }
  __device__ __forceinline__ void fail() { atomicExch(err, 1u); }
  __device__ __forceinline__ unsigned *error() { return err; }
  __device__ __forceinline__ unsigned long long limit() { return limit_ns; }
};

}  // namespace odba
