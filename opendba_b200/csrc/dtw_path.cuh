// The row-pair step of the sweeps, and the moves recorded by the path sweeps of
// the DBA round (DBAUpdate's DTWDistance launches with a path matrix,
// dba.hpp:589-617).
//
// Each cell also records the reference's move choice (dtw.hpp:202-227):
//   if (diag > up) move = (up > right) ? RIGHT : UP
//   else           move = (diag > right) ? RIGHT : DIAGONAL
// over the three candidate costs rounded separately (fma(d, d, pred), or the
// free predecessor on the open-end top row).  Ties therefore resolve
// DIAGONAL > UP > RIGHT, i.e. move = DIAGONAL if diag == min, else UP if
// up == min, else RIGHT.  Two bits per cell are kept as two bit planes: D
// (the diagonal candidate equals the minimum) and U (the up candidate does),
// each set by one compare and one predicated OR of an immediate.  The codes the
// reference derives from position alone (row 0, (0, 0), the open-end
// OPEN_RIGHT) are rebuilt by the backtrack.
#pragma once

#include "dtw_device.cuh"

namespace odba {

// Sets bit J of w if a == b: one compare and one predicated OR of an
// immediate (no select, no shifted constant in a register).
template <int J>
__device__ __forceinline__ void or_bit_if_eq(unsigned &w, float a, float b) {
  asm("{\n\t.reg .pred p;\n\tsetp.eq.f32 p, %1, %2;\n\t@p or.b32 %0, %0, %3;\n\t}"
      : "+r"(w)
      : "f"(a), "f"(b), "n"(1u << J));
}
template <int J>
__device__ __forceinline__ void or_bit_if_eq(unsigned &w, double a, double b) {
  asm("{\n\t.reg .pred p;\n\tsetp.eq.f64 p, %1, %2;\n\t@p or.b32 %0, %0, %3;\n\t}"
      : "+r"(w)
      : "d"(a), "d"(b), "n"(1u << J));
}

// Move codes the sweep records (dtw.hpp:10-16).
constexpr int kMoveDiag = 1, kMoveRight = 2, kMoveUp = 3;

// Where a step's move bits go: BITS-bit planes (D, then U) of row ROW (0: a, 1: b)
// in the step's words -- 8: all four planes in one word (D and U of row a, then of
// row b); 16: a word per row, D in the low half; 32: a word per plane.
template <int BITS, int ROW>
struct MoveSlot {
  static constexpr int wd = BITS == 32 ? 2 * ROW : ROW, wu = BITS == 32 ? 2 * ROW + 1 : ROW;
  static constexpr int bd = BITS == 8 ? 16 * ROW : 0, bu = bd + (BITS == 32 ? 0 : BITS);
};

// One cell; PATH adds its move bits (bit J of its row's planes) to w.
template <typename T, bool PATH, bool TOP, int BITS, int ROW, int J>
__device__ __forceinline__ T row_pair_cell(T d, T up, T diag, T left, bool top, bool fd,
                                           unsigned (&w)[4]) {
  if constexpr (PATH) {
    using S = MoveSlot<BITS, ROW>;
    const T uv = Num<T>::cell(d, up);
    T dv = Num<T>::cell(d, diag);
    T rv = Num<T>::cell(d, left);
    if (TOP) {
      rv = top ? left : rv;
      dv = (top && fd) ? diag : dv;
    }
    const T v = Num<T>::min3(uv, dv, rv);
    or_bit_if_eq<S::bd + J>(w[S::wd], dv, v);
    or_bit_if_eq<S::bu + J>(w[S::wu], uv, v);
    return v;
  } else if constexpr (TOP) {
    return cell_rule<T>(d, up, diag, left, top, fd);
  } else {
    return Num<T>::cell(d, Num<T>::min3(up, diag, left));
  }
}

// Two rows of a lane's R columns, row b one column behind row a: the two
// chains interleave, and since row a at column j reads the old col[j - 1] as its
// diagonal before row b writes the new one, no column changes registers (in
// column order all of them would rotate).  PASS: with `pass` set row b is row a
// again (row a is the matrix's last; its costs are then in col).
template <typename T>
struct RowPairState {
  T a_left, a_diag, b_left, b_diag, va_prev;
  unsigned w[4];
};
template <typename T, int R, bool PATH, bool TOP, bool PASS, int BITS, int J>
struct RowPairCols {
  static __device__ __forceinline__ void run(T (&col)[R], const YCols<T, R> &yv,
                                             RowDiffs<T, R> &df, RowPairState<T> &z, bool top_a,
                                             bool top_b, bool fd0, bool pass) {
    if constexpr (J < R) {
      const T up = col[J];
      const T va = row_pair_cell<T, PATH, TOP, BITS, 0, J>(df.a(yv, J), up, z.a_diag, z.a_left,
                                                           top_a, J == 0 && fd0, z.w);
      z.a_diag = up;
      z.a_left = va;
      if constexpr (J > 0) {
        T vb = row_pair_cell<T, PATH, TOP, BITS, 1, J - 1>(
            df.b(yv, J - 1), z.va_prev, z.b_diag, z.b_left, top_b, J == 1 && fd0, z.w);
        if (PASS) vb = pass ? z.va_prev : vb;
        z.b_diag = z.va_prev;
        z.b_left = vb;
        col[J - 1] = vb;
      }
      z.va_prev = va;
      RowPairCols<T, R, PATH, TOP, PASS, BITS, J + 1>::run(col, yv, df, z, top_a, top_b, fd0, pass);
    }
  }
};
// words: the step's moves (BITS / 8 of them; PATH).
template <typename T, int R, bool PATH, bool TOP, bool PASS, int BITS = 8>
__device__ __forceinline__ T step_row_pair(T (&col)[R], const YCols<T, R> &yv, const XPair<T> &x,
                                           T la, T lb, T dg, bool top_a, bool top_b, bool fd0,
                                           unsigned (&words)[4], bool pass) {
  static_assert(!PATH || R <= BITS, "a bit per column");
  RowPairState<T> z{la, dg, lb, la, T(0), {0u, 0u, 0u, 0u}};
  RowDiffs<T, R> df(x);
  RowPairCols<T, R, PATH, TOP, PASS, BITS, 0>::run(col, yv, df, z, top_a, top_b, fd0, pass);
  col[R - 1] = row_pair_cell<T, PATH, TOP, BITS, 1, R - 1>(
      df.b(yv, R - 1), z.va_prev, z.b_diag, z.b_left, top_b, R == 1 && fd0, z.w);
  if (PASS) col[R - 1] = pass ? z.va_prev : col[R - 1];
  if (PATH) {
    if (BITS == 8) {
      words[0] = z.w[0] | z.w[1];
    } else {
#pragma unroll
      for (int i = 0; i < BITS / 8; ++i) words[i] = z.w[i];
    }
  }
  return z.a_left;
}

}  // namespace odba
