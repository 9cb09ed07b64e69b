// Moves recorded by the path sweep of the DBA round (DBAUpdate's DTWDistance
// launches with a path matrix, dba.hpp:589-617).
//
// Each cell also records the reference's move choice (dtw.hpp:202-227):
//   if (diag > up) move = (up > right) ? RIGHT : UP
//   else           move = (diag > right) ? RIGHT : DIAGONAL
// over the three candidate costs rounded separately (fma(d, d, pred), or the
// free predecessor on the open-end top row).  Ties therefore resolve
// DIAGONAL > UP > RIGHT, i.e. move = DIAGONAL if diag == min, else UP if
// up == min, else RIGHT.  Two bits per cell are kept as two bit planes: D
// (the diagonal candidate equals the minimum) and U (the up candidate does),
// each set by one compare and one predicated OR of an immediate; decode_move
// applies the priority.  The codes the reference derives from position alone
// (row 0, (0, 0), the open-end OPEN_RIGHT) are rebuilt by the backtrack.
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

}  // namespace odba
