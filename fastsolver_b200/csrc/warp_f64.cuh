// warp_f64.cuh -- warp-level building blocks shared by the FP64 kernels.
#pragma once

namespace hodlr {

// C += A B on the FP64 tensor pipe, one 16 x 8 x 4 block.  Fragments of m16n8k4
// .f64 (g = lane / 4, t = lane % 4): A a0 = A[g][t], a1 = A[g + 8][t]; B b =
// B[t][g]; C c0..c3 = C[g][2t], C[g][2t + 1], C[g + 8][2t], C[g + 8][2t + 1].
__device__ inline void dmma(double (&c)[4], double a0, double a1, double b) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, "
      "{%0, %1, %2, %3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b));
}

// Pivot searches: of the lanes whose `high` is the warp's largest (mx; more than
// one of them), the one with the largest low word, lowest position on ties.
__device__ inline int tied_lane(unsigned high, unsigned mx, unsigned low, int pos) {
  bool top = high == mx;
  const unsigned ml = __reduce_max_sync(0xffffffffu, top ? low : 0u);
  top = top && low == ml;
  const unsigned pm = __reduce_min_sync(0xffffffffu, top ? (unsigned)pos : 0xffffffffu);
  return __ffs(__ballot_sync(0xffffffffu, top && (unsigned)pos == pm)) - 1;
}

}  // namespace hodlr
