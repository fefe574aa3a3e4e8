// k64_dev.cuh -- device helpers of the FP64 drop-in's fused kernels.
#pragma once

#include "swap_dev.cuh"

namespace swapk {

// x / d for a grid spacing d with r = 1/d rounded: exactly the rounded
// quotient.  P2 (every spacing a power of two): r is exact, and x * r is x / d
// with the same single rounding.  Otherwise Markstein's correction (P.
// Markstein, IBM J. Res. Dev. 34, 1990): q = x*r, then q + (x - q*d)*r in
// fused operations is the rounded quotient when r is the rounded reciprocal
// and nothing underflows or overflows; x outside 2^-900..2^900 takes the
// division.  (The host keeps r = 0 for a spacing outside 2^-60..2^60 or with
// an all-ones significand, the exception of the theorem.)
template <bool P2>
__device__ __forceinline__ double quotient(double x, double d, double r) {
  if (P2) return x * r;
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  if (e - 123u > 1800u || r == 0.0) {
    if (((unsigned)__double2hiint(x) << 1 | (unsigned)__double2loint(x)) == 0u && r != 0.0) return x * r;  // +-0
    return x / d;
  }
  const double q = x * r;
  return __fma_rn(__fma_rn(-q, d, x), r, q);
}

// The bits of a double as an integer that orders like it (NaN beyond the
// infinities): a comparison costs a few integer instructions instead of one
// of the FP64 pipe's 16-clock slots.
__device__ __forceinline__ long long ordered(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

// cell_search (swap_dev.cuh) with integer comparisons and an FP32 guess: the
// same index for every x, 0 when x is outside (q(1), q(n)] or not a number.
__device__ __forceinline__ int find_cell(const double* __restrict__ q, int n, double x, float q1, float inv_d) {
  const long long xb = ordered(x);
  int i = (int)((__double2float_rn(x) - q1) * inv_d) + 1;
  i = i < 1 ? 1 : (i > n - 1 ? n - 1 : i);
  while (i > 1 && !(xb > ordered(q[i]))) --i;
  while (i < n - 1 && xb > ordered(q[i + 1])) ++i;
  return xb > ordered(q[i]) && xb <= ordered(q[i + 1]) ? i : 0;
}

}  // namespace swapk
