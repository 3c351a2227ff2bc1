// recip.cuh -- division by a pivot known long before its dividend: a few dependent
// operations off a stored reciprocal, rounded as the division is.
#pragma once

#include <cuda_runtime.h>

namespace ab2 {
namespace {

// FP64, r = RN(1/p): q0 = RN(x r) is within 2^-52 of x/p, one correction
// q1 = RN(q0 + r RN(x - q0 p)) leaves the rounding of a value within 2^-103 of
// x/p (so q1 is one of the two doubles around it), and then
// q2 = RN(q1 + r (x - q1 p)), whose residual is exact, is x/p correctly rounded
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990, theorem on the quotient
// from a correctly rounded reciprocal and a neighbouring quotient).  That holds
// where nothing over- or underflows: recip() marks pivots outside
// 2^-400..2^400 with a NaN, and a q0 outside 2^-400..2^400 (so also NaN,
// infinities and zeros) sends the quotient to the plain division.
template <class T>
struct Recip;
template <>
struct Recip<double> {
  using type = double;
  static constexpr bool keep_pivot = true;
  __device__ static double of(double p) {
    const int e = (__double2hiint(p) >> 20) & 0x7FF;
    return (unsigned)(e - (1023 - 400)) <= 800u ? 1.0 / p : __longlong_as_double(0x7FF8000000000000LL);
  }
  __device__ static __forceinline__ double div(double x, double p, double r, bool& bad) {
    const double q0 = __dmul_rn(x, r);
    const double q1 = __fma_rn(__fma_rn(-q0, p, x), r, q0);
    const int e = (__double2hiint(q0) >> 20) & 0x7FF;
    bad = (unsigned)(e - (1023 - 400)) > 800u;
    return __fma_rn(__fma_rn(-q1, p, x), r, q1);
  }
  __device__ static __forceinline__ double slow(double x, double p, double) { return x / p; }
};
// FP32, r = RN64(1/p): x r in FP64 is within 2^-52 of x/p, and a quotient of
// two 24-bit numbers is never nearer than 2^-49 to the middle of two floats
// (an odd 25-bit middle m would need |x - m p| of at least one unit), so
// rounding x r to float rounds x/p.  Zeros, infinities and NaNs come out as
// the division's; only results below the normal range (coarser middles) go to
// the plain division, whose pivot is 1/r rounded to float.
template <>
struct Recip<float> {
  using type = double;
  static constexpr bool keep_pivot = false;
  __device__ static double of(float p) { return 1.0 / (double)p; }
  __device__ static __forceinline__ float div(float x, float, double r, bool& bad) {
    const float q = (float)((double)x * r);
    bad = fabsf(q) < 1.17549435e-38f && x != 0.0f;
    return q;
  }
  __device__ static __forceinline__ float slow(float x, float, double r) { return x / (float)(1.0 / r); }
};

}  // namespace
}  // namespace ab2
