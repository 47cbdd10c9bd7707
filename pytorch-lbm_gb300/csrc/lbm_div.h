// Quotients by a divisor whose reciprocal is at hand (device and host code).
#pragma once
#include <cmath>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace lbm {

// x / d from r = 1 / d correctly rounded: q = x r, then q + r (x - d q) with the
// remainder in a fused multiply-add (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990).
// Three operations where the division's general form takes about ten; several
// quotients by one d share its reciprocal.  Correctly rounded as long as the
// remainder is representable and the quotient normal (float: |x| above 2^-100 and
// |x / d| above 2^-126), within an ulp below that.  Where the remainder is not a
// number (x, d or the quotient infinite, d zero) the value is x r: as x / d, an
// infinity or zero, or NaN where that is.  (The division itself outside of the
// first range, by a test of x and q: 1024x1024 float 40 -> 73 us a step.)
template <typename T>
struct Div {
  T d, r;
  __host__ __device__ __forceinline__ T operator()(T x) const {
    const T q = x * r, e = std::fma(std::fma(-d, q, x), r, q);
    return e == e ? e : q;
  }
  // of numerators that are finite or NaN, quotients that do not overflow
  __host__ __device__ __forceinline__ T bounded(T x) const {
    const T q = x * r;
    return std::fma(std::fma(-d, q, x), r, q);
  }
};

// x / d by a constant d = cs2 or 2 cs2 (cs2 = 1/3 in T): x times the double-length
// reciprocal hi + lo, hi rounded towards zero and lo > 0 (so an infinite x gives
// that infinity), in two operations: x hi + rnd(x lo), rounded once.  Its error is
// within 0.5 + 2^-p of an ulp (p the type's bits): the correctly rounded quotient for
// every float mantissa but one (0x1.555554p0, a tie but for 2^-24 of an ulp, one ulp
// off); below 2^-100 (float) within an ulp.  (Div's form with its selection in these
// places: 1024x1024 float 40 -> 42 us a step.)
template <typename T>
struct ByCs2;
template <>
struct ByCs2<float> {
  static constexpr float d = 0x1.555556p-2f, hi = 0x1.7ffffep+1f, lo = 0x1.4p-23f;
};
template <>
struct ByCs2<double> {
  static constexpr double d = 0x1.5555555555555p-2, hi = 0x1.8p+1, lo = 0x1.8p-53;
};
static_assert(ByCs2<float>::d == (float)(1.0 / 3.0) && ByCs2<double>::d == 1.0 / 3.0, "cs2");
template <typename T>
struct DivConst {
  T hi, lo;
  __host__ __device__ __forceinline__ T operator()(T x) const { return std::fma(x, hi, x * lo); }
};
template <typename T>
__host__ __device__ __forceinline__ DivConst<T> by_cs2() { return DivConst<T>{ByCs2<T>::hi, ByCs2<T>::lo}; }
template <typename T>
__host__ __device__ __forceinline__ DivConst<T> by_two_cs2() {
  return DivConst<T>{T(0.5) * ByCs2<T>::hi, T(0.5) * ByCs2<T>::lo};
}

}  // namespace lbm
