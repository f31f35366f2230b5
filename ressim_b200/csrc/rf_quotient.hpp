// rf_quotient.hpp — s / d from the reciprocal of d, correctly rounded (rf_pencil.cu).  Host and device
// code share it; the CPU tests compile it with g++ and compare with the division.
#pragma once

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define RF_QUO_HD __host__ __device__ __forceinline__
#else
#define RF_QUO_HD inline
#endif

namespace rf {

RF_QUO_HD double quotient_nan() {  // 0x7ff80000 in its high word
#ifdef __CUDA_ARCH__
  return __hiloint2double(0x7ff80000, 0);
#else
  return __builtin_nan("");
#endif
}

RF_QUO_HD unsigned quotient_bits(float v) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(v);
#else
  unsigned b;
  std::memcpy(&b, &v, sizeof(b));
  return b;
#endif
}

// s / d from rd, the correctly rounded reciprocal of d; `ok` false: the quotient needs the general
// division.
// FP64: Markstein's theorem (IBM J. Res. Dev. 34, 1990): with y = RN(1/d) and q within one ulp of
// s/d, r = s - d q is exact and RN(q + r y) = RN(s/d).  q = RN(s y + RN(s y_lo)) with
// y_lo ~ 1/d - y is within half an ulp and a little.  The guards (and the pivot's range in
// pen_recip) keep every intermediate normal.
// A zero quotient may lose its sign (FP64).
// FP32: q = s * RN64(1/d) in FP64 is within 2^-52 (relative) of s/d.  A rounding boundary of FP32 has at
// most 25 bits, so a quotient of two 24-bit numbers is either 2^-49 away from it, and RN32(q) = RN32(s/d),
// or on it, which needs the boundary to have fewer bits than s: between two subnormals.  Those next
// to such a tie, 2^-150 from the rounded result, take the division (about one in 2^20 of the
// subnormal quotients, none of the normal range; a result of zero is right on the tie's other side too).
// No pivot's reciprocal is a NaN here.
RF_QUO_HD double pen_div(double s, double d, double rd, bool& ok) {
  const double rlo = fma(-d, rd, 1.0) * rd;
  const double q = fma(s, rd, s * rlo);
  const double r = fma(-d, q, s);
  const double m = fabs(s);
  ok = m < 1e250 && (m > 1e-250 || m == 0.0) && rd == rd;
  return fma(r, rd, q);
}
RF_QUO_HD float pen_div(float s, float, double rd, bool& ok) {
  const double q = double(s) * rd;
  const float f = float(q);
  ok = true;
  if ((quotient_bits(f) & 0x7fffffffu) - 1u < 0x00800000u)
    ok = !(fabs(fabs(q - double(f)) - 0x1p-150) < 0x1p-170);
  return f;
}
// Pivots whose reciprocal or residual could leave the normal range take the general division.
RF_QUO_HD double pen_recip(double d) {
  const double m = fabs(d);
  return m > 1e-30 && m < 1e30 ? 1.0 / d : quotient_nan();
}
RF_QUO_HD double pen_recip(float d) { return 1.0 / double(d); }

}  // namespace rf
