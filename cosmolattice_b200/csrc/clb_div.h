// clb_div.h - division by a divisor known when a handle is made (also compiles as plain C++).
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define CLB_DIV_FN __host__ __device__ __forceinline__
#else
#define CLB_DIV_FN inline
#endif

namespace clb {

// A divisor fixed for a handle's life (the lattice spacing and its square), with what a division by
// it needs.  The FP64 kernels keep the reference's divisions; div_by gives the correctly rounded
// quotient, the bits of a / y, in four FP64 instructions without a branch:
//   q0 = RN(x rh + RN(x rl)), rh + rl = 1/y to twice the precision, so q0 is a faithful rounding;
//   q  = RN(q0 + rh RN(x - q0 y)), Markstein's correction (IBM J. Res. Dev. 34, 1990): with rh =
//        RN(1/y) and q0 faithful the remainder is exact and q = RN(x / y).
// (Outside |x| in about [1e-290, 1e290] / max(1, 1/y) the last bit can differ, a negative zero may lose
// its sign, and an infinite x gives NaN: a run whose state has left the finite numbers reports
// CLB_ENONFINITE either way.)
// The compiler's division is a call on its slow path and a branch per quotient, which serialises
// the ~30 of a gauge kick's site: with div_by the lphi4U1 FP64 kick at 128^3 went from 190 to 118
// us, the lphi4SU2U1 FP64 step at 192^3 from 4.54 to 4.00 ms and its tangent step at 80^3 from 2.34
// to 1.90 ms, all with the same states to the last bit.
struct DivBy {
  double y, rh, rl;
  float rf; // FP32 form: multiplies by the reciprocal of the rounded divisor
};
inline DivBy make_div(double y, float yf)
{
  const double rh = 1.0 / y;
  return DivBy{y, rh, std::fma(-rh, y, 1.0) / y, 1.0f / yf};
}
CLB_DIV_FN double div_by(double x, const DivBy &d)
{
#ifdef __CUDA_ARCH__
  const double q = __fma_rn(x, d.rh, __dmul_rn(x, d.rl));
  return __fma_rn(__fma_rn(-q, d.y, x), d.rh, q);
#else
  const double q = std::fma(x, d.rh, x * d.rl);
  return std::fma(std::fma(-q, d.y, x), d.rh, q);
#endif
}
CLB_DIV_FN float div_by(float x, const DivBy &d)
{
#ifdef __CUDA_ARCH__
  return __fmul_rn(x, d.rf); // never contracted: every instantiation of a kernel rounds alike
#else
  return x * d.rf;
#endif
}

} // namespace clb
