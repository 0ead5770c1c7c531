// clb_trig.h - sine and cosine of link phases (also compiles as plain C++).
#pragma once

#include <cmath>

#include "clb_div.h"

namespace clb {

// The phases dx g A of the links and dx g a dt pi of the link steps are small (a fraction of a
// radian even where the gauge fields are large), and there the general sincos spends most of its
// ~60 FP64 instructions on the reduction and its branches.  Up to 1/32 the Taylor polynomials to
// x^7 and x^8 are exact to 0.03 of the last place, so the results are correctly rounded but for a
// few in a hundred; beyond, the library's.  A gauge kick forms 6 (lphi4U1) to 21 (the tangent form of
// lphi4SU2U1) of them per site.  Where a field has grown so far that some lanes of a warp are beyond
// (phases of rms 0.0125 and more, dx g A), the kick takes both: us per VV2 step at rms 0.005 / 0.0125 /
// 0.02 / 0.06, lphi4U1 128^3 FP64 160 / 167 / 189 / 194, 99^3 FP32 65 / 68 / 74 / 77 (271 and 110 at every
// angle with the general function, before the other changes to these kicks); lphi4SU2U1, whose kicks
// read stored phases, 128^3 FP64 883 / 884 / 887 / 887, 95^3 FP32 278 / 277 / 279 / 279.
constexpr double kSmallPhase = 0.03125;

#ifdef __CUDA_ARCH__
#define CLB_FMA(a, b, c) __fma_rn(a, b, c)
#define CLB_MUL(a, b) __dmul_rn(a, b)
#define CLB_FMAF(a, b, c) __fmaf_rn(a, b, c)
#define CLB_MULF(a, b) __fmul_rn(a, b)
#else
#define CLB_FMA(a, b, c) std::fma(a, b, c)
#define CLB_MUL(a, b) ((a) * (b))
#define CLB_FMAF(a, b, c) std::fma(a, b, c)
#define CLB_MULF(a, b) ((a) * (b))
#endif

// (sin x / x - 1) / x^2 and (cos x - 1) / x^2 as polynomials in z = x^2 <= kSmallPhase^2
CLB_DIV_FN double sinc_poly(double z)
{
  return CLB_FMA(z, CLB_FMA(z, -1.0 / 5040, 1.0 / 120), -1.0 / 6);
}
CLB_DIV_FN double cosm_poly(double z)
{
  return CLB_FMA(z, CLB_FMA(z, CLB_FMA(z, 1.0 / 40320, -1.0 / 720), 1.0 / 24), -0.5);
}

CLB_DIV_FN void sincos_link(double x, double *s, double *c)
{
  if (std::fabs(x) <= kSmallPhase) {
    const double z = CLB_MUL(x, x);
    *s = CLB_FMA(CLB_MUL(x, z), sinc_poly(z), x);
    *c = CLB_FMA(z, cosm_poly(z), 1.0);
    return;
  }
#ifdef __CUDA_ARCH__
  ::sincos(x, s, c);
#else
  *s = std::sin(x);
  *c = std::cos(x);
#endif
}
CLB_DIV_FN void sincos_link(float x, float *s, float *c)
{
  if (std::fabs(x) <= (float)kSmallPhase) {
    const float z = CLB_MULF(x, x);
    *s = CLB_FMAF(CLB_MULF(x, z), CLB_FMAF(z, 1.0f / 120, -1.0f / 6), x);
    *c = CLB_FMAF(z, CLB_FMAF(z, 1.0f / 24, -0.5f), 1.0f);
    return;
  }
#ifdef __CUDA_ARCH__
  ::sincosf(x, s, c);
#else
  *s = std::sin(x);
  *c = std::cos(x);
#endif
}

} // namespace clb
