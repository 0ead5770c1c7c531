// clb_su2_body.cuh - lphi4SU2U1 site arithmetic, kick, drift and measurement kernels, templated on
// the storage type S (double or float) and the arithmetic type T of the site kernels.  The FP64
// form uses S = T = double and rounds in the reference's order (the unit is compiled without FMA
// contraction); the FP32 form stores and stencils in float (S = T = float) with every kick and
// drift increment added in FP64 and rounded once, and measures in FP64 (T = double over float
// storage).  Included by clb_su2.cuh.
#pragma once

#include "clb_su2.cuh"

#include <type_traits>

namespace clb {
namespace su2d {

template <class T> struct C2 {
  T re, im;
};
// The FP32 form is bound to no rounding order: its products contract into FMAs, written out so that
// the plain and the tangent-linear kernels round alike (the unit is compiled without contraction).
// 128^3 FP32 step 746 -> 723 us, its tangent step at 80^3 (where products with plain numbers also
// lost their zero derivatives) 509 -> 397 us.
template <class T> struct Is32 {
  static constexpr bool v = sizeof(typename TanTraits<T>::base) == 4;
};
__device__ __forceinline__ float mad(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ Tan<float> mad(Tan<float> a, Tan<float> b, Tan<float> c)
{
  return Tan<float>(__fmaf_rn(a.v, b.v, c.v), __fmaf_rn(a.d, b.v, __fmaf_rn(a.v, b.d, c.d)));
}
template <class T> __device__ __forceinline__ C2<T> cmul(C2<T> a, C2<T> b)
{
  if constexpr (Is32<T>::v)
    return C2<T>{mad(a.re, b.re, -(a.im * b.im)), mad(a.re, b.im, a.im * b.re)};
  else
    return C2<T>{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
template <class T> __device__ __forceinline__ C2<T> cadd(C2<T> a, C2<T> b) { return C2<T>{a.re + b.re, a.im + b.im}; }
template <class T> __device__ __forceinline__ C2<T> csub(C2<T> a, C2<T> b) { return C2<T>{a.re - b.re, a.im - b.im}; }
template <class T> __device__ __forceinline__ C2<T> conj_(C2<T> a) { return C2<T>{a.re, -a.im}; }
template <class T> struct Q4 {
  T w, x, y, z;
};
template <class T> __device__ __forceinline__ Q4<T> qmul(const Q4<T> &a, const Q4<T> &b)
{
  if constexpr (Is32<T>::v)
    return Q4<T>{mad(a.w, b.w, -mad(a.x, b.x, mad(a.y, b.y, a.z * b.z))),
                 mad(a.w, b.x, mad(b.w, a.x, mad(a.z, b.y, -(a.y * b.z)))),
                 mad(a.w, b.y, mad(b.w, a.y, mad(a.x, b.z, -(a.z * b.x)))),
                 mad(a.w, b.z, mad(b.w, a.z, mad(a.y, b.x, -(a.x * b.y))))};
  return Q4<T>{a.w * b.w - (a.x * b.x + a.y * b.y + a.z * b.z), a.w * b.x + b.w * a.x - (a.y * b.z - a.z * b.y),
               a.w * b.y + b.w * a.y - (a.z * b.x - a.x * b.z), a.w * b.z + b.w * a.z - (a.x * b.y - a.y * b.x)};
}
template <class T> __device__ __forceinline__ Q4<T> qdag(const Q4<T> &a) { return Q4<T>{a.w, -a.x, -a.y, -a.z}; }
template <class T> struct D2 {
  C2<T> u, v;
};
// U (u, v) with U = [[q0 + i q3, q2 + i q1], [-q2 + i q1, q0 - i q3]]
template <class T> __device__ __forceinline__ D2<T> qapply(const Q4<T> &q, const D2<T> &d)
{
  return D2<T>{cadd(cmul(C2<T>{q.w, q.z}, d.u), cmul(C2<T>{q.y, q.x}, d.v)),
               cadd(cmul(C2<T>{-q.y, q.x}, d.u), cmul(C2<T>{q.w, -q.z}, d.v))};
}
template <class T> __device__ __forceinline__ D2<T> dscale(C2<T> c, const D2<T> &d) { return D2<T>{cmul(c, d.u), cmul(c, d.v)}; }
template <class T> __device__ __forceinline__ C2<T> sprod(const D2<T> &a, const D2<T> &b)
{
  return cadd(cmul(conj_(a.u), b.u), cmul(conj_(a.v), b.v));
}
// i sigma_b applied to a doublet (i z = (-im, re): products with 0 and 1 are left out)
template <class T> __device__ __forceinline__ D2<T> isig(int b, const D2<T> &d)
{
  auto I = [](C2<T> z) { return C2<T>{-z.im, z.re}; };
  if (b == 0) return D2<T>{I(d.v), I(d.u)};
  if (b == 1) return D2<T>{d.v, C2<T>{-d.u.re, -d.u.im}};
  return D2<T>{I(d.u), C2<T>{d.v.im, -d.v.re}};
}
// Divisions of the kernels: the FP64 form keeps the reference's rounding (a / b); the FP32 form,
// bound to no rounding order, multiplies by the reciprocal; the tangent-linear types divide as Tan
// does.
template <class T> __device__ __forceinline__ T kdiv(T a, T b) { return a / b; }
template <> __device__ __forceinline__ float kdiv<float>(float a, float b) { return a * (1.0f / b); }
// the FP32 tangent-linear form: the value part as kdiv<float> forms it (bitwise the plain form)
template <> __device__ __forceinline__ Tan<float> kdiv<Tan<float>>(Tan<float> a, Tan<float> b)
{
  const float r = 1.0f / b.v, q = a.v * r;
  return Tan<float>(q, (a.d - q * b.d) * r);
}

// x / dx and x / dx^2 (DivBy) of a tangent pair: the bits of kdiv by the spacing
__device__ __forceinline__ Tan<double> div_by(Tan<double> a, const DivBy &d)
{
  return Tan<double>(clb::div_by(a.v, d), clb::div_by(a.d, d));
}
__device__ __forceinline__ Tan<float> div_by(Tan<float> a, const DivBy &d) { return Tan<float>(a.v * d.rf, a.d * d.rf); }
using clb::div_by;
// 1 / y of such a divisor, as a plain number of T's precision
template <class T> __device__ __forceinline__ typename TanTraits<T>::base recip(const DivBy &d)
{
  if constexpr (Is32<T>::v)
    return d.rf;
  else
    return d.rh;
}

template <class T> __device__ __forceinline__ T ipw(T x, int n)
{
  if (n < 0) return T(1) / ipw(x, -n);
  T r = x;
#pragma unroll
  for (int i = 1; i < n; ++i) r = r * x;
  return n == 0 ? T(1) : r;
}

// Read-only view of one state at one site (storage S, arithmetic T), with the oracle's names.
// With T = Tan<S> a value reads as (f, df): the state and its tangent.
template <class S, class T> struct Site {
  const S *f;
  const S *df;
  // U(1) link phases exp(-i dx g A_i) for g = gQ of phi (C) and of Phi (D), kept by the drift:
  // [i][0 C, 1 D][site][cos, sin]; null: formed from A here
  const S *ph;
  const Params *a;
  uint32_t s, op[3], om[3]; // the site and its neighbours' offsets, modulo 2^32 (a state of more sites fits no GPU)
  typename TanTraits<T>::base dx;
  T gC, gD, gS, qG, qH, c4;
  __device__ __forceinline__ T F(int c, uint32_t t) const
  {
    const size_t i = fidx(*a, c, t);
    if constexpr (TanTraits<T>::is)
      return T((typename TanTraits<T>::base)f[i], (typename TanTraits<T>::base)df[i]);
    else
      return (T)f[i];
  }
  // the quadruple at index i of the field buffer
  __device__ __forceinline__ Q4<T> quad(size_t i) const
  {
    const V4<S> v = ld4c(f + i);
    if constexpr (TanTraits<T>::is) {
      using B = typename TanTraits<T>::base;
      const V4<S> d = ld4c(df + i);
      return Q4<T>{T((B)v.v[0], (B)d.v[0]), T((B)v.v[1], (B)d.v[1]), T((B)v.v[2], (B)d.v[2]), T((B)v.v[3], (B)d.v[3])};
    } else {
      return Q4<T>{(T)v.v[0], (T)v.v[1], (T)v.v[2], (T)v.v[3]};
    }
  }
  __device__ __forceinline__ Q4<T> link(int i, uint32_t t) const { return quad(fidx(*a, 10 + 4 * i, t)); }
  __device__ __forceinline__ D2<T> dbl(uint32_t t) const
  {
    const Q4<T> q = quad(fidx(*a, 3, t));
    return D2<T>{C2<T>{q.w, q.x}, C2<T>{q.y, q.z}};
  }
  __device__ __forceinline__ C2<T> cs(uint32_t t) const { return C2<T>{F(1, t), F(2, t)}; }
  // the stored phases when the arithmetic type is the storage type (the same cos and sin of the
  // same argument, formed by the drift), else formed here
  __device__ __forceinline__ C2<T> phaseCD(int which, int i, uint32_t t) const
  {
    if constexpr (std::is_same<S, T>::value) {
      if (ph) {
        if constexpr (sizeof(S) == 8) {
          const double2 q = __ldg(reinterpret_cast<const double2 *>(ph + ((size_t)(2 * i + which) * a->n3 + t) * 2));
          return C2<T>{q.x, q.y};
        } else {
          const float2 q = __ldg(reinterpret_cast<const float2 *>(ph + ((size_t)(2 * i + which) * a->n3 + t) * 2));
          return C2<T>{q.x, q.y};
        }
      }
    }
    return phase(which == 0 ? gC : gD, i, t);
  }
  __device__ __forceinline__ C2<T> phaseC(int i, uint32_t t) const { return phaseCD(0, i, t); }
  __device__ __forceinline__ C2<T> phaseD(int i, uint32_t t) const { return phaseCD(1, i, t); }
  __device__ __forceinline__ C2<T> phase(T g, int i, uint32_t t) const
  {
    const T th = (-dx * g) * F(7 + i, t);
    C2<T> r;
    sincos_link(th, &r.im, &r.re);
    return r;
  }
  __device__ __forceinline__ T normD(uint32_t t) const
  {
    const Q4<T> d = quad(fidx(*a, 3, t));
    return sqrt(((d.w * d.w + d.x * d.x) + d.y * d.y) + d.z * d.z);
  }
  __device__ __forceinline__ T normC(uint32_t t) const { return sqrt(F(1, t) * F(1, t) + F(2, t) * F(2, t)); }
  __device__ __forceinline__ T potTerm(int k) const
  {
    const T nD = normD(s);
    if (k == 0) return c4 * ipw(nD, 4);
    if (k == 1) return qG * ipw(nD * F(0, s), 2);
    return 2 * qH * ipw(nD * normC(s), 2);
  }
  __device__ __forceinline__ T pot() const { return (potTerm(0) + potTerm(1)) + potTerm(2); }
  // pot() from |Phi|, |phi| and S at this site, formed as potTerm forms them
  __device__ __forceinline__ T pot_at(T nD, T nC, T Sv) const
  {
    return (c4 * ipw(nD, 4) + qG * ipw(nD * Sv, 2)) + 2 * qH * ipw(nD * nC, 2);
  }
  __device__ __forceinline__ uint32_t pl(int i) const { return s + op[i]; }
  __device__ __forceinline__ uint32_t mi(int i) const { return s + om[i]; }
  __device__ __forceinline__ uint32_t plmi(int i, int j) const { return i == j ? s : s + op[i] + om[j]; }
  __device__ __forceinline__ D2<T> wD(int i) const { return dscale(phaseD(i, s), qapply(link(i, s), dbl(pl(i)))); }
  __device__ __forceinline__ C2<T> wC(int i) const { return cmul(phaseC(i, s), cs(pl(i))); }
  __device__ __forceinline__ T lapl(int comp) const
  {
    const T c = F(comp, s);
    T t[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) t[d] = (F(comp, pl(d)) + F(comp, mi(d))) - 2 * c;
    return recip<T>(a->ddx2) * ((t[0] + t[1]) + t[2]);
  }
  __device__ __forceinline__ T fd(int comp, uint32_t t0, uint32_t t1) const { return div_by(F(comp, t1) - F(comp, t0), a->ddx); }
  __device__ __forceinline__ Q4<T> plaq(int i, int j) const
  {
    return qmul(qmul(qmul(link(i, s), link(j, pl(i))), qdag(link(i, pl(j)))), qdag(link(j, s)));
  }
  __device__ __forceinline__ Q4<T> plaqBack(int i, int j) const
  {
    const uint32_t sm = mi(j);
    return qdag(qmul(qmul(qmul(link(i, s), qdag(link(j, plmi(i, j)))), qdag(link(i, sm))), link(j, sm)));
  }
};

template <class S, class T> __device__ __forceinline__ Site<S, T> make_site(const S *f, const Params &a, uint32_t s)
{
  Site<S, T> v;
  v.f = f;
  v.df = nullptr;
  v.ph = nullptr;
  v.a = &a;
  v.s = s;
  v.dx = (typename TanTraits<T>::base)a.dx;
  v.gC = (T)a.gC;
  v.gD = (T)a.gD;
  v.gS = (T)a.gS;
  v.qG = (T)a.qG;
  v.qH = (T)a.qH;
  v.c4 = (T)a.c4;
  site_offsets(a.divN, s, v.op, v.om);
  return v;
}

// Derivatives of the couplings along the tangent direction, in the model's order: qG, qH, gQ of
// phi, gQ of Phi under U(1), gQ of Phi under SU(2), c4.
struct CoupDot {
  double v[6];
};

// Tangent-linear view: the state f with its tangent df, and the couplings with their tangents.
template <class S>
__device__ __forceinline__ Site<S, Tan<S>> make_site_tan(const S *f, const S *df, const Params &a, uint32_t s,
                                                        const CoupDot &cd)
{
  using T = Tan<S>;
  Site<S, T> v;
  v.f = f;
  v.df = df;
  v.ph = nullptr;
  v.a = &a;
  v.s = s;
  v.dx = (S)a.dx;
  auto cp = [&](double x, int k) { return T((S)x, (S)cd.v[k]); };
  v.qG = cp(a.qG, 0);
  v.qH = cp(a.qH, 1);
  v.gC = cp(a.gC, 2);
  v.gD = cp(a.gD, 3);
  v.gS = cp(a.gS, 4);
  v.c4 = cp(a.c4, 5);
  site_offsets(a.divN, s, v.op, v.om);
  return v;
}

// ---- momentum kernels at one site (momentum-component order) ----------------------------------
// Direction d's term of the gradient energies cGrad2 and dGrad2 below, from the forward product w
// (the phi or Phi value at x + d parallel transported to x) and the value c at x.
template <class S, class T> __device__ __forceinline__ T cgrad_term(const Site<S, T> &v, const C2<T> &w, const C2<T> &c)
{
  const C2<T> d0 = csub(w, c);
  const C2<T> d{div_by(d0.re, v.a->ddx), div_by(d0.im, v.a->ddx)};
  return d.re * d.re + d.im * d.im;
}
template <class S, class T> __device__ __forceinline__ T dgrad_term(const Site<S, T> &v, const D2<T> &w, const D2<T> &c)
{
  const C2<T> du0 = csub(w.u, c.u), dv0 = csub(w.v, c.v);
  const DivBy &dd = v.a->ddx;
  const C2<T> du{div_by(du0.re, dd), div_by(du0.im, dd)}, dv{div_by(dv0.re, dd), div_by(dv0.im, dd)};
  return (du.re * du.re + du.im * du.im) + (dv.re * dv.re + dv.im * dv.im);
}

// g2: also form cGrad2 (covLapC) or dGrad2 (covLapD) from the same forward products.
template <class S, class T> __device__ __forceinline__ C2<T> covLapC(const Site<S, T> &v, T *g2 = nullptr)
{
  C2<T> plus{0, 0}, minus{0, 0};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const C2<T> w = cmul(v.phaseC(d, v.s), v.cs(v.pl(d)));
    if (g2) {
      const T n2 = cgrad_term(v, w, v.cs(v.s));
      *g2 = d == 0 ? n2 : *g2 + n2;
    }
    const C2<T> m = cmul(conj_(v.phaseC(d, v.mi(d))), v.cs(v.mi(d)));
    plus = d == 0 ? w : cadd(plus, w);
    minus = d == 0 ? m : cadd(minus, m);
  }
  const DivBy &dx2 = v.a->ddx2;
  const C2<T> c = v.cs(v.s);
  return C2<T>{div_by((plus.re + minus.re) - 6 * c.re, dx2), div_by((plus.im + minus.im) - 6 * c.im, dx2)};
}

template <class S, class T> __device__ __forceinline__ void covLapD(const Site<S, T> &v, T out[4], T *g2 = nullptr)
{
  D2<T> plus{}, minus{};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const D2<T> w = qapply(v.link(d, v.s), dscale(v.phaseD(d, v.s), v.dbl(v.pl(d))));
    if (g2) {
      const T n2 = dgrad_term(v, w, v.dbl(v.s));
      *g2 = d == 0 ? n2 : *g2 + n2;
    }
    const uint32_t sm = v.mi(d);
    const D2<T> m = qapply(qdag(v.link(d, sm)), dscale(conj_(v.phaseD(d, sm)), v.dbl(sm)));
    if (d == 0) {
      plus = w;
      minus = m;
    } else {
      plus = D2<T>{cadd(plus.u, w.u), cadd(plus.v, w.v)};
      minus = D2<T>{cadd(minus.u, m.u), cadd(minus.v, m.v)};
    }
  }
  const DivBy &dx2 = v.a->ddx2;
  const D2<T> c = v.dbl(v.s);
  out[0] = div_by((plus.u.re + minus.u.re) - 6 * c.u.re, dx2);
  out[1] = div_by((plus.u.im + minus.u.im) - 6 * c.u.im, dx2);
  out[2] = div_by((plus.v.re + minus.v.re) - 6 * c.v.re, dx2);
  out[3] = div_by((plus.v.im + minus.v.im) - 6 * c.v.im, dx2);
}

// Kick coefficients pow(aI, 1+alpha), pow(aI, 3+alpha), its half and pow(aI, -1+alpha).
template <class T> struct Coef {
  T A, B, B2, G;
};

// SECT: 0 all components; 1 S, phi, Phi and A (K[0..9]); 2 the SU(2) field (K[10..18]);
// 3 S, phi and Phi (K[0..6]); 4 A (K[7..9]); 5 S and phi (K[0..2]); 6 Phi (K[3..6]).  Each
// component's kernel is the same expression in every SECT that holds it.
__host__ __device__ constexpr bool sect_sphi(int sect) { return sect == 0 || sect == 1 || sect == 3 || sect == 5; }
__host__ __device__ constexpr bool sect_dbl(int sect) { return sect == 0 || sect == 1 || sect == 3 || sect == 6; }
__host__ __device__ constexpr bool sect_scalars(int sect) { return sect_sphi(sect) || sect_dbl(sect); }
__host__ __device__ constexpr bool sect_u1(int sect) { return sect == 0 || sect == 1 || sect == 4; }
__host__ __device__ constexpr bool sect_su2(int sect) { return sect == 0 || sect == 2; }
// momentum sectors [sect_g0, sect_g1) of SECT (0 S, 1 phi, 2 Phi, 3 A, 4 SU(2))
__host__ __device__ constexpr int sect_g0(int sect) { return sect == 2 ? 4 : sect == 4 ? 3 : sect == 6 ? 2 : 0; }
__host__ __device__ constexpr int sect_g1(int sect)
{
  return sect == 1 || sect == 4 ? 4 : sect == 3 || sect == 6 ? 3 : sect == 5 ? 2 : 5;
}
// whether SECT writes partial slot k of a kick sweep: the momentum sums of its sectors (k < 5 and
// k >= 11), the gradient sums of S, phi (5, 6) and Phi (7), B^2 of A (8) and SU(2) (9), V (10,
// with S and phi)
__host__ __device__ constexpr bool sect_owns(int sect, int k)
{
  return k < 5 || k >= 11 ? ((k < 5 ? k : k - 11) >= sect_g0(sect) && (k < 5 ? k : k - 11) < sect_g1(sect))
         : k == 7 ? sect_dbl(sect) : k == 8 ? sect_u1(sect) : k == 9 ? sect_su2(sect) : sect_sphi(sect);
}

// Per-site terms of the volume averages a kick sweep reduces with RF (fieldfunctionals.h):
// gradient energies of S, phi and Phi, B^2 of A and of SU(2), and V.  They equal, to the last
// bit, what sGrad2, cGrad2, dGrad2, aB2, gB2 and Site::pot give at the site.
template <class T> struct SiteAvg {
  T g2S, g2C, g2D, b2A, b2G, pot;
};
template <class S, class T> __device__ __forceinline__ T sGrad2(const Site<S, T> &v);
template <class S, class T> __device__ __forceinline__ T aB2(const Site<S, T> &v, const T (*g)[3] = nullptr);
template <class S, class T> __device__ __forceinline__ T gB2(const Site<S, T> &v, const T *dev = nullptr);

// The Wilson term 2 - 2 w of a plaquette in <B^2>, in two steps so that the parts of a kick can hand on one
// value: plaq_dev() of the plaquette, then gap().  FP64 links keep the expression as it stands (plaq_dev
// is w).  Links held in FP32 give a w next to 1 whose rounding (6e-8) is of the size of the gap itself on
// a fine lattice, and the factor 4 / (dx^4 g^2) carries it through the start's a-dot into all momenta:
// with links of rms 1e-3 the magnetic energy was off by 1e-5 to 2e-3 and the tangent observable by up to
// a tenth, and every change of the products' rounding shifted a(t).  There plaq_dev is the gap, formed as
// 2 (x^2 + y^2 + z^2) / (1 + w), the same for a unit quaternion and free of the cancellation.  Its tangent
// stays -2 dw, which does not cancel, and is the reference expression's for link tangents of any kind (the
// quotient's is the same along the group only).
template <class S, class T> __device__ __forceinline__ T gap(T dev)
{
  if constexpr (sizeof(S) == 4)
    return dev;
  else
    return 2 - 2 * dev;
}
template <class S, class T> __device__ __forceinline__ T plaq_dev(const Q4<T> &P)
{
  if constexpr (sizeof(S) == 4 && TanTraits<T>::is) {
    using B = typename TanTraits<T>::base;
    return T(plaq_dev<S>(Q4<B>{P.w.v, P.x.v, P.y.v, P.z.v}), -2 * P.w.d);
  } else if constexpr (sizeof(S) == 4) {
    return P.w > 0 ? kdiv(2 * ((P.x * P.x + P.y * P.y) + P.z * P.z), 1 + P.w) : 2 - 2 * P.w;
  } else {
    return P.w;
  }
}

// (1/dx)^3 / gS; the tangent form's gS can carry a derivative
template <class S, class T> __device__ __forceinline__ T su2_ngrad(const Site<S, T> &v)
{
  if constexpr (std::is_same<T, double>::value)
    return v.a->ngrad;
  else if constexpr (std::is_same<T, float>::value)
    return v.a->ngrad_f;
  else
    return kdiv(T(ipw(recip<T>(v.a->ddx), 3)), v.gS);
}

// AVG: also form the SiteAvg terms of the sectors in SECT into *av, from the covariant products,
// differences and plaquettes the kernels form anyway.
template <int SECT = 0, bool AVG = false, class S, class T>
__device__ __forceinline__ void kernels(const Site<S, T> &v, const Coef<T> &C, T K[NP], SiteAvg<T> *av = nullptr)
{
  const Params &a = *v.a;
  const uint32_t s = v.s;
  const T A = C.A, B = C.B, B2 = C.B2, G = C.G;
  const T qG = v.qG, qH = v.qH, c4 = v.c4;
  const typename TanTraits<T>::base rfo2 = (typename TanTraits<T>::base)a.rfo2;
  if constexpr (sect_scalars(SECT)) {
    const T nD = v.normD(s), nC = v.normC(s), Sv = v.F(0, s);
    if constexpr (sect_sphi(SECT)) {
      K[0] = A * v.lapl(0) - B * (2 * qG * ipw(nD, 2) * Sv);
      const C2<T> cl = covLapC(v, AVG ? &av->g2C : nullptr);
      const T ndC = 4 * qH * ipw(nD, 2) * nC;
      K[1] = A * cl.re - B2 * (kdiv(ndC, nC) * v.F(1, s));
      K[2] = A * cl.im - B2 * (kdiv(ndC, nC) * v.F(2, s));
    }
    if constexpr (sect_dbl(SECT)) {
      T dl[4];
      covLapD(v, dl, AVG ? &av->g2D : nullptr);
      const T ndD = c4 * (4 * ipw(nD, 3)) + nD * (2 * qG * ipw(Sv, 2) + 4 * qH * ipw(nC, 2));
      const Q4<T> d = v.quad(fidx(a, 3, s));
      const T dv[4] = {d.w, d.x, d.y, d.z};
#pragma unroll
      for (int c = 0; c < 4; ++c) K[3 + c] = A * dl[c] - B2 * (kdiv(ndD, nD) * dv[c]);
    }
    if constexpr (AVG && sect_sphi(SECT)) {
      av->g2S = sGrad2(v);
      av->pot = v.pot_at(nD, nC, Sv);
    }
  }
  if constexpr (sect_u1(SECT)) {
    const D2<T> D0 = v.dbl(s);
    const C2<T> C0 = v.cs(s);
    T g0s[3][3]; // g0s[i][j]: forward difference of A_j along i
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const T lap = v.lapl(7 + i);
      T grad = 0;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const T g0 = v.fd(7 + j, s, v.pl(i));
        g0s[i][j] = g0;
        const T g1 = v.fd(7 + j, v.mi(j), v.plmi(i, j));
        const T t = div_by(g0 - g1, a.ddx);
        grad = j == 0 ? t : grad + t;
      }
      const T Jc = v.gC * cmul(conj_(v.wC(i)), C0).im;
      const T Jd = v.gD * sprod(v.wD(i), D0).im;
      const T J = 2 * recip<T>(a.ddx) * rfo2 * (Jc + Jd);
      K[7 + i] = G * (lap - grad) - A * J;
    }
    if constexpr (AVG) av->b2A = aB2(v, g0s);
  }
  if constexpr (sect_su2(SECT)) {
    const D2<T> Dg = v.dbl(s);
    const T normGrad = su2_ngrad(v) * G;
    const T normSrc = recip<T>(a.ddx) * A;
    T dev[3]; // plaq_dev of plaq(1, 0), plaq(2, 0), plaq(2, 1)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      T gr[3] = {0, 0, 0}, gb[3] = {0, 0, 0};
      bool first = true;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (j == i) continue;
        const Q4<T> P = v.plaq(i, j), Pb = v.plaqBack(i, j);
        if (j < i) dev[i + j - 1] = plaq_dev<S>(P);
        const T pv[3] = {P.x, P.y, P.z}, bv[3] = {Pb.x, Pb.y, Pb.z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          gr[c] = first ? pv[c] : gr[c] + pv[c];
          gb[c] = first ? bv[c] : gb[c] + bv[c];
        }
        first = false;
      }
      const D2<T> W = v.wD(i);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const T J = rfo2 / 2 * (v.gS * sprod(W, isig(c, Dg)).re);
        K[10 + 3 * i + c] = -normGrad * (gr[c] - gb[c]) - normSrc * J;
      }
    }
    if constexpr (AVG) av->b2G = gB2(v, dev);
  }
}

// ---- per-site averages (fieldfunctionals.h) -------------------------------------------------------
template <class S, class T> __device__ __forceinline__ T sGrad2(const Site<S, T> &v)
{
  T acc = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const T g = v.fd(0, v.s, v.pl(j));
    acc = j == 0 ? g * g : acc + g * g;
  }
  return acc;
}
template <class S, class T> __device__ __forceinline__ T cGrad2(const Site<S, T> &v)
{
  const C2<T> c = v.cs(v.s);
  T acc = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const T n2 = cgrad_term(v, v.wC(j), c);
    acc = j == 0 ? n2 : acc + n2;
  }
  return acc;
}
template <class S, class T> __device__ __forceinline__ T dGrad2(const Site<S, T> &v)
{
  const D2<T> c = v.dbl(v.s);
  T acc = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const T n2 = dgrad_term(v, qapply(v.link(j, v.s), dscale(v.phaseD(j, v.s), v.dbl(v.pl(j)))), c);
    acc = j == 0 ? n2 : acc + n2;
  }
  return acc;
}
// aB2's g and gB2's dev: the differences and plaquettes as kernels() formed them
template <class S, class T> __device__ __forceinline__ T Fij(const Site<S, T> &v, int i, int j)
{
  return v.fd(7 + j, v.s, v.pl(i)) - v.fd(7 + i, v.s, v.pl(j));
}
template <class S, class T> __device__ __forceinline__ T aB2(const Site<S, T> &v, const T (*g)[3])
{
  auto F = [&](int i, int j) { return g ? g[i][j] - g[j][i] : Fij(v, i, j); };
  const T f21 = F(1, 0), f31 = F(2, 0), f32 = F(2, 1);
  return f21 * f21 + (f31 * f31 + f32 * f32);
}
template <class S, class T> __device__ __forceinline__ T gB2(const Site<S, T> &v, const T *dev)
{
  const T c = kdiv(T(4.0), ipw(v.dx, 4) * ipw(v.gS, 2));
  const T t10 = gap<S>(dev ? dev[0] : plaq_dev<S>(v.plaq(1, 0))), t20 = gap<S>(dev ? dev[1] : plaq_dev<S>(v.plaq(2, 0))),
          t21 = gap<S>(dev ? dev[2] : plaq_dev<S>(v.plaq(2, 1)));
  return c * (t10 + (t20 + t21));
}
// The SiteAvg terms of the sectors in SECT, formed on their own (a sweep that does not kick).
template <int SECT, class S, class T> __device__ __forceinline__ SiteAvg<T> site_avg(const Site<S, T> &v)
{
  SiteAvg<T> av{};
  if constexpr (sect_sphi(SECT)) {
    av.g2S = sGrad2(v);
    av.g2C = cGrad2(v);
    av.pot = v.pot();
  }
  if constexpr (sect_dbl(SECT)) av.g2D = dGrad2(v);
  if constexpr (sect_u1(SECT)) av.b2A = aB2(v);
  if constexpr (sect_su2(SECT)) av.b2G = gB2(v);
  return av;
}

// First momentum component of sector g (0 S, 1 phi, 2 Phi, 3 A, 4 SU(2)); g = 5: one past the last.
__host__ __device__ constexpr int sector_c0(int g) { return g == 0 ? 0 : g == 1 ? 1 : g == 2 ? 3 : g == 3 ? 7 : g == 4 ? 10 : NP; }

// momentum sums of sectors [G0, G1) (FP64) from momentum values q[19], reading only their
// components q[sector_c0(G0) .. sector_c0(G1))
template <int G0 = 0, int G1 = 5, class R> __device__ __forceinline__ void pi2s(const R *qs, double out[5])
{
  double q[NP];
  for (int c = sector_c0(G0); c < sector_c0(G1); ++c) q[c] = (double)qs[c];
  if (G0 <= 0 && G1 > 0) out[0] = q[0] * q[0];
  if (G0 <= 1 && G1 > 1) out[1] = q[1] * q[1] + q[2] * q[2];
  if (G0 <= 2 && G1 > 2) out[2] = ((q[3] * q[3] + q[4] * q[4]) + q[5] * q[5]) + q[6] * q[6];
  if (G0 <= 3 && G1 > 3) out[3] = (q[7] * q[7] + q[8] * q[8]) + q[9] * q[9];
  if (G1 == 5) {
    double acc = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double ai = 0;
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const double e = q[10 + 3 * i + b];
        ai = b == 0 ? 4 * (e * e) : ai + 4 * (e * e);
      }
      acc = i == 0 ? ai : acc + ai;
    }
    out[4] = acc;
  }
}

__device__ __forceinline__ int sector(int c) { return c == 0 ? 0 : c < 3 ? 1 : c < 7 ? 2 : c < 10 ? 3 : 4; }

// Kick sweep: NK (0..2) in-place kicks with the kernel at the current fields, each increment added
// in FP64 and rounded to the storage type once.  Partials: [0..4] momentum sums after the first kick
// (or as they are, NK = 0), [5..10] <grad^2> S, phi, Phi, <B^2> U(1), SU(2), <V>; [11..15] the
// momentum sums after the second kick.
// Resident 128-thread blocks per SM: FP32 gains from four (128 registers, 1.28x), FP64 keeps three
// (170 registers); more spills than occupancy pays for beyond that.
#ifndef CLB_SU2_KICK_MINB_F32
#define CLB_SU2_KICK_MINB_F32 4
#endif
#ifndef CLB_SU2_KICK_MINB_F64
#define CLB_SU2_KICK_MINB_F64 3
#endif
// SECT (as kernels()): 0 every sector in one sweep; else a part of a split sweep, run one after the
// other over the same grid: 1 in halves, 3 in three parts, 5 and 6 in four, each with the SU(2) part, that
// of the three and four parts with A (k_kick_links).  Each part updates, reduces and writes only its own components and partial slots
// (sect_owns), so the parts hold fewer registers than the whole.  The kicks read the fields only, so
// the parts' order is free.  Four blocks per SM timed best for the parts, FP64 and FP32.
#ifndef CLB_SU2_HALF_MINB_F32
#define CLB_SU2_HALF_MINB_F32 4
#endif
#ifndef CLB_SU2_HALF_MINB_F64
#define CLB_SU2_HALF_MINB_F64 4
#endif
// the FP64 S, phi, Phi part (SECT 3); four blocks timed best at 192^3 (4.99 ms per step, 5.37 with three)
#ifndef CLB_SU2_P3_MINB_F64
#define CLB_SU2_P3_MINB_F64 CLB_SU2_HALF_MINB_F64
#endif
// the FP64 four-part sweep's S and phi part (SECT 5) and Phi part (SECT 6)
#ifndef CLB_SU2_P5_MINB_F64
#define CLB_SU2_P5_MINB_F64 CLB_SU2_HALF_MINB_F64
#endif
#ifndef CLB_SU2_P6_MINB_F64
#define CLB_SU2_P6_MINB_F64 CLB_SU2_HALF_MINB_F64
#endif
template <class S, int NK, bool RF, bool RP, int SECT = 0>
__global__ void __launch_bounds__(128, SECT == 0   ? (sizeof(S) == 4 ? CLB_SU2_KICK_MINB_F32 : CLB_SU2_KICK_MINB_F64)
                                       : sizeof(S) == 4 ? CLB_SU2_HALF_MINB_F32
                                       : SECT == 3      ? CLB_SU2_P3_MINB_F64
                                       : SECT == 5      ? CLB_SU2_P5_MINB_F64
                                       : SECT == 6      ? CLB_SU2_P6_MINB_F64
                                                        : CLB_SU2_HALF_MINB_F64)
    k_kick(const S *__restrict__ f, S *__restrict__ p, Params a, Kick kc, const State *__restrict__ stp,
           double *__restrict__ partials, const S *__restrict__ ph)
{
  constexpr int G0 = sect_g0(SECT), G1 = sect_g1(SECT);                   // sectors [G0, G1)
  constexpr int C0 = sector_c0(G0), C1 = sector_c0(G1);                    // momentum components [C0, C1)
  __shared__ double smem[(128 / 32) * kRed];
  griddep_wait();
  griddep_launch();
  const State st = *stp;
  double acc[kRed];
#pragma unroll
  for (int k = 0; k < kRed; ++k) acc[k] = 0;
  for_sites(a.N, a.n3, a.order, [&](uint32_t s) {
    Site<S, S> v = make_site<S, S>(f, a, s);
    v.ph = ph;
    S q[NP];
#pragma unroll
    for (int c = C0; c < C1; ++c) q[c] = p[(size_t)c * a.n3 + s];
    SiteAvg<S> av; // with RF: formed by kernels() when the sweep kicks, else by site_avg()
    if (NK > 0) {
      S K[NP];
      kernels<SECT, RF>(v, Coef<S>{(S)st.kA, (S)st.kB, (S)st.kB2, (S)st.kG}, K, &av);
#pragma unroll
      for (int k = 0; k < NK; ++k) {
#pragma unroll
        for (int c = C0; c < C1; ++c) q[c] = (S)((double)q[c] + kc.h[k][sector(c)] * (double)K[c]);
        if (RP) {
          double t[5];
          pi2s<G0, G1>(q, t);
#pragma unroll
          for (int g = G0; g < G1; ++g) acc[(k == 0 ? 0 : 11) + g] += t[g];
        }
      }
#pragma unroll
      for (int c = C0; c < C1; ++c) p[(size_t)c * a.n3 + s] = q[c];
    } else if (RP) {
      double t[5];
      pi2s<G0, G1>(q, t);
#pragma unroll
      for (int g = G0; g < G1; ++g) acc[g] += t[g];
    }
    if (RF && NK == 0) av = site_avg<SECT>(v);
    if (RF) {
      if (sect_sphi(SECT)) {
        acc[5] += (double)av.g2S;
        acc[6] += (double)av.g2C;
      }
      if (sect_dbl(SECT)) acc[7] += (double)av.g2D;
      if (sect_u1(SECT)) acc[8] += (double)av.b2A;
      if (sect_su2(SECT)) acc[9] += (double)av.b2G;
      if (sect_sphi(SECT)) acc[10] += (double)av.pot;
    }
  });
  if (RF || RP) {
    block_reduce<kRed, 128>(acc, smem);
    if (threadIdx.x == 0)
#pragma unroll
      for (int k = 0; k < kRed; ++k)
        if (sect_owns(SECT, k)) partials[(size_t)blockIdx.x * kRed + k] = acc[k];
  }
}

// Drifts (velocityverlet.h:181-222; the leapfrog's forms leapfrog.h:203-236 have lf = 1), in FP64
// and rounded to the storage type once.  The link step's exponential from n = |p|, as the reference
// forms it (FP64 storage); rounded to FP32 afterwards it comes from n^2 directly where that is
// small, without the square root and the division.
template <class S> __device__ __forceinline__ Q4<double> qexp(double p1, double p2, double p3)
{
  const double n2 = p1 * p1 + p2 * p2 + p3 * p3;
  if (sizeof(S) == 4 && n2 <= kSmallPhase * kSmallPhase) {
    const double sn = __fma_rn(n2, sinc_poly(n2), 1.0);
    return Q4<double>{__fma_rn(n2, cosm_poly(n2), 1.0), sn * p1, sn * p2, sn * p3};
  }
  const double n = sqrt(n2);
  if (n == 0) return Q4<double>{1, 0, 0, 0};
  double s, c;
  sincos_link(n, &s, &c);
  const double sn = s / n;
  return Q4<double>{c, sn * p1, sn * p2, sn * p3};
}
// The U(1) link phases of A_i(x) for both couplings, exactly as Site::phase forms them, into the
// phase arrays the kick reads.
template <class S> __device__ __forceinline__ void put_phases(S *__restrict__ ph, const Params &a, int i, size_t s, S A)
{
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const S th = (-(S)a.dx * (S)(which == 0 ? a.gC : a.gD)) * A;
    S c, sn;
    sincos_link(th, &sn, &c);
    S *q = ph + ((size_t)(2 * i + which) * a.n3 + s) * 2;
    if constexpr (sizeof(S) == 8)
      *reinterpret_cast<double2 *>(q) = double2{c, sn};
    else
      *reinterpret_cast<float2 *>(q) = float2{c, sn};
  }
}
template <class S> __global__ void __launch_bounds__(256) k_phases(const S *__restrict__ f, S *__restrict__ ph, Params a)
{
  for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < a.n3; s += (size_t)gridDim.x * blockDim.x)
    for (int i = 0; i < 3; ++i) put_phases(ph, a, i, s, f[fidx(a, 7 + i, s)]);
}

template <class S>
__global__ void __launch_bounds__(256)
    k_drift(S *__restrict__ f, const S *__restrict__ p, Params a, double w, int lf, const State *__restrict__ stp,
            S *__restrict__ ph, double dtd)
{
  // dtd: the time step of this drift (the position Verlet's half drifts pass dt/2)
  griddep_wait();
  griddep_launch();
  const double dt = dtd, p3 = stp->p3, p1 = stp->p1;
  const double cC = lf ? p3 * dt : p3 * dt * w;
  const double cA = lf ? p1 * dt : p1 * w * dt;
  const double cG = lf ? p1 * a.dx * dt * a.gS : w * p1 * a.dx * dt * a.gS;
  const double dtw = lf ? dt : dt * w;
  const size_t n3 = a.n3;
  for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < n3; s += (size_t)gridDim.x * blockDim.x) {
    S pv[NP]; // all at once: the sweep waits on loads (95^3 FP32 56.0 us against 59.8)
#pragma unroll
    for (int c = 0; c < NP; ++c) pv[c] = p[c * n3 + s];
    f[s] = (S)((double)f[s] + p3 * (dtw * (double)pv[0]));
    for (int c = 1; c < 3; ++c) f[c * n3 + s] = (S)((double)f[c * n3 + s] + cC * (double)pv[c]);
    {
      S *fd = f + fidx(a, 3, s);
      V4<S> d = ld4(fd);
      for (int c = 0; c < 4; ++c) d.v[c] = (S)((double)d.v[c] + cC * (double)pv[3 + c]);
      st4(fd, d.v[0], d.v[1], d.v[2], d.v[3]);
    }
    for (int i = 0; i < 3; ++i) {
      S *fa = f + fidx(a, 7 + i, s);
      const S A = (S)((double)*fa + cA * (double)pv[7 + i] * 1.0);
      *fa = A;
      put_phases(ph, a, i, s, A);
    }
    for (int i = 0; i < 3; ++i) {
      const S *pu = pv + 10 + 3 * i;
      S *fu = f + fidx(a, 10 + 4 * i, s);
      const V4<S> q = ld4(fu);
      const Q4<double> E = qexp<S>(cG * (double)pu[0], cG * (double)pu[1], cG * (double)pu[2]);
      const Q4<double> U = qmul(E, Q4<double>{(double)q.v[0], (double)q.v[1], (double)q.v[2], (double)q.v[3]});
      st4(fu, (S)U.w, (S)U.x, (S)U.y, (S)U.z);
    }
  }
}

// Re-unitarisation of the stored links (FP32 form): U <- U / |U| in FP64.
template <class S> __global__ void __launch_bounds__(256) k_unitarize(S *__restrict__ f, Params a)
{
  const size_t n3 = a.n3;
  for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < 3 * n3; s += (size_t)gridDim.x * blockDim.x) {
    S *fu = f + a.oU + 4 * s;
    const V4<S> q = ld4(fu);
    const double w = q.v[0], x = q.v[1], y = q.v[2], z = q.v[3];
    const double r = 1.0 / sqrt(((w * w + x * x) + y * y) + z * z);
    st4(fu, (S)(w * r), (S)(x * r), (S)(y * r), (S)(z * r));
  }
}

// ---- measurement sums (one sweep) ----------------------------------------------------------------
// [0..4] momentum sums of the five sectors, [5..10] field sums as in the kick sweep, [11..13] the
// three potential terms, means [14..41] (seven rows of f, f^2, m, m^2 with raw values), Gauss
// U(1) [42..45] (|LHS-RHS|, |sum|, |RHS|, |LHS|), Gauss SU(2) [46..57] (same per algebra index).
template <class S>
__global__ void __launch_bounds__(128)
    k_measure(const S *__restrict__ f, const S *__restrict__ p, Params a, double am, double ag,
              double *__restrict__ partials)
{
  __shared__ double smem[(128 / 32) * kMeas];
  double acc[kMeas];
  for (int k = 0; k < kMeas; ++k) acc[k] = 0;
  const size_t n3 = a.n3;
  const double dx = a.dx;
  for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < n3; s += (size_t)gridDim.x * blockDim.x) {
    const Site<S, double> v = make_site<S, double>(f, a, (uint32_t)s);
    double q[NP];
    for (int c = 0; c < NP; ++c) q[c] = (double)p[(size_t)c * n3 + s];
    double t[5];
    pi2s(q, t);
    for (int g = 0; g < 5; ++g) acc[g] += t[g];
    acc[5] += sGrad2(v);
    acc[6] += cGrad2(v);
    acc[7] += dGrad2(v);
    acc[8] += aB2(v);
    acc[9] += gB2(v);
    acc[10] += v.pot();
    for (int k = 0; k < 3; ++k) acc[11 + k] += v.potTerm(k);
    auto row = [&](int r, double fv, double mv) {
      acc[14 + 4 * r] += fv;
      acc[15 + 4 * r] += fv * fv;
      acc[16 + 4 * r] += mv;
      acc[17 + 4 * r] += mv * mv;
    };
    const double r2 = sqrt(2.0);
    row(0, v.F(0, s), q[0] * am);
    row(1, r2 * v.F(1, s), r2 * q[1] * am);
    row(2, r2 * v.F(2, s), r2 * q[2] * am);
    {
      const double pa = q[1] * am, pb = q[2] * am;
      row(3, v.normC(s), sqrt(pa * pa + pb * pb));
    }
    {
      double pd = 0;
      for (int c = 0; c < 4; ++c) pd += q[3 + c] * q[3 + c];
      row(4, v.normD(s), sqrt(pd) * am);
    }
    {
      const double e1 = q[7] * ag, e2 = q[8] * ag, e3 = q[9] * ag;
      const double b1 = Fij(v, 2, 1), b2 = Fij(v, 0, 2), b3 = Fij(v, 1, 0);
      row(5, sqrt(e1 * e1 + e2 * e2 + e3 * e3), sqrt(b1 * b1 + b2 * b2 + b3 * b3));
    }
    {
      double e = 0;
      for (int c = 0; c < 9; ++c) e += 4 * q[10 + c] * q[10 + c];
      row(6, ag * sqrt(e), sqrt(gB2(v)));
    }
    // Gauss U(1)
    {
      double l[3];
      for (int i = 0; i < 3; ++i) l[i] = q[7 + i] - (double)p[(size_t)(7 + i) * n3 + v.mi(i)];
      const double LHS = div_by((l[0] + l[1]) + l[2], a.ddx);
      const double nrm = 2 / dx * a.rfo2;
      const double imc = cmul(conj_(C2<double>{q[1], q[2]}), v.cs(s)).im;
      const double imd = sprod(D2<double>{C2<double>{q[3], q[4]}, C2<double>{q[5], q[6]}}, v.dbl(s)).im;
      const double rho = nrm * a.gC * imc + nrm * a.gD * imd;
      const double RHS = -dx * rho;
      const double L1 = div_by(l[0], a.ddx), L2 = div_by(l[1], a.ddx), L3 = div_by(l[2], a.ddx);
      const double diff = LHS - (RHS + 0.0), sum = L1 * L1 + L2 * L2 + L3 * L3 + (RHS + 0.0) * (RHS + 0.0);
      acc[42] += sqrt(diff * diff);
      acc[43] += sqrt(sum * sum);
      acc[44] += sqrt(RHS * RHS);
      acc[45] += sqrt(LHS * LHS);
    }
    // Gauss SU(2)
    {
      double L[3];
      for (int i = 0; i < 3; ++i) {
        const uint32_t sm = v.mi(i);
        const Q4<double> Ui = v.link(i, sm);
        const size_t pb = (size_t)(10 + 3 * i) * n3 + sm;
        const Q4<double> r =
            qmul(qmul(qdag(Ui), Q4<double>{0, (double)p[pb], (double)p[pb + n3], (double)p[pb + 2 * n3]}), Ui);
        const double rv[3] = {r.x, r.y, r.z};
        for (int b = 0; b < 3; ++b) {
          const double tt = (1 / dx) * (q[10 + 3 * i + b] - rv[b]);
          L[b] = i == 0 ? tt : L[b] + tt;
        }
      }
      const D2<double> D0 = v.dbl(s);
      const D2<double> pd{C2<double>{q[3], q[4]}, C2<double>{q[5], q[6]}};
      for (int b = 0; b < 3; ++b) {
        const double R = (-1.0) * (a.rfo2 / 2 * (a.gS * sprod(isig(b, D0), pd).re));
        const double df = L[b] - R, sm = L[b] + R;
        acc[46 + 4 * b] += sqrt(df * df);
        acc[47 + 4 * b] += sqrt(sm * sm);
        acc[48 + 4 * b] += sqrt(R * R);
        acc[49 + 4 * b] += sqrt(L[b] * L[b]);
      }
    }
  }
  block_reduce<kMeas, 128>(acc, smem);
  if (threadIdx.x == 0)
    for (int k = 0; k < kMeas; ++k) partials[(size_t)blockIdx.x * kMeas + k] = acc[k];
}

// ---- tangent-linear form ---------------------------------------------------------------------------
// The kernels below evolve (state, tangent) pairs: every expression is the plain kernel's, in
// Tan arithmetic, so the state follows the plain evolution bitwise and the tangent is its exact
// derivative along the coupling direction (and the tangent of the start state).

// derivative of pi2s along the momentum tangent dq (sectors [G0, G1) as pi2s)
template <int G0 = 0, int G1 = 5, class R> __device__ __forceinline__ void pi2s_tan(const R *qs, const R *dqs, double out[5])
{
  double q[NP], d[NP];
  for (int c = sector_c0(G0); c < sector_c0(G1); ++c) {
    q[c] = (double)qs[c];
    d[c] = (double)dqs[c];
  }
  if (G0 <= 0 && G1 > 0) out[0] = 2 * (q[0] * d[0]);
  if (G0 <= 1 && G1 > 1) out[1] = 2 * (q[1] * d[1] + q[2] * d[2]);
  if (G0 <= 2 && G1 > 2) out[2] = 2 * (((q[3] * d[3] + q[4] * d[4]) + q[5] * d[5]) + q[6] * d[6]);
  if (G0 <= 3 && G1 > 3) out[3] = 2 * ((q[7] * d[7] + q[8] * d[8]) + q[9] * d[9]);
  if (G1 == 5) {
    double acc = 0;
#pragma unroll
    for (int c = 10; c < NP; ++c) acc += 8 * (q[c] * d[c]);
    out[4] = acc;
  }
}

// Tangent kick sweep: k_kick on (p, dp) with kernels and field sums in Tan<S>; partials
// [block][2 kRed]: the kRed sums of k_kick, then their tangents.
// The parameters are grid constants and the loops over components unrolled, here and in kernels(): the
// compiler otherwise kept a copy of the parameters and the components' arrays in local memory (944 bytes
// a thread in the A part, 80 now; FP32 80^3 391 us per tangent step before, 370 with it).
// SECT as k_kick; the SU(2) part 2 runs here in FP32 only (k_kick_links).
// Resident blocks per SM of the tangent kick parts: four in FP32, in FP64 three, and four for the S
// and phi part and the Phi part.  80^3, us per launch at 2 / 3 / 4 blocks: FP64 S and phi 84 / 77 /
// 58, Phi 122 / 109 / 104, A 142 / 127 / 132, SU(2) 366 / 374 / 371; FP32 tangent step 567 / 509 /
// 569 at 3 / 4 / 5.  The value part stays the plain evolution's bitwise either way.
#ifndef CLB_SU2_TAN_MINB_F64
#define CLB_SU2_TAN_MINB_F64 3
#endif
#ifndef CLB_SU2_TAN_P56_MINB_F64
#define CLB_SU2_TAN_P56_MINB_F64 4
#endif
#ifndef CLB_SU2_TAN_MINB_F32
#define CLB_SU2_TAN_MINB_F32 4
#endif
template <class S, int NK, bool RF, bool RP, int SECT = 0>
__global__ void __launch_bounds__(128, sizeof(S) == 4             ? CLB_SU2_TAN_MINB_F32
                                       : SECT == 5 || SECT == 6 ? CLB_SU2_TAN_P56_MINB_F64
                                                                : CLB_SU2_TAN_MINB_F64)
    k_kick_tan(const S *__restrict__ f, const S *__restrict__ df, S *__restrict__ p, S *__restrict__ dp, const __grid_constant__ Params a,
               const __grid_constant__ Kick kc, const TState *__restrict__ stp, const __grid_constant__ CoupDot cd, double *__restrict__ partials)
{
  using T = Tan<S>;
  constexpr int G0 = sect_g0(SECT), G1 = sect_g1(SECT);                   // sectors [G0, G1)
  constexpr int C0 = sector_c0(G0), C1 = sector_c0(G1);                    // momentum components [C0, C1)
  __shared__ double smem[(128 / 32) * 2 * kRed];
  griddep_wait();
  griddep_launch();
  const Coef<T> C{T(stp->kA), T(stp->kB), T(stp->kB2), T(stp->kG)};
  double acc[2 * kRed];
#pragma unroll
  for (int k = 0; k < 2 * kRed; ++k) acc[k] = 0;
  for_sites(a.N, a.n3, a.order, [&](uint32_t s) {
    const Site<S, T> v = make_site_tan<S>(f, df, a, s, cd);
    S q[NP], dq[NP];
#pragma unroll
    for (int c = C0; c < C1; ++c) {
      q[c] = p[(size_t)c * a.n3 + s];
      dq[c] = dp[(size_t)c * a.n3 + s];
    }
    auto add_pi = [&](int base) {
      double t[5], td[5];
      pi2s<G0, G1>(q, t);
      pi2s_tan<G0, G1>(q, dq, td);
#pragma unroll
      for (int g = G0; g < G1; ++g) {
        acc[base + g] += t[g];
        acc[kRed + base + g] += td[g];
      }
    };
    SiteAvg<T> av;
    if (NK > 0) {
      T K[NP];
      kernels<SECT, RF>(v, C, K, &av);
#pragma unroll
      for (int k = 0; k < NK; ++k) {
#pragma unroll
        for (int c = C0; c < C1; ++c) {
          const double h = kc.h[k][sector(c)];
          q[c] = (S)((double)q[c] + h * (double)K[c].v);
          dq[c] = (S)((double)dq[c] + h * (double)K[c].d);
        }
        if (RP) add_pi(k == 0 ? 0 : 11);
      }
#pragma unroll
      for (int c = C0; c < C1; ++c) {
        p[(size_t)c * a.n3 + s] = q[c];
        dp[(size_t)c * a.n3 + s] = dq[c];
      }
    } else if (RP) {
      add_pi(0);
    }
    if (RF && NK == 0) av = site_avg<SECT>(v);
    if (RF) {
      auto addf = [&](int k, T r) {
        acc[5 + k] += (double)r.v;
        acc[kRed + 5 + k] += (double)r.d;
      };
      if (sect_sphi(SECT)) {
        addf(0, av.g2S);
        addf(1, av.g2C);
      }
      if (sect_dbl(SECT)) addf(2, av.g2D);
      if (sect_u1(SECT)) addf(3, av.b2A);
      if (sect_su2(SECT)) addf(4, av.b2G);
      if (sect_sphi(SECT)) addf(5, av.pot);
    }
  });
  if (RF || RP) {
    block_reduce<2 * kRed, 128>(acc, smem);
    if (threadIdx.x == 0)
#pragma unroll
      for (int k = 0; k < 2 * kRed; ++k) // value and tangent slots alike
        if (sect_owns(SECT, k % kRed)) partials[(size_t)blockIdx.x * 2 * kRed + k] = acc[k];
  }
}

// The SU(2) part of a split kick sweep, plain (T = S) or tangent-linear (T = Tan<S>, FP64): thread
// d * 128 + t takes direction d of the site that thread t of a 128-thread block of k_kick or k_kick_tan
// takes, with the same arithmetic; direction 0 adds up the site's sums in the same order, so partials
// are the same bits.  One thread per site ran 2300 instructions with few loads in flight at 16 warps per
// SM (37 % of issue, DRAM at 30 %); a third of them per thread, in one copy for all directions, needs
// fewer registers: 24 warps in FP64, 36 in FP32.  Whole steps, us: FP64 192^3 3068 against 3512, 95^3 418
// against 466, 128^3 915 against 1046, 48^3 74 against 88; FP32 95^3 284 against 323, 48^3 54.6 against
// 65.3.  Tangent FP64 80^3 734 against 848, 40^3 167 against 212 (with the loops of kernels() unrolled).
// The FP32 tangent form stays with one thread per site: 80^3 370 us against 438 at two blocks per SM
// here and 476 at one.
// WA: with the A component of the same direction, whose currents need the same covariant products, links
// and phases: FP64 192^3 2833 us per step against 3066 with the A part in a sweep of its own, 95^3 390
// against 418; FP32 95^3 267 against 284, 48^3 50.1 against 54.3.
#ifndef CLB_SU2_DIR_MINB_F64
#define CLB_SU2_DIR_MINB_F64 2
#endif
#ifndef CLB_SU2_DIR_MINB_F32
#define CLB_SU2_DIR_MINB_F32 3
#endif
template <class S, class T, bool WA, int NK, bool RF, bool RP>
__global__ void __launch_bounds__(3 * 128, TanTraits<T>::is ? 1 : sizeof(S) == 8 ? CLB_SU2_DIR_MINB_F64 : CLB_SU2_DIR_MINB_F32)
    k_kick_links(const S *__restrict__ f, const S *__restrict__ df, S *__restrict__ p, S *__restrict__ dp, const __grid_constant__ Params a,
                 const __grid_constant__ Kick kc, const SweepState<T> *__restrict__ stp, const __grid_constant__ CoupDot cd, double *__restrict__ partials,
                 const S *__restrict__ ph)
{
  constexpr bool TAN = TanTraits<T>::is;
  constexpr int W = TAN ? 2 : 1;
  __shared__ double smem[(3 * 128 / 32) * 3 * W];
  __shared__ double xe[2][NK][2][128];                        // pi^2 of directions 1 and 2 after each kick
  __shared__ double xd[TAN ? 2 : 1][NK][2][3][TAN ? 128 : 1]; // the terms of its tangent
  // plaq_dev of plaq(1, 0), plaq(2, 0), plaq(2, 1), and its tangent: plain numbers, since a shared array
  // of pairs would be set to zero by every thread at its own time
  __shared__ typename TanTraits<T>::base xw[W][2][3][128];
  static_assert(!(WA && TAN), "the A part of the tangent form has its own sweep");
  __shared__ double xq[2][NK][2][WA ? 128 : 1]; // pi_A^2 of directions 1 and 2 after each kick
  __shared__ S xg[2][4][WA ? 128 : 1];          // the differences d_1 A_0, d_1 A_2, d_2 A_0, d_2 A_1
  const int d = threadIdx.x / 128, t = threadIdx.x % 128;
  const int j1 = d == 0 ? 1 : 0, j2 = d == 2 ? 1 : 2; // the other directions, ascending
  const size_t U = a.oU + (size_t)d * 4 * a.n3, U1 = a.oU + (size_t)j1 * 4 * a.n3, U2 = a.oU + (size_t)j2 * 4 * a.n3;
  const size_t pc = (size_t)(10 + 3 * d) * a.n3;
  const uint32_t N = a.divN.d;
  auto stride = [&](int k) { return k == 0 ? N * N : k == 1 ? N : 1u; };
  const uint32_t sd = stride(d), s1 = stride(j1), s2 = stride(j2);
  griddep_wait();
  griddep_launch();
  const T A = T(stp->kA), G = T(stp->kG);
  const typename TanTraits<T>::base rfo2 = (typename TanTraits<T>::base)a.rfo2;
  double acc[3 * W]; // pi^2 after the first kick, <B^2>, pi^2 after the second; then their tangents
#pragma unroll
  for (int k = 0; k < 3 * W; ++k) acc[k] = 0;
  double accA[3] = {0, 0, 0}; // the same of A
  int buf = 0;
  for_sites_grouped<128>(a.N, a.n3, a.order, t, [&](size_t site, bool in) {
    const uint32_t s = (uint32_t)site;
    Site<S, T> v;
    if constexpr (TAN)
      v = make_site_tan<S>(f, df, a, s, cd);
    else
      v = make_site<S, S>(f, a, s);
    v.ph = ph;
    // as site_offsets, of this thread's three directions
    const uint32_t xy = fast_div(s, a.divN), x = fast_div(xy, a.divN), y = xy - x * N, z = s - xy * N;
    auto next = [&](int k, uint32_t st) { return (k == 0 ? x : k == 1 ? y : z) + 1 == N ? 0u - (N - 1) * st : st; };
    auto prev = [&](int k, uint32_t st) { return (k == 0 ? x : k == 1 ? y : z) == 0 ? (N - 1) * st : 0u - st; };
    const uint32_t op = next(d, sd), o1 = next(j1, s1), o2 = next(j2, s2), m1 = prev(j1, s1), m2 = prev(j2, s2);
    auto at = [&](size_t base, uint32_t r) { return v.quad(base + 4 * (size_t)r); };
    S q[3], dq[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      q[c] = p[pc + c * a.n3 + s];
      if (TAN) dq[c] = dp[pc + c * a.n3 + s];
    }
    const Q4<T> Ud = at(U, s);
    auto plaq = [&](size_t Uj, uint32_t oj) {
      return qmul(qmul(qmul(Ud, at(Uj, s + op)), qdag(at(U, s + oj))), qdag(at(Uj, s)));
    };
    auto plaqBack = [&](size_t Uj, uint32_t mj) {
      return qdag(qmul(qmul(qmul(Ud, qdag(at(Uj, s + op + mj))), qdag(at(U, s + mj))), at(Uj, s + mj)));
    };
    T gr[3], gb[3], dev1, dev2;
    {
      const Q4<T> P = plaq(U1, o1), B = plaqBack(U1, m1);
      gr[0] = P.x, gr[1] = P.y, gr[2] = P.z, dev1 = plaq_dev<S>(P);
      gb[0] = B.x, gb[1] = B.y, gb[2] = B.z;
    }
    {
      const Q4<T> P = plaq(U2, o2), B = plaqBack(U2, m2);
      gr[0] = gr[0] + P.x, gr[1] = gr[1] + P.y, gr[2] = gr[2] + P.z, dev2 = plaq_dev<S>(P);
      gb[0] = gb[0] + B.x, gb[1] = gb[1] + B.y, gb[2] = gb[2] + B.z;
    }
    const T normGrad = su2_ngrad(v) * G, normSrc = recip<T>(a.ddx) * A;
    const D2<T> Dg = v.dbl(s), Wd = dscale(v.phaseD(d, s), qapply(Ud, v.dbl(s + op)));
    double e[NK], ed[NK][3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const T J = rfo2 / 2 * (v.gS * sprod(Wd, isig(c, Dg)).re);
      const T K = -normGrad * (gr[c] - gb[c]) - normSrc * J;
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        const double h = kc.h[k][4];
        if constexpr (TAN) {
          q[c] = (S)((double)q[c] + h * (double)K.v);
          dq[c] = (S)((double)dq[c] + h * (double)K.d);
          ed[k][c] = 8 * ((double)q[c] * (double)dq[c]);
        } else {
          q[c] = (S)((double)q[c] + h * (double)K);
        }
        const double e2 = 4 * ((double)q[c] * (double)q[c]);
        e[k] = c == 0 ? e2 : e[k] + e2;
      }
    }
    if (in)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        p[pc + c * a.n3 + s] = q[c];
        if (TAN) dp[pc + c * a.n3 + s] = dq[c];
      }
    double eA[NK];
    S ga[3];
    if constexpr (WA) { // kernels()' A component of this direction, with the SU(2) part's W and Phi
      const S *Ad = f + fidx(a, 7, 0) + (size_t)d * a.n3;
      S *pA = p + (size_t)(7 + d) * a.n3;
      S qA = pA[s];
      const uint32_t on[3] = {next(0, N * N), next(1, N), next(2, 1)}, om[3] = {prev(0, N * N), prev(1, N), prev(2, 1)};
      const S c = Ad[s];
      S tl[3], grad = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) tl[k] = (Ad[s + on[k]] + Ad[s + om[k]]) - 2 * c;
      const S lap = recip<S>(a.ddx2) * ((tl[0] + tl[1]) + tl[2]);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        ga[j] = v.fd(7 + j, s, s + op);
        const S g1 = v.fd(7 + j, s + om[j], d == j ? s : s + op + om[j]);
        const S tg = div_by(ga[j] - g1, a.ddx);
        grad = j == 0 ? tg : grad + tg;
      }
      const C2<S> wC = cmul(v.phaseC(d, s), v.cs(s + op));
      const S Jc = v.gC * cmul(conj_(wC), v.cs(s)).im;
      const S Jd = v.gD * sprod(Wd, Dg).im;
      const S J = 2 * recip<S>(a.ddx) * rfo2 * (Jc + Jd);
      const S K = G * (lap - grad) - A * J;
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        qA = (S)((double)qA + kc.h[k][3] * (double)K);
        eA[k] = (double)qA * (double)qA;
      }
      if (in) pA[s] = qA;
    }
    if (RP || RF) {
      if (d > 0) {
        if (RP)
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            xe[buf][k][d - 1][t] = e[k];
            if (TAN)
#pragma unroll
              for (int c = 0; c < 3; ++c) xd[buf][k][d - 1][c][t] = ed[k][c];
          }
        auto put_dev = [&](int k, const T &x) {
          if constexpr (TAN) {
            xw[0][buf][k][t] = x.v;
            xw[1][buf][k][t] = x.d;
          } else {
            xw[0][buf][k][t] = x;
          }
        };
        if (RF) put_dev(d - 1, dev1);
        if (RF && d == 2) put_dev(2, dev2);
        if constexpr (WA) {
          if (RP)
#pragma unroll
            for (int k = 0; k < NK; ++k) xq[buf][k][d - 1][t] = eA[k];
          if (RF) {
            xg[buf][2 * d - 2][t] = ga[0];
            xg[buf][2 * d - 1][t] = d == 1 ? ga[2] : ga[1];
          }
        }
      }
      __syncthreads(); // the next site's values go to the other buffer
      if (d == 0 && in) {
        if (RP)
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            acc[2 * k] += (e[k] + xe[buf][k][0][t]) + xe[buf][k][1][t];
            if constexpr (WA) accA[2 * k] += (eA[k] + xq[buf][k][0][t]) + xq[buf][k][1][t];
            if constexpr (TAN) {
              double td = (ed[k][0] + ed[k][1]) + ed[k][2];
#pragma unroll
              for (int m = 0; m < 6; ++m) td += xd[buf][k][m / 3][m % 3][t];
              acc[3 + 2 * k] += td;
            }
          }
        if (RF) {
          auto get_dev = [&](int k) -> T {
            if constexpr (TAN)
              return T(xw[0][buf][k][t], xw[1][buf][k][t]);
            else
              return xw[0][buf][k][t];
          };
          const T dev[3] = {get_dev(0), get_dev(1), get_dev(2)};
          const T b2 = gB2(v, dev);
          if constexpr (WA) { // aB2
            const S f21 = xg[buf][0][t] - ga[1], f31 = xg[buf][2][t] - ga[2], f32 = xg[buf][3][t] - xg[buf][1][t];
            accA[1] += (double)(f21 * f21 + (f31 * f31 + f32 * f32));
          }
          if constexpr (TAN) {
            acc[1] += (double)b2.v;
            acc[4] += (double)b2.d;
          } else {
            acc[1] += (double)b2;
          }
        }
      }
      buf ^= 1;
    }
  });
  if (RF || RP) {
    block_reduce<3 * W, 128>(acc, smem); // direction 0's four warps
    if (threadIdx.x == 0)
#pragma unroll
      for (int w = 0; w < W; ++w) {
        double *row = partials + ((size_t)blockIdx.x * W + w) * kRed;
        row[4] = acc[3 * w];
        row[9] = acc[3 * w + 1];
        row[15] = acc[3 * w + 2];
      }
    if constexpr (WA) {
      __syncthreads();
      block_reduce<3, 128>(accA, smem);
      if (threadIdx.x == 0) {
        double *row = partials + (size_t)blockIdx.x * kRed;
        row[3] = accA[0];
        row[8] = accA[1];
        row[14] = accA[2];
      }
    }
  }
}

// exp of an algebra element with its tangent; the value is qexp's.  d(sin n / n)/dn =
// (n cos n - sin n) / n^2 is taken from its Taylor series below n = 0.1, where the closed form
// cancels.
template <class S> __device__ __forceinline__ Q4<Tan<double>> qexp_tan(Tan<double> p1, Tan<double> p2, Tan<double> p3)
{
  using T = Tan<double>;
  const double n2 = p1.v * p1.v + p2.v * p2.v + p3.v * p3.v;
  if (sizeof(S) == 4 && n2 <= kSmallPhase * kSmallPhase) {
    // d(sin n / n) = ds n dn and d(cos n) = -(sin n / n) n dn, with n dn = p . dp
    const double sn = __fma_rn(n2, sinc_poly(n2), 1.0), cn = __fma_rn(n2, cosm_poly(n2), 1.0);
    const double ndn = (p1.v * p1.d + p2.v * p2.d) + p3.v * p3.d;
    const double sd = -(1.0 / 3 - n2 * (1.0 / 30 - n2 * (1.0 / 840 - n2 * (1.0 / 45360)))) * ndn;
    return Q4<T>{T(cn, -sn * ndn), T(sn * p1.v, sd * p1.v + sn * p1.d), T(sn * p2.v, sd * p2.v + sn * p2.d),
                 T(sn * p3.v, sd * p3.v + sn * p3.d)};
  }
  const double n = sqrt(n2);
  if (n == 0) return Q4<T>{T(1.0), T(0.0, p1.d), T(0.0, p2.d), T(0.0, p3.d)};
  double s1, cn;
  sincos_link(n, &s1, &cn);
  const double sn = s1 / n;
  const double dn = ((p1.v * p1.d + p2.v * p2.d) + p3.v * p3.d) / n;
  double ds;
  if (n < 0.1) {
    const double x = n * n;
    ds = -n * (1.0 / 3 - x * (1.0 / 30 - x * (1.0 / 840 - x / 45360)));
  } else {
    ds = (n * cn - s1) / (n * n);
  }
  const double sd = ds * dn;
  return Q4<T>{T(cn, -s1 * dn), T(sn * p1.v, sd * p1.v + sn * p1.d), T(sn * p2.v, sd * p2.v + sn * p2.d),
               T(sn * p3.v, sd * p3.v + sn * p3.d)};
}

// Tangent drift: k_drift on (f, df) with the drift coefficients' tangents (through aS, and g_SU2 in
// the link step).
template <class S>
__global__ void __launch_bounds__(256)
    k_drift_tan(S *__restrict__ f, S *__restrict__ df, const S *__restrict__ p, const S *__restrict__ dp, Params a,
                double w, int lf, const TState *__restrict__ stp, CoupDot cd)
{
  griddep_wait();
  griddep_launch();
  using T = Tan<double>;
  const double dt = a.dt;
  const T p3 = stp->p3, p1 = stp->p1;
  const T gS(a.gS, cd.v[4]);
  const T cC = lf ? p3 * dt : p3 * dt * w;
  const T cA = lf ? p1 * dt : p1 * w * dt;
  const T cG = lf ? p1 * a.dx * dt * gS : w * p1 * a.dx * dt * gS;
  const double dtw = lf ? dt : dt * w;
  const size_t n3 = a.n3;
  auto ld = [](const S *x, const S *dx, size_t i) { return T((double)x[i], (double)dx[i]); };
  auto put = [](S *x, S *dx, size_t i, T r) {
    x[i] = (S)r.v;
    dx[i] = (S)r.d;
  };
  auto ld4t = [&](size_t i) {
    const V4<S> v = ld4(f + i), d = ld4(df + i);
    V4<T> r;
#pragma unroll
    for (int k = 0; k < 4; ++k) r.v[k] = T((double)v.v[k], (double)d.v[k]);
    return r;
  };
  auto put4 = [&](size_t i, T x, T y, T z, T w) {
    st4(f + i, (S)x.v, (S)y.v, (S)z.v, (S)w.v);
    st4(df + i, (S)x.d, (S)y.d, (S)z.d, (S)w.d);
  };
  for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < n3; s += (size_t)gridDim.x * blockDim.x) {
    put(f, df, s, ld(f, df, s) + p3 * (dtw * ld(p, dp, s)));
#pragma unroll
    for (int c = 1; c < 3; ++c) put(f, df, c * n3 + s, ld(f, df, c * n3 + s) + cC * ld(p, dp, c * n3 + s));
    {
      const size_t fb = fidx(a, 3, s);
      V4<T> d = ld4t(fb);
#pragma unroll
      for (int c = 0; c < 4; ++c) d.v[c] = d.v[c] + cC * ld(p, dp, (3 + c) * n3 + s);
      put4(fb, d.v[0], d.v[1], d.v[2], d.v[3]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const size_t fa = fidx(a, 7 + i, s);
      put(f, df, fa, ld(f, df, fa) + cA * ld(p, dp, (7 + i) * n3 + s) * 1.0);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const size_t pb = (size_t)(10 + 3 * i) * n3 + s, fb = fidx(a, 10 + 4 * i, s);
      const V4<T> q = ld4t(fb);
      const Q4<T> E = qexp_tan<S>(cG * ld(p, dp, pb), cG * ld(p, dp, pb + n3), cG * ld(p, dp, pb + 2 * n3));
      const Q4<T> U = qmul(E, Q4<T>{q.v[0], q.v[1], q.v[2], q.v[3]});
      put4(fb, U.w, U.x, U.y, U.z);
    }
  }
}

// Tangent re-unitarisation (FP32 form): U <- U / |U| on (f, df).
template <class S> __global__ void __launch_bounds__(256) k_unitarize_tan(S *__restrict__ f, S *__restrict__ df, Params a)
{
  using T = Tan<double>;
  const size_t n3 = a.n3;
  for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < 3 * n3; s += (size_t)gridDim.x * blockDim.x) {
    const V4<S> v = ld4(f + a.oU + 4 * s), d = ld4(df + a.oU + 4 * s);
    T q[4], u[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) q[c] = T((double)v.v[c], (double)d.v[c]);
    const T r = 1.0 / sqrt(((q[0] * q[0] + q[1] * q[1]) + q[2] * q[2]) + q[3] * q[3]);
#pragma unroll
    for (int c = 0; c < 4; ++c) u[c] = q[c] * r;
    st4(f + a.oU + 4 * s, (S)u[0].v, (S)u[1].v, (S)u[2].v, (S)u[3].v);
    st4(df + a.oU + 4 * s, (S)u[0].d, (S)u[1].d, (S)u[2].d, (S)u[3].d);
  }
}

// Elements [j0, j0 + n) of a state's FP64 array (component by component, N^3 each) from or to their places
// in a field or momentum buffer.
template <class Fn> __device__ __forceinline__ void for_state(const Params &a, bool field, size_t j0, size_t n, Fn fn)
{
  const size_t step = (size_t)gridDim.x * blockDim.x;
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  size_t c = (j0 + i) / a.n3, s = j0 + i - c * a.n3;
  for (;;) {
    fn(i, field ? fidx(a, (int)c, s) : c * a.n3 + s);
    i += step;
    if (i >= n) return;
    for (s += step; s >= a.n3; s -= a.n3) ++c;
  }
}
template <class S>
__global__ void __launch_bounds__(256)
    k_state_get(const S *__restrict__ src, Params a, bool field, size_t j0, size_t n, double *__restrict__ dst)
{
  for_state(a, field, j0, n, [&](size_t i, size_t at) { dst[i] = (double)src[at]; });
}
template <class S>
__global__ void __launch_bounds__(256)
    k_state_set(const double *__restrict__ src, Params a, bool field, size_t j0, size_t n, S *__restrict__ dst)
{
  for_state(a, field, j0, n, [&](size_t i, size_t at) { dst[at] = (S)src[i]; });
}

} // namespace su2d
} // namespace clb
