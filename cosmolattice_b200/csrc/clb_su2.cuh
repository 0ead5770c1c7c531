// clb_su2.cuh - sm_100a kernels of lphi4SU2U1: real scalar S, complex scalar phi, SU(2) doublet
// Phi, one U(1) and one SU(2) gauge field (models/lphi4SU2U1.h).
//
// Restates, in the reference's operation order (this unit is compiled without FMA contraction so
// plain expressions round where the reference's expression templates round):
//   ScalarSingletKernels::get     evolvers/kernels/scalarsingletkernels.h:30-40
//   ComplexScalarKernels::get     evolvers/kernels/complexscalarkernels.h:28-35
//   SU2DoubletKernels::get        evolvers/kernels/su2doubletkernels.h:28-33
//   U1Kernels::get                evolvers/kernels/u1kernels.h:31-52
//   SU2Kernels::get               evolvers/kernels/su2kernels.h:30-54
//   covariant Laplacians, links   definitions/gaugederivatives.h:48-115
//   currents, charge densities    definitions/mattercurrents.h:27-119
//   averages                      definitions/fieldfunctionals.h:52-223
//   Gauss laws                    definitions/gausslaws.h:34-80
//   energies, scale factor        definitions/energies.h:37-239, scalefactorkernels.h:27-80
// SU(2) representation: a link is a unit quaternion (q0, q) = q0 + i q.sigma; an algebra element
// (pi_1, pi_2, pi_3) = i pi_a sigma_a; exp(i p.sigma) = cos|p| + i sin|p| p/|p|; plaq(U, i, j) =
// U_i(x) U_j(x+i) U_i(x+j)^+ U_j(x)^+; plaqBack(U, i, j) = [U_i(x) U_j(x+i-j)^+ U_i(x-j)^+ U_j(x-j)]^+,
// so sum_j (plaq - plaqBack) is the force of the Wilson term of fieldfunctionals.h:201-209; a
// doublet is (Phi_0 + i Phi_1, Phi_2 + i Phi_3) and scalar_prod(A, B) = A^+ B.
//
// Layout: 22 field and 19 momentum components of N^3 sites (x slowest), FP64 or FP32 (FP32 links are
// re-unitarised every few steps by the host schedule; all volume sums stay FP64).  Fields: S | phi (2) |
// Phi (4) | A_x..A_z | links U_i (4 each, i = x, y, z).  Momenta: S | phi (2) | Phi (4) | A (3) |
// pi_SU2 (3 per direction).  On the device S, phi and A and all momenta are one array per component;
// Phi and each U_i hold a site's four values together (fidx): a kick reads 24 links and 7 Phi per
// site, and a quadruple is one 32-byte (FP64) or 16-byte (FP32) load with one address instead of
// four.  The stored link phases are (cos, sin) pairs per direction and coupling, because a part of the
// kick reads those of one coupling.  With 32-bit site indices and divisions by multiplication
// (FastDiv), ms per step: 192^3 FP64 3.35 against 4.02 with one array per component, 95^3 FP32 0.315
// against 0.357.

#pragma once

#include "clb_internal.cuh"
#include "clb_scalar.cuh"
#include "clb_tangent.cuh"

namespace clb {
namespace su2d {

constexpr int NF = 22, NP = 19;
constexpr int kRed = 16;  // kick-sweep partial slots
constexpr int kMeas = 64; // measurement partial slots

struct Params {
  int N;
  size_t n3;
  double dx, dx2, inv_dx;
  DivBy ddx, ddx2;          // divisions by dx and dx^2
  double ngrad;             // (1/dx)^3 / gS (su2kernels.h:44), in the form's arithmetic below
  float ngrad_f;
  double qG, qH, gC, gD, gS, c4;
  double rfo2, rof2; // (fStar/omegaStar)^2 and its inverse
  double alpha, fm2, dt, inv_n3;
  int order; // site order of the kick sweeps (for_sites)
  FastDiv divN;
  size_t oD, oU; // element offsets of Phi and of the links in the field buffer (fidx)
};

// Elements of the field buffer and the offsets of its quadruples, 32-byte aligned in FP64.
inline size_t field_offsets(size_t n3, size_t &oD, size_t &oU)
{
  oD = (6 * n3 + 3) / 4 * 4;
  oU = oD + 4 * n3;
  return oU + 12 * n3;
}
// Index of field component c at site s.
__host__ __device__ __forceinline__ size_t fidx(const Params &a, int c, size_t s)
{
  return c < 3 ? (size_t)c * a.n3 + s
         : c < 7 ? a.oD + 4 * s + (size_t)(c - 3)
         : c < 10 ? (size_t)(c - 4) * a.n3 + s
                  : a.oU + ((size_t)((c - 10) >> 2) * a.n3 + s) * 4 + (size_t)((c - 10) & 3);
}
// A site's quadruple: p is aligned to four elements.
template <class S> struct V4 {
  S v[4];
};
__device__ __forceinline__ V4<float> ld4(const float *p)
{
  const float4 t = *reinterpret_cast<const float4 *>(p);
  return V4<float>{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ V4<double> ld4(const double *p)
{
  V4<double> r;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(r.v[0]), "=d"(r.v[1]), "=d"(r.v[2]), "=d"(r.v[3])
               : "l"(p));
  return r;
}
// ... from an array that the kernel does not write
__device__ __forceinline__ V4<float> ld4c(const float *p)
{
  const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
  return V4<float>{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ V4<double> ld4c(const double *p)
{
  V4<double> r;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(r.v[0]), "=d"(r.v[1]), "=d"(r.v[2]), "=d"(r.v[3])
      : "l"(p));
  return r;
}
__device__ __forceinline__ void st4(float *p, float a, float b, float c, float d)
{
  *reinterpret_cast<float4 *>(p) = float4{a, b, c, d};
}
__device__ __forceinline__ void st4(double *p, double a, double b, double c, double d)
{
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// Scale factor, the cached averages of the five sectors (S, phi, Phi, A, SU(2)) and the sweep
// coefficients derived from a and aS; T = double, or Tan<double> in the tangent-linear form.
template <class T> struct StateT {
  T aI, aSI, aIM, aDotI, aDotSI, aDotSIM;
  T pi2[5], pi2SI[5], pi2SIM[5];
  T g2S, g2C, g2D, b2A, b2G, potI;
  T g2S_SI, g2C_SI, g2D_SI, b2A_SI, b2G_SI, potSI; // position Verlet: half-step field averages
  T kA, kB, kB2, kG; // pow(aI, 1+alpha), pow(aI, 3+alpha), /2, pow(aI, -1+alpha)
  T kS;              // pow(aI, 2 alpha + 1)
  T p3, p1;          // pow(aSI, alpha-3), pow(aSI, alpha-1); position Verlet: of aI
  int32_t status, pad;
};
using State = StateT<double>;
using TState = StateT<Tan<double>>;
// the state that a kick sweep of arithmetic type T reads
template <class T> using SweepState = typename std::conditional<TanTraits<T>::is, TState, State>::type;

// Applies fn(x.m, y.m) to every floating member m of two scalar states.
template <class A, class B, class Fn> inline void zip_state(StateT<A> &x, const StateT<B> &y, Fn fn)
{
  fn(x.aI, y.aI);
  fn(x.aSI, y.aSI);
  fn(x.aIM, y.aIM);
  fn(x.aDotI, y.aDotI);
  fn(x.aDotSI, y.aDotSI);
  fn(x.aDotSIM, y.aDotSIM);
  for (int g = 0; g < 5; ++g) {
    fn(x.pi2[g], y.pi2[g]);
    fn(x.pi2SI[g], y.pi2SI[g]);
    fn(x.pi2SIM[g], y.pi2SIM[g]);
  }
  fn(x.g2S, y.g2S);
  fn(x.g2C, y.g2C);
  fn(x.g2D, y.g2D);
  fn(x.b2A, y.b2A);
  fn(x.b2G, y.b2G);
  fn(x.potI, y.potI);
  fn(x.g2S_SI, y.g2S_SI);
  fn(x.g2C_SI, y.g2C_SI);
  fn(x.g2D_SI, y.g2D_SI);
  fn(x.b2A_SI, y.b2A_SI);
  fn(x.b2G_SI, y.b2G_SI);
  fn(x.potSI, y.potSI);
  fn(x.kA, y.kA);
  fn(x.kB, y.kB);
  fn(x.kB2, y.kB2);
  fn(x.kG, y.kG);
  fn(x.kS, y.kS);
  fn(x.p3, y.p3);
  fn(x.p1, y.p1);
}

struct Kick {
  double h[2][5]; // kick factors of up to two kicks: S, phi, Phi, A, SU(2)
};

template <class T> __device__ __host__ inline T ipw_h(T x, int n)
{
  if (n < 0) return 1.0 / ipw_h(x, -n);
  T r = x;
  for (int i = 1; i < n; ++i) r = r * x;
  return n == 0 ? T(1.0) : r;
}

// ---- tail: volume sums and the scale-factor update --------------------------------------------
template <class T> struct EnT {
  T ks, gs, kc, gc, kd, gd, ea, ba, eg, bg;
};
using En = EnT<double>;
template <class T> __device__ __host__ inline EnT<T> energies_of(const StateT<T> &s, const Params &p)
{
  const T a6 = ipw_h(s.aI, -6), a2 = ipw_h(s.aI, -2), e4 = 0.5 * p.rof2 * ipw_h(s.aI, -4);
  return EnT<T>{0.5 * s.pi2[0] * a6, 0.5 * s.g2S * a2, s.pi2[1] * a6, s.g2C * a2, s.pi2[2] * a6, s.g2D * a2,
                e4 * s.pi2[3] * 1.0, e4 * s.b2A / 1.0, e4 * s.pi2[4], e4 * s.b2G};
}
template <class T> __device__ __forceinline__ T sf_kernel(const StateT<T> &s, const Params &p)
{
  const double al = p.alpha;
  const EnT<T> E = energies_of(s, p);
  return s.kS / 3.0 * p.fm2 *
         ((((al - 2) * ((E.ks + E.kc) + E.kd) + al * ((E.gs + E.gc) + E.gd)) +
           (al - 1) * ((1.0 * (E.ea + E.ba) + E.eg) + E.bg)) +
          (al + 1) * s.potI);
}
template <class T> __device__ __host__ inline T rho_of(const StateT<T> &s, const Params &p)
{
  const EnT<T> E = energies_of(s, p);
  return ((((((((((E.ks + E.kc) + E.kd) + E.gs) + E.gc) + E.gd) + E.ea) + E.ba) + E.eg) + E.bg) + 0.0) + s.potI;
}

// Tail.  T = double: partials [block][kRed]; T = Tan<double>: [block][2 kRed], the values then their
// tangents.  The sums' grouping is the same in both, so the value part of a tangent run follows
// the plain run.  After the sums one warp holds the state in every lane, and the powers of a are
// formed side by side, one per lane.
constexpr int kTailGroups = 32, kTailThreads = 512;
__device__ __forceinline__ double bcast_t(double r, int l) { return bcast(r, l); }
__device__ __forceinline__ Tan<double> bcast_t(Tan<double> r, int l) { return Tan<double>(bcast(r.v, l), bcast(r.d, l)); }
template <class T>
__global__ void __launch_bounds__(kTailThreads)
    k_tail(const double *__restrict__ partials, TailOp op, StateT<T> *__restrict__ stp, Params p)
{
  constexpr int W = TanTraits<T>::is ? 2 : 1;
  __shared__ double smem[kRed * W * (kTailGroups + 1)];
  griddep_wait();
  griddep_launch();
  // the state is read beside the partials, not after their sum
  constexpr int SW = sizeof(StateT<T>) / sizeof(double);
  static_assert(SW * sizeof(double) == sizeof(StateT<T>), "whole words");
  __shared__ double ss[SW];
  if (threadIdx.x < 32)
    for (int i = threadIdx.x; i < SW; i += 32) ss[i] = reinterpret_cast<const double *>(stp)[i];
  __syncwarp();
  double r[kRed * W];
  for (int k = 0; k < kRed * W; ++k) r[k] = 0;
  if (op.nblocks > 0) rows_reduce<kRed * W, kRed * W, kTailGroups>(partials, op.nblocks, smem, r);
  if (threadIdx.x >= 32) return;
  const int lane = (int)threadIdx.x;
  StateT<T> s = *reinterpret_cast<const StateT<T> *>(ss);
  T v[kRed];
  for (int k = 0; k < kRed; ++k) {
    if constexpr (TanTraits<T>::is)
      v[k] = T(r[k], r[kRed + k]);
    else
      v[k] = r[k];
    v[k] = v[k] * p.inv_n3;
  }
  const double dt = p.dt;
  const uint32_t fl = op.flags;
  auto store_fields = [&]() {
    s.g2S = v[5];
    s.g2C = v[6];
    s.g2D = v[7];
    s.b2A = v[8];
    s.b2G = v[9];
    s.potI = v[10];
  };
  if (fl & T_STORE_ALL) {
    store_fields();
    for (int g = 0; g < 5; ++g) s.pi2[g] = s.pi2SI[g] = v[g];
  }
  auto write_hist = [&]() {
    double *h = op.hist + op.hist_row * kHistCols;
    h[0] = val(s.aI);
    h[1] = val(s.aDotI);
    h[2] = val(s.pi2[2]);
    h[3] = val(s.g2D);
    h[4] = val(s.potI);
  };
  const bool hist = op.hist != nullptr && op.hist_row >= 0 && lane == 0;
  if (fl & T_STORE_FIELDS) store_fields();
  if (hist && (fl & T_HIST_EARLY)) write_hist();
  if (fl & T_STORE_PI2_I)
    for (int g = 0; g < 5; ++g) s.pi2[g] = v[g];
  if (fl & T_STORE_PI2_LF)
    for (int g = 0; g < 5; ++g) {
      s.pi2SIM[g] = s.pi2SI[g];
      s.pi2SI[g] = v[g];
      s.pi2[g] = 0.5 * (s.pi2SIM[g] + s.pi2SI[g]);
    }
  if (fl & T_CORRECT_ADOT) s.aDotI = sqrt(pow(s.aI, 2 * p.alpha + 2) / 3. * p.fm2 * rho_of(s, p));
  // the a-kicks of one tail act with the same averages at the same a
  const T F = fl & kTailSF ? sf_kernel(s, p) : T(0.0);
  if (fl & T_VV_KICK_ONE) s.aDotI = s.aDotSI + (dt / 2) * F * op.w;
  if (hist && !(fl & T_HIST_EARLY)) write_hist();
  if (fl & T_LF_SYNC) s.aDotI = s.aDotSI + dt / 2.0 * F;
  if (fl & T_LF_CTOR) s.aDotSI = s.aDotI - dt / 2.0 * F;
  if (fl & T_LF_KICK) {
    s.aDotSIM = s.aDotSI;
    s.aDotSI += dt * F;
    s.aDotI = (s.aDotSIM + s.aDotSI) / 2.0;
  }
  if (fl & T_LF_DRIFT) {
    s.aIM = s.aI;
    s.aI += dt * s.aDotSI;
    s.aSI = (s.aIM + s.aI) / 2.0;
  }
  if (fl & T_VV_KICK_HALF) s.aDotSI = s.aDotI + (dt / 2) * F * op.w2;
  if (fl & T_STORE_PI2_B)
    for (int g = 0; g < 5; ++g) s.pi2[g] = v[11 + g];
  if (fl & T_VV_DRIFT) {
    s.aIM = s.aI;
    s.aI += dt * s.aDotSI * op.w2;
    s.aSI = (s.aIM + s.aI) / 2.0;
  }
  // PositionVerlet (positionverlet.h:160-163, 207-276), as in the scalar tail; getSI is the
  // scale-factor kernel of the half-step averages at aI
  if (fl & T_PV_STORE_SI) {
    s.g2S_SI = v[5];
    s.g2C_SI = v[6];
    s.g2D_SI = v[7];
    s.b2A_SI = v[8];
    s.b2G_SI = v[9];
    s.potSI = v[10];
  }
  if (fl & T_PV_STORE_PI2)
    for (int g = 0; g < 5; ++g) {
      s.pi2SIM[g] = s.pi2[g]; // pi2AvIM
      s.pi2[g] = v[g];
      s.pi2SI[g] = 0.5 * (s.pi2[g] + s.pi2SIM[g]);
    }
  if (fl & T_PV_KICK) {
    StateT<T> si = s;
    for (int g = 0; g < 5; ++g) si.pi2[g] = s.pi2SI[g];
    si.g2S = s.g2S_SI;
    si.g2C = s.g2C_SI;
    si.g2D = s.g2D_SI;
    si.b2A = s.b2A_SI;
    si.b2G = s.b2G_SI;
    si.potI = s.potSI;
    s.aDotI += dt * sf_kernel(si, p) * op.w;
  }
  if (fl & T_PV_DRIFT_A2) {
    s.aI += dt / 2.0 * s.aDotI * op.w;
    s.aSI = (s.aIM + s.aI) / 2.0;
  }
  if (fl & T_PV_DRIFT_A1) {
    s.aIM = s.aI;
    s.aI += dt / 2.0 * s.aDotI * op.w2;
    s.aSI = s.aI;
  }
  // fixed background: the host's closed-form values (fixedbackgroundexpansion.h:37-45)
  if (fl & T_FB_AIM) s.aIM = s.aI;
  if (fl & T_FB_AI) s.aI = T(op.fa);
  if (fl & T_FB_ASI) s.aSI = T(op.fb);
  if (fl & T_FB_PV_HALF) {
    s.aIM = s.aI;
    s.aI = T(op.fb);
    s.aSI = s.aI;
  }
  if (fl & T_FB_ADOT) s.aDotI = T(op.fb);
  const T ad = (fl & T_PV_MODE) ? ((fl & (T_PV_DRIFT_A1 | T_FB_PV_HALF)) ? s.aIM : s.aI) : s.aSI;
  const double al = p.alpha;
  const double e = lane == 0 ? 1 + al : lane == 1 ? 3 + al : lane == 2 ? -1 + al : lane == 3 ? al - 3
                                                                : lane == 4 ? al - 1 : 2 * al + 1;
  const T pw = pow(lane == 3 || lane == 4 ? ad : s.aI, e);
  s.kA = bcast_t(pw, 0);
  s.kB = bcast_t(pw, 1);
  s.kB2 = s.kB / 2;
  s.kG = bcast_t(pw, 2);
  s.p3 = bcast_t(pw, 3);
  s.p1 = bcast_t(pw, 4);
  s.kS = bcast_t(pw, 5);
  bool ok = finite_(s.aI) && finite_(s.aDotI) && finite_(s.aDotSI) && finite_(s.potI);
  for (int g = 0; g < 5; ++g) ok = ok && finite_(s.pi2[g]);
  if (!ok) s.status = 1;
  if (lane == 0) *stp = s;
}

} // namespace su2d
} // namespace clb

#include "clb_su2_body.cuh"
