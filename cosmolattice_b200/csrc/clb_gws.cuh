// clb_gws.cuh - storage of the gravitational-wave sector and the kick and drift kernels that every
// model's GWs share; only the source differs (clb_gws.cu: the scalar singlets; clb_u1.cu: lphi4U1;
// clb_su2.cu: lphi4SU2U1).
//
// u_ij is stored as five components (u_11, u_12, u_13, u_22, u_23; u_33 = -u_11 - u_22, the storage
// gwsprojector.h reads) of N^3 sites each, x slowest.  The kick (GWsKernels::get, gwskernels.h:27-33,
// applied by LeapFrog::kickGWs) is
//   pi_u += h [a^(1+alpha) lapl(u) + a^(1+alpha) 2 Pi],
// with lapl the seven-point Laplacian of each component (gaugederivatives.h:42-46) and Pi the
// traceless part (Pi_11 - tr/3, Pi_12, Pi_13, Pi_22 - tr/3, Pi_23) of the anisotropic tensor
// (PITensor.h:52-57) that the source forms at the site.  The drift (LeapFrog::driftGWs) is
// u += pow(a_SI, alpha - 3) (dt pi_u).  FP64 pins every rounding (Ar<double>, divisions rounded).
#pragma once

#include "clb_internal.cuh"
#include "clb_scalar.cuh"

#include <utility>

namespace clb {

struct GWSector {
  void *u = nullptr, *pi = nullptr;   // 5 x N^3 each, the storage type of the handle's fields
  void *u2 = nullptr, *pi2 = nullptr; // the other pair of the drift-and-kick sweep (null: no memory for it)
  bool fp32 = false;                 // FP32 storage and arithmetic (the handle's FP32 form)
  bool synced = true;                // momenta at integer time (after clb_initialize or a sync)
  double *d_fk = nullptr;            // five in-place D2Z buffers of the spectrum
  void *d_bins = nullptr;            // its bin partials and sums
  size_t bins_bytes = 0;
};

// x / dx: FP64 as the reference's rounded division, FP32 divides.
__device__ __forceinline__ double gw_div(double x, const DivBy &d) { return div_by(x, d); }
__device__ __forceinline__ float gw_div(float x, const DivBy &d) { return x / (float)d.y; }

constexpr int kGWBlocks = 148 * 8;

// Tensor index k of the pair (i, j), i <= j: 00, 01, 02, 11, 12, 22.
__host__ __device__ constexpr int gw_pair_i(int k) { return k < 3 ? 0 : k < 5 ? 1 : 2; }
__host__ __device__ constexpr int gw_pair_j(int k) { return k < 3 ? k : k < 5 ? k - 2 : 2; }

// pi_u += h K(u; a_I) at every site, the source src(s, x, y, z, xp, yp, zp, P) giving the
// anisotropic tensor P at site s = (x, y, z) (xp, yp, zp: its forward neighbours' coordinates);
// kA points at the device copy of pow(a_I, 1 + alpha).  The kick on its own: the first of a call, a sync's,
// and every one of a handle without the second pair of arrays.  It loads its neighbours where they lie, at
// 48 registers; in the form of the sweep below, without its drift, it waits for loads at a quarter of
// the warps (128^3 FP64 117 us against 76; a call per step with GWs 189 us a step against 150, FP32 150
// against 101).
template <class R, class Src>
__global__ void __launch_bounds__(256) k_gw_kick(const R *__restrict__ u, R *__restrict__ piu, int N, double inv_dx2d,
                                                 double hd, const double *__restrict__ kA_ptr, Src src)
{
  using A = Ar<R>;
  const size_t n3 = (size_t)N * N * N;
  const R kA = (R)*kA_ptr, h = (R)hd, inv_dx2 = (R)inv_dx2d, two = R(2), third = R(1.0 / 3.0);
  for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < n3; s += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(s % N), y = (int)((s / N) % N), x = (int)(s / ((size_t)N * N));
    const int xp = x + 1 == N ? 0 : x + 1, xm = x == 0 ? N - 1 : x - 1;
    const int yp = y + 1 == N ? 0 : y + 1, ym = y == 0 ? N - 1 : y - 1;
    const int zp = z + 1 == N ? 0 : z + 1, zm = z == 0 ? N - 1 : z - 1;
    R P[6];
    src(s, x, y, z, xp, yp, zp, P);
    const R tr3 = A::mul(A::add(A::add(P[0], P[3]), P[5]), third);
    const R S[5] = {A::sub(P[0], tr3), P[1], P[2], A::sub(P[3], tr3), P[4]};
    const R kA2 = A::mul(kA, two);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const R *U = u + (size_t)c * n3;
      const R uc = U[s];
      const R tx = A::sub(A::add(U[((size_t)xp * N + y) * N + z], U[((size_t)xm * N + y) * N + z]), A::mul(two, uc));
      const R ty = A::sub(A::add(U[((size_t)x * N + yp) * N + z], U[((size_t)x * N + ym) * N + z]), A::mul(two, uc));
      const R tz = A::sub(A::add(U[((size_t)x * N + y) * N + zp], U[((size_t)x * N + y) * N + zm]), A::mul(two, uc));
      const R lap = A::mul(inv_dx2, A::add(A::add(tx, ty), tz));
      const R K = A::add(A::mul(kA, lap), A::mul(kA2, S[c]));
      piu[(size_t)c * n3 + s] = A::add(piu[(size_t)c * n3 + s], A::mul(h, K));
    }
  }
}

// The GW sweep between two steps: first u += pow(a_SI, alpha - 3) (dt pi_u), then the kick of k_gw_kick on
// the drifted u.  pd points at the device copy of pow(a_SI, alpha - 3), or aSI at a_SI's (from_aSI: the
// position-Verlet tails keep a_SI as the reference does, positionverlet.h:213-235, but their drift
// coefficient is a_I's).
//
// Memory-bound: the drift and the kick act on the same state, so one sweep reads u and pi_u (10 values a
// site) and writes both, where a drift and a kick sweep move 31.  A block marches a 32 x 8 (z, y) tile along
// LX planes.  Each thread loads its site (and one thread in three a cell of the rows and columns next to
// the tile) two planes ahead into registers, drifts the values when their plane comes and shares them
// through shared memory (two planes, so one barrier per plane); the planes before and after stay in
// registers.  (Loads one plane ahead: 145 us at 128^3 FP64; a cp.async ring of raw planes, drifted at each
// read: 130, held by shared-memory reads.)  The neighbouring tiles read the undrifted state, so the sweep
// writes another pair of arrays.  128^3 FP64: 76 us (ncu), against 36 (drift) + 74 (kick); what GWs add to
// a step in the two forms, us: FP64 128^3 84 / 121, 256^3 580 / 944; FP32 128^3 67 / 77, 256^3 456 / 534.
constexpr int kGWTileZ = 32, kGWTileY = 8;
template <class R, class Src>
__global__ void __launch_bounds__(kGWTileZ *kGWTileY, 2)
    k_gw_sweep(const R *__restrict__ u, const R *__restrict__ pi, R *__restrict__ uo, R *__restrict__ po, int N, int LX, double inv_dx2d, double dtd,
               double hd, const double *__restrict__ kA_ptr, const double *__restrict__ pd_ptr,
               const double *__restrict__ aSI, double alpha, int from_aSI, Src src)
{
  using A = Ar<R>;
  constexpr int BZ = kGWTileZ, BY = kGWTileY, ROW = BZ + 2, PL = (BY + 2) * ROW;
  __shared__ R sm[2][5][PL];
  const size_t n3 = (size_t)N * N * N, plane = (size_t)N * N;
  const R kA = (R)*kA_ptr, h = (R)hd, inv_dx2 = (R)inv_dx2d, two = R(2), third = R(1.0 / 3.0), dt = (R)dtd;
  const R pd = from_aSI ? (R)apow(*aSI, alpha - 3) : (R)*pd_ptr;
  const int tz = threadIdx.x % BZ, ty = threadIdx.x / BZ;
  const int z0 = blockIdx.x * BZ, y0 = blockIdx.y * BY, x0 = blockIdx.z * LX, x1 = min(N, x0 + LX);
  const int hz = min(BZ, N - z0), hy = min(BY, N - y0);
  const int z = z0 + tz, y = y0 + ty;
  const bool valid = tz < hz && ty < hy;
  auto wrap = [&](int v) { return v < 0 ? v + N : (v >= N ? v - N : v); };
  // the halo cell of this thread: rows y0 - 1 and y0 + hy (first two warps), columns z0 - 1 and
  // z0 + hz (half of the third)
  int hr = -1, hc = 0;
  if (ty < 2) {
    if (tz < hz) {
      hr = ty == 0 ? 0 : hy + 1;
      hc = tz + 1;
    }
  } else if (ty == 2 && tz < 2 * BY && (tz & (BY - 1)) < hy) {
    hr = (tz & (BY - 1)) + 1;
    hc = tz < BY ? 0 : hz + 1;
  }
  const bool hal = hr >= 0;
  const size_t own = valid ? (size_t)y * N + z : 0;
  const size_t halo = hal ? (size_t)wrap(y0 - 1 + hr) * N + wrap(z0 - 1 + hc) : 0;
  const int cell = (ty + 1) * ROW + tz + 1, hcell = hr * ROW + hc;
  // raw values of one plane: the site's and the halo cell's
  struct Raw {
    R u[5], p[5], hu[5], hp[5];
  };
  auto load = [&](Raw &r, int xp, bool with_halo) {
    const size_t o = (size_t)wrap(xp) * plane;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      if (valid) {
        r.u[c] = u[c * n3 + o + own];
        r.p[c] = pi[c * n3 + o + own];
      }
      if (with_halo && hal) {
        r.hu[c] = u[c * n3 + o + halo];
        r.hp[c] = pi[c * n3 + o + halo];
      }
    }
  };
  auto moved = [&](R v, R p) -> R { return drift_val<R>(v, p, pd, dt); };
  auto share = [&](int b, const R (&v)[5], const Raw &r) {
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      if (valid) sm[b][c][cell] = v[c];
      if (hal) sm[b][c][hcell] = moved(r.hu[c], r.hp[c]);
    }
  };
  Raw raw{};
  R prev[5], cur[5], pc[5];
  load(raw, x0 - 1, false);
#pragma unroll
  for (int c = 0; c < 5; ++c) prev[c] = moved(raw.u[c], raw.p[c]);
  load(raw, x0, true);
#pragma unroll
  for (int c = 0; c < 5; ++c) {
    cur[c] = moved(raw.u[c], raw.p[c]);
    pc[c] = raw.p[c];
  }
  share(0, cur, raw);
  load(raw, x0 + 1, x0 + 1 < x1);
  __syncthreads();
  int b = 0;
  for (int x = x0; x < x1; ++x, b ^= 1) {
    R nxt[5], pn[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      nxt[c] = moved(raw.u[c], raw.p[c]);
      pn[c] = raw.p[c];
    }
    if (x + 1 < x1) {
      share(b ^ 1, nxt, raw);
      load(raw, x + 2, x + 2 < x1); // plane x1 at most: its own sites only
    }
    if (valid) {
      const size_t s = (size_t)x * plane + own;
      R P[6];
      src(s, x, y, z, wrap(x + 1), wrap(y + 1), wrap(z + 1), P);
      const R tr3 = A::mul(A::add(A::add(P[0], P[3]), P[5]), third);
      const R S[5] = {A::sub(P[0], tr3), P[1], P[2], A::sub(P[3], tr3), P[4]};
      const R kA2 = A::mul(kA, two);
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        const R *m = sm[b][c] + cell;
        const R uc = cur[c];
        const R tx = A::sub(A::add(nxt[c], prev[c]), A::mul(two, uc));
        const R tyv = A::sub(A::add(m[ROW], m[-ROW]), A::mul(two, uc));
        const R tzv = A::sub(A::add(m[1], m[-1]), A::mul(two, uc));
        const R lap = A::mul(inv_dx2, A::add(A::add(tx, tyv), tzv));
        const R K = A::add(A::mul(kA, lap), A::mul(kA2, S[c]));
        const size_t i = c * n3 + s;
        uo[i] = uc;
        po[i] = A::add(pc[c], A::mul(h, K));
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      prev[c] = cur[c];
      cur[c] = nxt[c];
      pc[c] = pn[c];
    }
  }
}

// u += pow(a_SI, alpha - 3) (dt pi_u); pd points at the device copy of pow(a_SI, alpha - 3).
template <class R>
__global__ void __launch_bounds__(256) k_gw_drift(R *__restrict__ u, const R *__restrict__ piu, size_t n, double dtd,
                                                  const double *__restrict__ pd_ptr)
{
  const R pd = (R)*pd_ptr, dt = (R)dtd;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    u[i] = drift_val<R>(u[i], piu[i], pd, dt);
}

// The same drift with the coefficient formed here from a_SI (aSI points at the device copy; the
// position-Verlet tails keep a_SI as the reference does, positionverlet.h:213-235, but their drift
// coefficient is a_I's).
template <class R>
__global__ void __launch_bounds__(256) k_gw_drift_a(R *__restrict__ u, const R *__restrict__ piu, size_t n, double dtd,
                                                    const double *__restrict__ aSI, double alpha)
{
  const R pd = (R)apow(*aSI, alpha - 3), dt = (R)dtd;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    u[i] = drift_val<R>(u[i], piu[i], pd, dt);
}

// A GW kick of weight w.
template <class R, class Src>
inline void launch_gw_kick(GWSector *g, int N, double dx, double dt, double w, const double *kA, const Src &src, cudaStream_t stream)
{
  k_gw_kick<R, Src><<<kGWBlocks, 256, 0, stream>>>(static_cast<const R *>(g->u), static_cast<R *>(g->pi), N, 1.0 / (dx * dx),
                                                   w * dt, kA, src);
}

// Whether the sweep pays for a state (u and pi_u) of so many bytes.  Below 37 MB both pairs of it stay in
// the 126 MB of L2, and from 60 MB on the state in place does not either; in between the in-place drift and
// kick find it there and the sweep's two pairs do not fit.  One / two sweeps, us per VV2 step with GWs: FP64
// 64^3 (21 MB) 22.1 / 26.9, 80^3 (41 MB) 39.1 / 37.2, 96^3 (71 MB) 53.8 / 64.0, 128^3 107 / 145, 256^3 695 /
// 1043; FP32 96^3 (35 MB) 40.1 / 43.3, 100^3 (40 MB) 52.5 / 45.9, 112^3 (56 MB) 66.3 / 60.7, 128^3 (84 MB)
// 82.5 / 94.1, 256^3 517 / 604.  (The gauge models' sources hold the sweep up at every size, lphi4U1 128^3
// 498 / 413, so they always take two.)
inline bool gw_sweep_pays(size_t state_bytes) { return state_bytes <= 37500000 || state_bytes > 60000000; }

// The sweep's runs: whole waves of the resident blocks (two per SM) x (the run + 3 planes, a block's start),
// between 4 and 32 planes.  128^3 FP64 107 us a step at this rule's 32 against 113 at 8 (four blocks per SM),
// 96^3 53.8 at 12 against 57.8 at 4, 176^3 261 at 16 against 274 at 32.
inline int gw_run(int N)
{
  const long long tiles = (long long)((N + kGWTileZ - 1) / kGWTileZ) * ((N + kGWTileY - 1) / kGWTileY), slots = 2 * 148;
  int LX = 1;
  long long best = 0;
  for (int l = N < 32 ? N : 32; l >= (N < 4 ? N : 4); --l) {
    const long long cost = (tiles * ((N + l - 1) / l) + slots - 1) / slots * (l + 3);
    if (best == 0 || cost < best) {
      best = cost;
      LX = l;
    }
  }
  return LX;
}

// The drift of a step (launch_gw_drift) and the kick of the next.
template <class R, class Src>
inline void launch_gw_sweep(GWSector *g, int N, double dx, double dt, const double *kA, const double *pd, const double *aSI,
                            double alpha, bool from_aSI, const Src &src, cudaStream_t stream)
{
  const int gz = (N + kGWTileZ - 1) / kGWTileZ, gy = (N + kGWTileY - 1) / kGWTileY;
  const int LX = gw_run(N);
  k_gw_sweep<R, Src><<<dim3(gz, gy, (N + LX - 1) / LX), kGWTileZ * kGWTileY, 0, stream>>>(
      static_cast<const R *>(g->u), static_cast<const R *>(g->pi), static_cast<R *>(g->u2), static_cast<R *>(g->pi2), N, LX,
      1.0 / (dx * dx), dt, dt, kA, pd, aSI, alpha, from_aSI, src);
  std::swap(g->u, g->u2);
  std::swap(g->pi, g->pi2);
}

// Launches the GW drift: with the tails' coefficient pd (VV, leapfrog), or from a_SI (position Verlet).
template <class R>
inline void launch_gw_drift(R *u, const R *piu, size_t n, double dt, const double *pd, const double *aSI, double alpha,
                            bool from_aSI, cudaStream_t stream)
{
  if (from_aSI)
    k_gw_drift_a<R><<<kGWBlocks, 256, 0, stream>>>(u, piu, n, dt, aSI, alpha);
  else
    k_gw_drift<R><<<kGWBlocks, 256, 0, stream>>>(u, piu, n, dt, pd);
}

// The gauge part of the anisotropic tensor (PITensor.h:58-111) at site s, added to P in the
// reference's order: P_ij += 2 Re[D_i phi conj(D_j phi)] (complex scalar), then the U(1) electric
// and magnetic terms -1/a^2/(fStar/omegaStar)^2 pi_A,i pi_A,j and ... B_i B_j.  phi (fr, fi at the
// components' bases) couples to A through the link complexPhase(ndxg A_i) with ndxg = (-dx) gQ;
// D_i phi = (U_i(x) phi(x + i) - phi(x)) / dx (forwardCovGradientCS, gaugederivatives.h:75-78);
// B = (F_23, F_31, F_12) with F(A, i, j) = forwDiff(A_j, i) - forwDiff(A_i, j) (a stated choice of
// TempLat's fieldStrength; the products B_i B_j do not depend on its sign).  first: P holds no
// singlet part yet, so the complex term starts it.
template <class R>
__device__ __forceinline__ void gw_gauge_tensor(const R *__restrict__ phr, const R *__restrict__ phi,
                                                const R *__restrict__ Ax, const R *__restrict__ pAx, size_t n3,
                                                const size_t (&nb)[3], size_t s, const DivBy &ddx, R ndxg, R aI, R rfo2, bool first,
                                                R (&P)[6])
{
  using A = Ar<R>;
  const R fr = phr[s], fi = phi[s];
  R dr[3], di[3], B[3], E[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const R th = A::mul(ndxg, Ax[(size_t)i * n3 + s]);
    R ur, ui;
    sincos_link(th, &ui, &ur);
    const R pr = phr[nb[i]], pm = phi[nb[i]];
    const R wr = A::sub(A::mul(ur, pr), A::mul(ui, pm)), wi = A::add(A::mul(ur, pm), A::mul(ui, pr));
    dr[i] = gw_div(A::sub(wr, fr), ddx);
    di[i] = gw_div(A::sub(wi, fi), ddx);
    E[i] = pAx[(size_t)i * n3 + s];
  }
  // forwDiff(A_j, i)
  auto fdA = [&](int j, int i) { return gw_div(A::sub(Ax[(size_t)j * n3 + nb[i]], Ax[(size_t)j * n3 + s]), ddx); };
  B[0] = A::sub(fdA(2, 1), fdA(1, 2));
  B[1] = A::sub(fdA(0, 2), fdA(2, 0));
  B[2] = A::sub(fdA(1, 0), fdA(0, 1));
  const R pref = (R(-1) / A::mul(aI, aI)) / rfo2;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int i = gw_pair_i(k), j = gw_pair_j(k);
    const R c = A::mul(R(2), A::add(A::mul(dr[i], dr[j]), A::mul(di[i], di[j])));
    const R e = A::mul(A::mul(pref, E[i]), E[j]);
    const R m = A::mul(A::mul(pref, B[i]), B[j]);
    P[k] = A::add(A::add(first ? c : A::add(P[k], c), e), m);
  }
}

} // namespace clb
