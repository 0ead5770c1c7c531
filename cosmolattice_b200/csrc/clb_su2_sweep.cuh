// clb_su2_sweep.cuh - the lphi4SU2U1 sector of a handle and the launches of its kick sweeps.  The
// launches are compiled in units of their own, one per storage type and form (clb_su2_sweep_*.cu),
// which the compiler takes side by side.
#pragma once

#include "clb_handle.cuh"
#include "clb_su2.cuh"

namespace clb {

using namespace su2d;

constexpr int kSU2Blocks = 148 * 8; // 128-thread grid-stride sweeps

struct SU2Sector {
  void *f = nullptr, *p = nullptr; // fields (nf elements, fidx) and 19 x N^3 momenta, double (FP64) or float (FP32 form)
  size_t nf = 0;
  bool fp32 = false;
  size_t esz = 8;
  State *d_st = nullptr;
  double *d_part = nullptr, *d_sums = nullptr;
  double *d_stage = nullptr; // FP64 values on their way in or out, stage_n at a time
  size_t stage_n = 0;
  void *ph = nullptr;        // U(1) link phases (6 x N^3 pairs, storage type), kept by the drifts
  // kick sweeps: 0 one sweep, 1 two halves, 2 three parts, 3 four parts (S and phi; Phi; A; SU(2))
  // (CLB_SU2_SPLIT sets both forms).  su2_create takes four parts in FP64 and three in FP32, by
  // timing at 192^3 VV2, when every part still had a thread per site and the fields were one array
  // per component (ms per step): FP64 9.20 whole, 6.53 halves, 5.10 three parts, 4.73 four parts;
  // FP32 4.93, 3.18, 2.90, 2.93.  The tangent-linear sweep takes four parts in both (256^3 VV2, ms
  // per tangent step, three / four parts: FP64 37.9, 31.4; FP32 21.5, 19.5).  The SU(2) part has a
  // thread per site and direction (k_kick_links; the FP32 tangent form one per site), and in the plain
  // form A with it, with which a step takes 2.83 ms at 192^3 FP64.  Every form gives the
  // same state to the last bit.
  int split = 2;
  int tan_split = 3;
  int64_t steps_since_unitarize = 0;
  Params prm{};
  // tangent-linear form: d(state) along the coupling direction tan_cd, active while tangent
  bool tangent = false;
  CoupDot tan_cd{};
  void *df = nullptr, *dp = nullptr;
  TState *d_tst = nullptr;
  double *d_tpart = nullptr, *d_tsums = nullptr;
};

// FP32 form: links re-unitarised every this many steps
constexpr int64_t kUnitarizeEvery = 10;

// The kick sweep (nk kicks, rf / rp: with the field / momentum sums) and its tangent-linear form.
template <class S> void su2_sweep(clb_handle *h, int nk, bool rf, bool rp, const Kick &kc);
template <class S> void su2_sweep_tan(clb_handle *h, int nk, bool rf, bool rp, const Kick &kc);

} // namespace clb
