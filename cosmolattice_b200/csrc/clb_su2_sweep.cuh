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
  // (CLB_SU2_SPLIT sets both forms).  The SU(2) part has a thread per site and direction (k_kick_links;
  // the FP32 tangent form one per site), and in the plain form A with it.  su2_create takes four parts in
  // FP64 and three in FP32: ms per VV2 step whole / halves / three / four parts, FP64 192^3 6.19 / 3.09 /
  // 2.85 / 2.82, 256^3 15.7 / 7.76 / 6.97 / 6.86, 96^3 0.660 / 0.380 / 0.369 / 0.364; FP32 192^3 3.32 / 2.00 /
  // 1.95 / 1.98, 256^3 8.50 / 4.87 / 4.64 / 4.72, 95^3 0.383 / 0.246 / 0.253 / 0.252 (48^3 is fastest in
  // halves: 0.061 against 0.065, FP32 0.044 against 0.047).  The tangent-linear sweep takes four parts in
  // both (three / four: FP64 80^3 0.790 / 0.690, 128^3 2.91 / 2.53; FP32 80^3 0.400 / 0.345, 128^3 1.37 /
  // 1.24).  Every form gives the same state to the last bit.
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
