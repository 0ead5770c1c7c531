// clb_su2_sweep_impl.cuh - the kick sweeps' launches (clb_su2_sweep.cuh).
#pragma once

#include "clb_su2_sweep.cuh"

namespace clb {

template <class S> void su2_sweep(clb_handle *h, int nk, bool rf, bool rp, const Kick &kc)
{
  SU2Sector *u = h->su2;
  const int kind = nk == 0 ? K_U1_REDUCE : K_U1_KICK;
  const S *f = static_cast<const S *>(u->f);
  S *p = static_cast<S *>(u->p);
  // kick sweeps run as two halves (sectors S, phi, Phi, A; then SU(2)), three parts (S, phi, Phi; A;
  // SU(2)) or four (S, phi; Phi; A; SU(2)), which hold fewer registers than one sweep over every sector;
  // of three and four the last two run in one launch (k_kick_links); reduction-only sweeps run whole
#define CLB_SU2K1(NK, RF, RP, SECT)                                                                                     \
  CLB_LAUNCH(h, kind,                                                                                                   \
             launch_pdl(k_kick<S, NK, RF, RP, SECT>, dim3(kSU2Blocks), dim3(128), 0, h, f, p, u->prm, kc,       \
                        (const State *)u->d_st, u->d_part, static_cast<const S *>(u->ph)))
#define CLB_SU2KL(WA, NK, RF, RP)                                                                                          \
  CLB_LAUNCH(h, kind,                                                                                                  \
             launch_pdl(k_kick_links<S, S, WA, NK, RF, RP>, dim3(kSU2Blocks), dim3(3 * 128), 0, h, f,              \
                        (const S *)nullptr, p, (S *)nullptr, u->prm, kc, (const State *)u->d_st, CoupDot{}, u->d_part, \
                        static_cast<const S *>(u->ph)))
#define CLB_SU2K(NK, RF, RP)                                                                                            \
  do {                                                                                                                 \
    if constexpr (NK > 0) {                                                                                            \
      if (u->split == 3) {                                                                                             \
        CLB_SU2K1(NK, RF, RP, 5);                                                                                      \
        CLB_SU2K1(NK, RF, RP, 6);                                                                                      \
      } else if (u->split == 2) {                                                                                      \
        CLB_SU2K1(NK, RF, RP, 3);                                                                                      \
      } else if (u->split) {                                                                                           \
        CLB_SU2K1(NK, RF, RP, 1);                                                                                      \
      } else {                                                                                                         \
        CLB_SU2K1(NK, RF, RP, 0);                                                                                      \
      }                                                                                                                \
      if (u->split > 1)                                                                                                \
        CLB_SU2KL(true, NK, RF, RP);                                                                                   \
      else if (u->split)                                                                                               \
        CLB_SU2KL(false, NK, RF, RP);                                                                                  \
    } else {                                                                                                           \
      CLB_SU2K1(NK, RF, RP, 0);                                                                                        \
    }                                                                                                                  \
  } while (0)
  if (nk == 0) {
    if (rf && rp)
      CLB_SU2K(0, true, true);
    else if (rf)
      CLB_SU2K(0, true, false);
    else
      CLB_SU2K(0, false, true);
  } else if (nk == 1) {
    if (rf && rp)
      CLB_SU2K(1, true, true);
    else if (rp)
      CLB_SU2K(1, false, true);
    else
      CLB_SU2K(1, false, false);
  } else {
    if (rf && rp)
      CLB_SU2K(2, true, true);
    else
      CLB_SU2K(2, false, false);
  }
#undef CLB_SU2K
#undef CLB_SU2KL
#undef CLB_SU2K1
}

template <class S> void su2_sweep_tan(clb_handle *h, int nk, bool rf, bool rp, const Kick &kc)
{
  SU2Sector *u = h->su2;
  const int kind = nk == 0 ? K_U1_REDUCE : K_U1_KICK;
  const S *f = static_cast<const S *>(u->f), *df = static_cast<const S *>(u->df);
  S *p = static_cast<S *>(u->p), *dp = static_cast<S *>(u->dp);
#define CLB_SU2T1(NK, RF, RP, SECT)                                                                                     \
  CLB_LAUNCH(h, kind,                                                                                                   \
             launch_pdl(k_kick_tan<S, NK, RF, RP, SECT>, dim3(kSU2Blocks), dim3(128), 0, h, f, df, p, dp,       \
                        u->prm, kc, (const TState *)u->d_tst, u->tan_cd, u->d_tpart))
#define CLB_SU2TL(NK, RF, RP)                                                                                          \
  do {                                                                                                                 \
    if constexpr (sizeof(S) == sizeof(double))                                                                         \
      CLB_LAUNCH(h, kind,                                                                                              \
                 launch_pdl(k_kick_links<S, Tan<S>, false, NK, RF, RP>, dim3(kSU2Blocks), dim3(3 * 128), 0, h, f, df, \
                            p, dp, u->prm, kc, (const TState *)u->d_tst, u->tan_cd, u->d_tpart, (const S *)nullptr));  \
    else                                                                                                               \
      CLB_SU2T1(NK, RF, RP, 2);                                                                                        \
  } while (0)
#define CLB_SU2T(NK, RF, RP)                                                                                            \
  do {                                                                                                                 \
    if constexpr (NK > 0) {                                                                                            \
      if (u->tan_split == 3) {                                                                                         \
        CLB_SU2T1(NK, RF, RP, 5);                                                                                      \
        CLB_SU2T1(NK, RF, RP, 6);                                                                                      \
        CLB_SU2T1(NK, RF, RP, 4);                                                                                      \
      } else if (u->tan_split == 2) {                                                                                  \
        CLB_SU2T1(NK, RF, RP, 3);                                                                                      \
        CLB_SU2T1(NK, RF, RP, 4);                                                                                      \
      } else if (u->tan_split) {                                                                                       \
        CLB_SU2T1(NK, RF, RP, 1);                                                                                      \
      } else {                                                                                                         \
        CLB_SU2T1(NK, RF, RP, 0);                                                                                      \
      }                                                                                                                \
      if (u->tan_split) CLB_SU2TL(NK, RF, RP);                                                                         \
    } else {                                                                                                           \
      CLB_SU2T1(NK, RF, RP, 0);                                                                                        \
    }                                                                                                                  \
  } while (0)
  if (nk == 0) {
    if (rf && rp)
      CLB_SU2T(0, true, true);
    else if (rf)
      CLB_SU2T(0, true, false);
    else
      CLB_SU2T(0, false, true);
  } else if (nk == 1) {
    if (rf && rp)
      CLB_SU2T(1, true, true);
    else if (rp)
      CLB_SU2T(1, false, true);
    else
      CLB_SU2T(1, false, false);
  } else {
    if (rf && rp)
      CLB_SU2T(2, true, true);
    else
      CLB_SU2T(2, false, false);
  }
#undef CLB_SU2T
#undef CLB_SU2TL
#undef CLB_SU2T1
}

} // namespace clb
