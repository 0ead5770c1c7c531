// clb_su2_sweep_f64.cu - lphi4SU2U1 kick sweeps in FP64 storage (without FMA contraction).
#include "clb_su2_sweep_impl.cuh"

namespace clb {
template void su2_sweep<double>(clb_handle *h, int nk, bool rf, bool rp, const Kick &kc);
}
