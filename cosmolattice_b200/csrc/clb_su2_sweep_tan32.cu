// clb_su2_sweep_tan32.cu - lphi4SU2U1 tangent-linear kick sweeps in FP32 storage (without FMA contraction).
#include "clb_su2_sweep_impl.cuh"

namespace clb {
template void su2_sweep_tan<float>(clb_handle *h, int nk, bool rf, bool rp, const Kick &kc);
}
