// k_weno.cu -- C2: WENO5 momentum advection (drop-in).
#include "fused.cuh"
#include "ops.cuh"

namespace fmf {
namespace op {

// cal_advu_weno5.f:38-255 -- zero the three outputs on the full halo, then the interior by
// the fused step's line kernels (202 -> 58 us at 64x32x32 against one thread per cell in
// the reference's operation order; both within rounding of the exact quotient).
void cal_advu_weno5(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv,
                    const double* u, const double* v, const double* w, double* au, double* av,
                    double* aw) {
  flat(s, g.n, [=] __device__(long t) {
    au[t] = 0.0;
    av[t] = 0.0;
    aw[t] = 0.0;
  });
  double* const adv[3] = {au, av, aw};
  fused::weno5_one(s, g, dxinv, dyinv, dzinv, u, v, w, adv);
}

}  // namespace op
}  // namespace fmf
