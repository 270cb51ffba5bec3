// The step size from the mesh minima of getdelt_lag's two limits
// (getdelt_lag, Getrhslag.f90:20705-20709; getsolvdg_lag, :1766-1773).
#pragma once
#include "lag2d_device.cuh"

namespace lag2d {

__host__ __device__ __forceinline__ void dt_apply(const Dev &d, double mcfl, double mvol, int ndt) {
  Scalars *S = d.sc_dev;
  double dt = S->dtfix;
  if (ndt == 1) {
    double dtcfl = fmin(1e10, mcfl), dtvol = fmin(1e10, mvol);
    if (S->itime == 1) dt = fmin(d.cfl * dtcfl, 0.1 * dtvol);
    else dt = fmin(fmin(d.cfl * dtcfl, 0.1 * dtvol), 1.01 * dt);
    if ((S->tacru + dt) > d.tend) dt = d.tend - S->tacru;
  }
  S->dtfix = dt;
  S->tacru = S->tacru + dt;
}

}  // namespace lag2d
