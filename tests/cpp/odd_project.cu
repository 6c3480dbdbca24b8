/* A user's project of three fields, one of them without a partner: their
 * rates are zero, so that dissipation alone changes them. */
#include <sledgehamr.h>

namespace ThreeFields {

SLEDGEHAMR_ADD_SCALARS(A, B)
SLEDGEHAMR_ADD_CONJUGATE_MOMENTA(C)

AMREX_GPU_DEVICE AMREX_FORCE_INLINE void
Rhs(const amrex::Array4<double> &rhs, const amrex::Array4<const double> &state, const int i,
    const int j, const int k, const int lev, const double time, const double dt,
    const double dx, const double *params) {
    for (int c = 0; c < Scalar::NScalars; ++c) rhs(i, j, k, c) = 0.;
}

SLEDGEHAMR_FINISH_SETUP

} // namespace ThreeFields

#include "sh_stage.cuh"
SH_DEFINE_PROJECT(ThreeFields, ::ThreeFields, false, 1)
