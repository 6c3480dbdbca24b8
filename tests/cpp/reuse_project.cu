/* A user's project built on a shipped one: the Rhs of AxionStringsLap1 with
 * a term of its own (params[2] times the momenta), registered with the plain
 * macro; compiled and linked by tests/test_gpu_user_projects.py. */
#include <sledgehamr.h>

#include "AxionStringsLap/AxionStringsLap.h"

namespace DrivenStrings {

SLEDGEHAMR_ADD_SCALARS(Psi1, Psi2)
SLEDGEHAMR_ADD_CONJUGATE_MOMENTA(Pi1, Pi2)

AMREX_GPU_DEVICE AMREX_FORCE_INLINE void
Rhs(const amrex::Array4<double> &rhs, const amrex::Array4<const double> &state, const int i,
    const int j, const int k, const int lev, const double time, const double dt,
    const double dx, const double *params) {
    AxionStringsLap1::Rhs(rhs, state, i, j, k, lev, time, dt, dx, params);
    for (int c = Scalar::Pi1; c <= Scalar::Pi2; ++c)
        rhs(i, j, k, c) += params[2] * state(i, j, k, c);
}

SLEDGEHAMR_FINISH_SETUP

} // namespace DrivenStrings

#include "sh_stage.cuh"
SH_DEFINE_PROJECT(DrivenStrings, ::DrivenStrings, false, 1)
