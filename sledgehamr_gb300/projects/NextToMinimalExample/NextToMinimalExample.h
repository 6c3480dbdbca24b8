/* NextToMinimalExample project: the MinimalExample equations with the
 * potential term scaled by lambda = params[0], which the project class hands
 * to the kernels through SetParamsRhs.
 * Reference: projects/NextToMinimalExample/NextToMinimalExample.h:11-43, :82-85.
 */
#ifndef SH_PROJECTS_NEXT_TO_MINIMAL_EXAMPLE_H_
#define SH_PROJECTS_NEXT_TO_MINIMAL_EXAMPLE_H_

#include <sledgehamr.h>

#include "../AxionStrings/stage_constants.h"

namespace NextToMinimalExample {

SLEDGEHAMR_ADD_SCALARS(Psi1, Psi2)
SLEDGEHAMR_ADD_CONJUGATE_MOMENTA(Pi1, Pi2)

AMREX_GPU_DEVICE AMREX_FORCE_INLINE void
Rhs(const amrex::Array4<double> &rhs, const amrex::Array4<const double> &state, const int i,
    const int j, const int k, const int lev, const double time, const double dt,
    const double dx, const double *params) {
    const sh_axion::StageConstants s = sh_axion::constants(params, time, params[0], 0.56233);
    const double psi1 = state(i, j, k, Scalar::Psi1), psi2 = state(i, j, k, Scalar::Psi2);
    const double pi1 = state(i, j, k, Scalar::Pi1), pi2 = state(i, j, k, Scalar::Pi2);
    const double v = sh_axion::potential(s, psi1, psi2);
    const double lap1 = sledgehamr::utils::Laplacian<2>(state, i, j, k, Scalar::Psi1, dx * dx);
    const double lap2 = sledgehamr::utils::Laplacian<2>(state, i, j, k, Scalar::Psi2, dx * dx);
    rhs(i, j, k, Scalar::Psi1) = pi1;
    rhs(i, j, k, Scalar::Psi2) = pi2;
    rhs(i, j, k, Scalar::Pi1) = sh_axion::accel(s, psi1, pi1, lap1, v);
    rhs(i, j, k, Scalar::Pi2) = sh_axion::accel(s, psi2, pi2, lap2, v);
}

inline void StageParams(double *params, const double time) {
    sh_axion::store_constants(params, time);
}

SLEDGEHAMR_FINISH_SETUP

class NextToMinimalExample : public sledgehamr::Sledgehamr {
  public:
    SLEDGEHAMR_INITIALIZE_PROJECT(NextToMinimalExample)
    void SetParamsRhs(std::vector<double> &params, const double time,
                      const int lev) override {
        params.push_back(lambda);
    }
    double lambda = 1.;
};

} // namespace NextToMinimalExample

#endif
