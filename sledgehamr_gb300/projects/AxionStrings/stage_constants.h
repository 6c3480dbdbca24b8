/* Per-launch constants of the axion-string equations at conformal time eta,
 *   Pi' = -2 Pi / eta + lap(Psi) - Psi lambda [eta^2 (|Psi|^2 - 1) + c]
 *       = friction Pi + lap(Psi) - Psi (v2 |Psi|^2 + v0),
 * formed on the host for every stage launch and handed over in the last
 * entries of the stage kernel's parameter array, which the kernel reads as
 * constant operands.  Formed in the hook they cost FP64 instructions of the
 * narrow pipe: a division per thread, and two products that the compiler
 * forms again for every cell to save registers (15 FP64 instructions per
 * cell and stage with them, 11 without, on the 128^3 level).  The potential
 * takes three FP64 operations per cell instead of five as written above;
 * v0 = -v2 exactly for c = 0.
 *
 * The entries are written for projects registered with a StageParams function
 * alone, so the hooks read them only in a translation unit that defines
 * SH_STAGE_CONSTANTS and registers its projects that way (the shipped
 * csrc/proj_*.cu).  Everywhere else - a project that calls a shipped Rhs, one
 * registered with SH_DEFINE_PROJECT, a kernel of one's own - they form the
 * constants themselves from the time and the project's parameters.
 */
#ifndef SH_PROJECTS_AXION_STRINGS_STAGE_CONSTANTS_H_
#define SH_PROJECTS_AXION_STRINGS_STAGE_CONSTANTS_H_

#include <sledgehamr.h>

namespace sh_axion {

struct StageConstants {
    double friction, v2, v0;
};

AMREX_GPU_HOST_DEVICE AMREX_FORCE_INLINE StageConstants make_constants(double eta, double lambda,
                                                                       double c) {
    return StageConstants{-2. / eta, lambda * (eta * eta), lambda * (c - eta * eta)};
}

/* first entry of the constants in the parameter array of a stage launch */
constexpr int kFirst = sledgehamr::kStageParams - 3;

inline void store_constants(double *params, double eta, double lambda, double c) {
    const StageConstants s = make_constants(eta, lambda, c);
    params[kFirst] = s.friction;
    params[kFirst + 1] = s.v2;
    params[kFirst + 2] = s.v0;
}

/* The constants inside a hook: those of the launch where it brings them,
 * else formed from the time, lambda and c. */
AMREX_GPU_HOST_DEVICE AMREX_FORCE_INLINE StageConstants constants(const double *params, double eta,
                                                                  double lambda, double c) {
#if defined(__CUDA_ARCH__) && defined(SH_STAGE_CONSTANTS)
    return StageConstants{params[kFirst], params[kFirst + 1], params[kFirst + 2]};
#else
    return make_constants(eta, lambda, c);
#endif
}

/* Pi' of one field component. */
AMREX_GPU_HOST_DEVICE AMREX_FORCE_INLINE double accel(const StageConstants &s, double psi,
                                                      double pi, double lap, double mod2) {
    return s.friction * pi + lap - psi * (s.v2 * mod2 + s.v0);
}

} // namespace sh_axion

#endif
