/* The axion-string equations at conformal time eta,
 *   Pi' = -2 Pi / eta + lap(Psi) - Psi lambda [eta^2 (|Psi|^2 - 1) + c].
 *
 * -2 / eta and eta^2 are formed on the host for every stage launch and handed
 * over in the last entries of the stage kernel's parameter array, which the
 * kernel reads as constant operands.  Formed in the hook they cost FP64
 * instructions of the narrow pipe: a division per thread, and products that
 * the compiler forms again for every cell to save registers (15 FP64
 * instructions per cell and stage with them, 12 without, on the 128^3 level).
 * |Psi|^2 - 1 is one sum, Psi1^2 + (Psi2^2 - 1), so that near the vacuum the
 * bracket errs no more than the equation written out, at late times half as
 * much.  Two constants
 * lambda eta^2 and lambda (c - eta^2) save one instruction (the 128^3 level
 * steps 4 % faster), but the second one's rounding error is of the size of
 * eta^2 and the same in every cell: up to twice the error of the rest.
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
    double friction, eta2, lambda, c;
};

AMREX_GPU_HOST_DEVICE AMREX_FORCE_INLINE StageConstants make_constants(double eta, double lambda,
                                                                       double c) {
    return StageConstants{-2. / eta, eta * eta, lambda, c};
}

/* first entry of the constants in the parameter array of a stage launch */
constexpr int kFirst = sledgehamr::kStageParams - 2;

inline void store_constants(double *params, double eta) {
    const StageConstants s = make_constants(eta, 1., 0.);
    params[kFirst] = s.friction;
    params[kFirst + 1] = s.eta2;
}

/* The constants inside a hook: those of the launch where it brings them,
 * else formed from the time. */
AMREX_GPU_HOST_DEVICE AMREX_FORCE_INLINE StageConstants constants(const double *params, double eta,
                                                                  double lambda, double c) {
#if defined(__CUDA_ARCH__) && defined(SH_STAGE_CONSTANTS)
    return StageConstants{params[kFirst], params[kFirst + 1], lambda, c};
#else
    return make_constants(eta, lambda, c);
#endif
}

/* lambda [eta^2 (|Psi|^2 - 1) + c] */
AMREX_GPU_HOST_DEVICE AMREX_FORCE_INLINE double potential(const StageConstants &s, double psi1,
                                                          double psi2) {
    return s.lambda * (s.eta2 * (psi1 * psi1 + (psi2 * psi2 - 1.)) + s.c);
}

/* Pi' of one field component. */
AMREX_GPU_HOST_DEVICE AMREX_FORCE_INLINE double accel(const StageConstants &s, double psi,
                                                      double pi, double lap, double v) {
    return s.friction * pi + lap - psi * v;
}

} // namespace sh_axion

#endif
