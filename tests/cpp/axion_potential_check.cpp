/* The axion-string rate as the shipped projects form it (stage_constants.h)
 * against long double, beside the equation written out in FP64: root mean
 * square error and mean error of the potential term over string-free cells,
 * |Psi|^2 near 1, at conformal times 0.1 to 300. */
#include "AxionStrings/stage_constants.h"

#include <cmath>
#include <cstdio>
#include <random>

int main() {
    std::mt19937_64 g(7);
    std::normal_distribution<double> gauss;
    std::uniform_real_distribution<double> angle(0., 6.28318530717958648);
    int bad = 0;
    for (double eta : {0.1, 1., 3., 10., 30., 100., 300.})
        for (int k = 0; k < 4; ++k) {
            const double lambda = k == 3 ? 0.7 : 1., c = k == 0 ? 0. : (k == 1 ? 0.56233 : 0.3);
            const sh_axion::StageConstants s = sh_axion::make_constants(eta, lambda, c);
            const int n = 40000;
            long double here2 = 0, here1 = 0, plain2 = 0, plain1 = 0;
            for (int q = 0; q < n; ++q) {
                const double r = 1. + gauss(g) * std::fmin(.3, 1. / eta), th = angle(g);
                const double a = r * std::cos(th), b = r * std::sin(th);
                const long double m = (long double)a * a + (long double)b * b - 1.0L;
                const long double exact =
                    -(long double)a * lambda * ((long double)eta * eta * m + c);
                const long double here =
                    sh_axion::accel(s, a, 0., 0., sh_axion::potential(s, a, b)) - exact;
                const long double plain =
                    -a * (lambda * (eta * eta * (a * a + b * b - 1.) + c)) - exact;
                here2 += here * here;
                plain2 += plain * plain;
                /* the mean along the field, where a wrong constant shows */
                here1 += here * a;
                plain1 += plain * a;
            }
            const double h = std::sqrt((double)(here2 / n)), p = std::sqrt((double)(plain2 / n));
            const double hb = std::fabs((double)(here1 / n)), pb = std::fabs((double)(plain1 / n));
            /* the mean of n errors of size p spreads by p / sqrt(n) */
            if (!(h <= 1.02 * p && hb <= pb + 4. * p / std::sqrt((double)n))) {
                std::printf("eta %g lambda %g c %g: rms %.2e (written out %.2e), mean %.1e (%.1e)\n",
                            eta, lambda, c, h, p, hb, pb);
                ++bad;
            }
        }
    return bad != 0;
}
