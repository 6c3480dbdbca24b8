/* Transforms of lines with the integer arithmetic of the axis kernel
 * (sh_fft.cuh): reads P and the number of lines from the command line and
 * the lines from stdin (complex FP64), writes their transforms to stdout.
 * A third argument: the fraction bits to take in place of the line's own. */
#include "sh_fft.cuh"

#include <cstdio>
#include <cstdlib>
#include <vector>

using namespace sh::fft;
namespace fx = sledgehamr::utils::fixed;

template <int R1, int R2>
static void line(double *z, int bits) {
    constexpr int P = R1 * R2;
    LinePart parts[R2];
    for (int n2 = 0; n2 < R2; ++n2)
        parts[n2] = line_part<R1>(
            [&](int n, int im) { return fx::hi_word(z[2 * (n2 + R2 * n) + im]); });
    const LineUnit u = line_unit<R1, R2>([&](int n) { return parts[n]; });
    const int A = u.A, F = bits ? bits : u.F;
    std::vector<Cx> s((size_t)P);
    for (int n2 = 0; n2 < R2; ++n2) {
        Cx v[R1];
        for (int n1 = 0; n1 < R1; ++n1) {
            const double *p = z + 2 * (n2 + R2 * n1);
            v[n1] = Cx{to_units(p[0], A, F), to_units(p[1], A, F)};
        }
        dft<R1>(v);
        for (int k1 = 0; k1 < R1; ++k1)
            s[(size_t)k1 * R2 + n2] =
                k1 == 0 ? v[0] : mul(v[k1], make_twiddle((long long)n2 * k1, P));
    }
    for (int k1 = 0; k1 < R1; ++k1) {
        Cx v[R2];
        for (int n2 = 0; n2 < R2; ++n2) v[n2] = s[(size_t)k1 * R2 + n2];
        dft<R2>(v);
        for (int k2 = 0; k2 < R2; ++k2) {
            z[2 * (k1 + R1 * k2)] = from_units(v[k2].x, A, F);
            z[2 * (k1 + R1 * k2) + 1] = from_units(v[k2].y, A, F);
        }
    }
}

typedef void (*Line)(double *, int);
static Line of(int P) {
    switch (P) { /* the radix pairs of sh_fft_{small,medium,large}.cu */
    case 32: return line<8, 4>;
    case 40: return line<8, 5>;
    case 48: return line<8, 6>;
    case 64: return line<8, 8>;
    case 72: return line<12, 6>;
    case 80: return line<10, 8>;
    case 96: return line<12, 8>;
    case 100: return line<10, 10>;
    case 120: return line<12, 10>;
    case 128: return line<16, 8>;
    case 144: return line<12, 12>;
    case 160: return line<16, 10>;
    case 192: return line<16, 12>;
    case 200: return line<20, 10>;
    case 240: return line<20, 12>;
    case 256: return line<16, 16>;
    case 288: return line<24, 12>;
    case 320: return line<16, 20>;
    case 384: return line<16, 24>;
    }
    return nullptr;
}

int main(int argc, char **argv) {
    const int P = argc > 2 ? std::atoi(argv[1]) : 0, n = argc > 2 ? std::atoi(argv[2]) : 0;
    const Line f = of(P);
    if (!f) return 2;
    std::vector<double> z((size_t)2 * P * n);
    if (std::fread(z.data(), sizeof(double), z.size(), stdin) != z.size()) return 3;
    for (int q = 0; q < n; ++q) f(z.data() + (size_t)2 * P * q, argc > 3 ? std::atoi(argv[3]) : 0);
    return std::fwrite(z.data(), sizeof(double), z.size(), stdout) != z.size();
}
