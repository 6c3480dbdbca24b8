/* Discrete Fourier transforms of a line of FP64 values in 64-bit integers.
 *
 * On GB300 an FP64 instruction issues at 2 lanes per clock and SM, which
 * bounds an FP64 transform; 32-bit integer adds and 32 x 32 -> 64-bit
 * multiply-adds issue at 64 and 32 lanes or so.  A line's values are
 * therefore written as integers in a unit of the line's own, transformed with
 * integer adds and products with twiddle factors of 62 fractional bits, and
 * rounded to FP64 once at the end.
 *
 * The unit is 2^-F of the power of two above the line's largest value.  Each
 * value and each product is rounded to it, an error of up to half a unit
 * wherever it is made, so F is as large as 64 bits allow for the line at hand
 * (line_unit): no sum on the way exceeds the sum of the line's magnitudes, and
 * a line with few large values gets up to 61 bits below the largest where one
 * of even values gets 52 to 54.  An FP64 transform rounds after every operation
 * to 2^-53 of the values at that point.  Error of a line (2-norm, 32 to 384
 * values; noise, smooth, steep, decaying and localised lines): 0.21 to 0.47 of
 * an FP64 transform's (pocketfft), 3.7e-17 to 9.5e-17; with frac_bits(P) for
 * every line, up to 7 times it.  The unit costs 3 % of a 256^3 spectrum.
 *
 * Bounds, for a line z of P = R1 R2 <= 512 values whose first-stage transforms
 * take R1 values each: the values stay below sum |z| throughout and below the
 * largest sum |z| over R1 of them up to the twiddle products, which need 2^60.5
 * (mul); products with constants need 2^62 and take sums of sqrt(2) times a
 * value.  So sum |z| <= 2^61.5 and the parts' <= 2^60.5 units suffice.  With
 * all values at the largest, frac_bits(P) holds too: P sqrt(2) 2^F < 2^63, and
 * what enters a product then is a partial sum.
 *
 * The functions are plain C++ for host and device.
 */
#ifndef SH_FFT_CUH_
#define SH_FFT_CUH_

#include <cmath>
#include <cstdint>

#include "sh_fixed_stencil.h"

#if defined(__CUDACC__)
#define SH_HD __host__ __device__ __forceinline__
#else
#define SH_HD inline
#endif

namespace sh {
namespace fft {

typedef long long i64;

struct Cx {
    i64 x, y;
};

SH_HD Cx operator+(Cx a, Cx b) { return Cx{a.x + b.x, a.y + b.y}; }
SH_HD Cx operator-(Cx a, Cx b) { return Cx{a.x - b.x, a.y - b.y}; }
/* -i a */
SH_HD Cx mul_mi(Cx a) { return Cx{a.y, -a.x}; }

/* cos(2 pi j / 240) 2^62, the first quarter: 240 is a multiple of every
 * radix below. */
constexpr int kWave = 240;
SH_HD constexpr i64 quarter(int j) {
    constexpr i64 t[kWave / 4 + 1] = {
        4611686018427387904ll, 4610105708808301149ll, 4605365863016315579ll, 4597469729504976441ll,
        4586422719889771737ll, 4572232405239281286ll, 4554908510886344500ll, 4534462909762803052ll,
        4510909614262386453ll, 4484264766637317327ll, 4454546627935218059ll, 4421775565483900917ll,
        4385974038932618941ll, 4347166584859344223ll, 4305379799954623004ll, 4260642322793532497ll,
        4212984814208232069ll, 4162439936274560413ll, 4109042329927080280ll, 4052828591217912280ll,
        3993837246235628775ll, 3932108724701397192ll, 3867685332260468641ll, 3800611221488001879ll,
        3730932361629093763ll, 3658696507093754878ll, 3583953164728422299ll, 3506753559886439970ll,
        3427150601320760278ll, 3345198844922927638ll, 3260954456333195553ll, 3174475172447402319ll,
        3085820261846986643ll, 2995050484179262453ll, 2902228048515791645ll, 2807416570717393844ll,
        2710681029835013083ll, 2612087723576322062ll, 2511704222868584951ll, 2409599325548919089ll,
        2305843009213693952ll, 2200506383259382060ll, 2093661640147730628ll, 1985382005928654379ll,
        1875741690054758654ll, 1764815834521887442ll, 1652680462370552856ll, 1539412425583540600ll,
        1425089352415399811ll, 1309789594189915007ll, 1193592171602022505ll, 1076576720560973279ll,
        958823437611858663ll, 840413024972904254ll, 721426635226200704ll, 601945815699777620ll,
        482052452579138307ll, 361828714786558535ll, 241356997666611639ll, 120719866516515088ll,
        0ll};
    return t[j];
}
/* cos(2 pi j / 240) 2^62 for any j >= 0 */
SH_HD constexpr i64 wave_cos(int j) {
    j %= kWave;
    return j <= 60 ? quarter(j) : (j <= 120 ? -quarter(120 - j)
                                            : (j <= 180 ? -quarter(j - 120) : quarter(240 - j)));
}
SH_HD constexpr i64 wave_sin(int j) { return wave_cos(j + 180); }

/* A factor c in 62 fractional bits, |c| < 1, as c = h 2^-31 + l 2^-62 with
 * 0 <= l < 2^31. */
SH_HD constexpr int part_h(i64 c) { return (int)(c >> 31); }
SH_HD constexpr int part_l(i64 c) { return (int)(c & 0x7FFFFFFFll); }

/* x c to the nearest unit for a constant |c| < 1 and |x| < 2^62: with x =
 * xh 2^31 + xl the product xl cl 2^-62 of the low parts, below one unit, is
 * left out and its mean added with the rounding (half and a quarter unit). */
constexpr i64 kRound = (1ll << 30) + (1ll << 29);
template <i64 C>
SH_HD i64 mulc(i64 x) {
    constexpr int ch = part_h(C), cl = part_l(C);
    const int xh = (int)(x >> 31), xl = (int)(x & 0x7FFFFFFFll);
    const i64 t = (i64)xh * cl + ((i64)xl * ch + kRound);
    return (i64)xh * ch + (t >> 31);
}

/* a times exp(-2 pi i J / 240) */
template <int J>
SH_HD Cx rotate(Cx a) {
    constexpr int j = J % kWave;
    if constexpr (j == 0) {
        return a;
    } else if constexpr (j % 60 == 0) {
        return j == 60 ? mul_mi(a) : (j == 120 ? Cx{-a.x, -a.y} : Cx{-a.y, a.x});
    } else if constexpr (j % 30 == 0) {
        /* odd multiples of 45 degrees: one factor */
        constexpr i64 c = quarter(30);
        const Cx b = j == 30 ? a : (j == 90 ? mul_mi(a)
                                            : (j == 150 ? Cx{-a.x, -a.y} : Cx{-a.y, a.x}));
        return Cx{mulc<c>(b.x + b.y), mulc<c>(b.y - b.x)};
    } else {
        constexpr i64 c = wave_cos(j), s = wave_sin(j);
        return Cx{mulc<c>(a.x) + mulc<s>(a.y), mulc<c>(a.y) - mulc<s>(a.x)};
    }
}

/* A runtime factor exp(-i phi) = c - i s, split as above. */
struct Twiddle {
    int ch, cl, sh, sl;
};
/* exp(-2 pi i j / P): cosl and sinl have 64 significant bits or more. */
inline Twiddle make_twiddle(long long j, int P) {
    const long double th = 2 * acosl(-1.0L) * (long double)(j % P) / P;
    auto split = [](long double x, int &h, int &l) {
        const long double top = ldexpl(1, 62) - 1;
        const long double v = roundl(ldexpl(x, 62));
        const i64 c = (i64)(v > top ? top : (v < -top ? -top : v));
        h = part_h(c);
        l = part_l(c);
        if (h == INT32_MIN) { /* its negative has to be an int too */
            ++h;
            l += INT32_MIN;
        }
    };
    Twiddle w;
    split(cosl(th), w.ch, w.cl);
    split(sinl(th), w.sh, w.sl);
    return w;
}
/* a (c - i s) for |a| <= 2^60.5 (then the four partial products of 2^31 units
 * stay below 2^63: sqrt(2) 2^29.5 2^31 + sqrt(2) 2^31 2^31) */
SH_HD Cx mul(Cx a, Twiddle w) {
    const int xh = (int)(a.x >> 31), xl = (int)(a.x & 0x7FFFFFFFll);
    const int yh = (int)(a.y >> 31), yl = (int)(a.y & 0x7FFFFFFFll);
    const i64 tx = (i64)xh * w.cl + ((i64)xl * w.ch + ((i64)yh * w.sl + ((i64)yl * w.sh + kRound)));
    const i64 ty =
        (i64)yh * w.cl + ((i64)yl * w.ch + ((i64)xh * -w.sl + ((i64)xl * -w.sh + kRound)));
    return Cx{(i64)xh * w.ch + ((i64)yh * w.sh + (tx >> 31)),
              (i64)yh * w.ch + ((i64)xh * -w.sh + (ty >> 31))};
}

/* Forward transforms of R values in place, natural order in and out. */
template <int R>
SH_HD void dft(Cx (&v)[R]);

/* R = A B: B transforms of A values, rotations, A transforms of B values. */
template <int A, int B, int N2, int K1>
SH_HD void rotate_column(Cx (&t)[A]) {
    if constexpr (K1 < A) {
        t[K1] = rotate<(kWave / (A * B)) * N2 * K1>(t[K1]);
        rotate_column<A, B, N2, K1 + 1>(t);
    }
}
template <int A, int B, int N2>
SH_HD void columns(Cx (&v)[A * B]) {
    if constexpr (N2 < B) {
        Cx t[A];
#pragma unroll
        for (int n = 0; n < A; ++n) t[n] = v[n * B + N2];
        dft<A>(t);
        rotate_column<A, B, N2, 1>(t);
#pragma unroll
        for (int n = 0; n < A; ++n) v[n * B + N2] = t[n];
        columns<A, B, N2 + 1>(v);
    }
}
template <int A, int B>
SH_HD void composite(Cx (&v)[A * B]) {
    columns<A, B, 0>(v);
    Cx out[A * B];
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
        Cx t[B];
#pragma unroll
        for (int n = 0; n < B; ++n) t[n] = v[k1 * B + n];
        dft<B>(t);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) out[k1 + A * k2] = t[k2];
    }
#pragma unroll
    for (int k = 0; k < A * B; ++k) v[k] = out[k];
}

template <int R>
SH_HD void dft(Cx (&v)[R]) {
    static_assert(kWave % R == 0, "radix");
    if constexpr (R == 2) {
        const Cx a = v[0];
        v[0] = a + v[1];
        v[1] = a - v[1];
    } else if constexpr (R == 3) {
        constexpr i64 s3 = wave_sin(80);
        const Cx t = v[1] + v[2], d = v[1] - v[2];
        const Cx m{v[0].x - (t.x >> 1), v[0].y - (t.y >> 1)};
        const Cx n{mulc<s3>(d.y), -mulc<s3>(d.x)}; /* -i sin d */
        v[0] = v[0] + t;
        v[1] = m + n;
        v[2] = m - n;
    } else if constexpr (R == 4) {
        const Cx a = v[0] + v[2], b = v[0] - v[2], c = v[1] + v[3], d = mul_mi(v[1] - v[3]);
        v[0] = a + c;
        v[1] = b + d;
        v[2] = a - c;
        v[3] = b - d;
    } else if constexpr (R == 5) {
        constexpr i64 c1 = wave_cos(48), c2 = wave_cos(96), s1 = wave_sin(48), s2 = wave_sin(96);
        const Cx t1 = v[1] + v[4], t2 = v[2] + v[3], t3 = v[1] - v[4], t4 = v[2] - v[3];
        const Cx m1{v[0].x + mulc<c1>(t1.x) + mulc<c2>(t2.x),
                    v[0].y + mulc<c1>(t1.y) + mulc<c2>(t2.y)};
        const Cx m2{v[0].x + mulc<c2>(t1.x) + mulc<c1>(t2.x),
                    v[0].y + mulc<c2>(t1.y) + mulc<c1>(t2.y)};
        const Cx n1 = mul_mi(Cx{mulc<s1>(t3.x) + mulc<s2>(t4.x), mulc<s1>(t3.y) + mulc<s2>(t4.y)});
        const Cx n2 = mul_mi(Cx{mulc<s2>(t3.x) - mulc<s1>(t4.x), mulc<s2>(t3.y) - mulc<s1>(t4.y)});
        v[0] = v[0] + t1 + t2;
        v[1] = m1 + n1;
        v[4] = m1 - n1;
        v[2] = m2 + n2;
        v[3] = m2 - n2;
    } else if constexpr (R == 6) {
        composite<3, 2>(v);
    } else if constexpr (R == 8) {
        composite<4, 2>(v);
    } else if constexpr (R == 10) {
        composite<5, 2>(v);
    } else if constexpr (R == 12) {
        composite<4, 3>(v);
    } else if constexpr (R == 16) {
        composite<4, 4>(v);
    } else if constexpr (R == 20) {
        composite<4, 5>(v);
    } else {
        static_assert(R == 24, "radix");
        composite<8, 3>(v);
    }
}

/* Fraction bits that any line of P values can have. */
constexpr int frac_bits(int P) { return P <= 256 ? 54 : 53; }

/* Of the R1 values of a line that a first-stage transform takes: the largest
 * biased exponent e and an upper bound m of sum |re| + |im| in units of
 * 2^(e - 1042), 2^-20 of the power of two above them. */
struct LinePart {
    int e;
    unsigned m;
};
SH_HD unsigned shift_right(unsigned m, unsigned d) {
#if defined(__CUDA_ARCH__)
    unsigned r;
    asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(m), "r"(d)); /* PTX clamps the count */
    return r;
#else
    return d < 32u ? m >> d : 0u;
#endif
}
/* high(n, im): high word of the real (imaginary) part of value n */
template <int R1, class High>
SH_HD LinePart line_part(High high) {
    namespace fx = sledgehamr::utils::fixed;
    int e = fx::kMinAnchor;
#pragma unroll
    for (int n = 0; n < 2 * R1; ++n) {
        const int x = fx::expo(high(n >> 1, n & 1));
        e = x > e ? x : e;
    }
    unsigned m = 2 * R1; /* what the shifts cut off */
#pragma unroll
    for (int n = 0; n < 2 * R1; ++n) {
        const int hi = high(n >> 1, n & 1);
        m += shift_right(((unsigned)hi & 0xFFFFFu) | 0x100000u, (unsigned)(e + 1 - fx::expo(hi)));
    }
    return LinePart{e, m};
}

/* The unit 2^(A - 1022 - F) of a line of P = R1 R2 values from its R2 parts:
 * sum |z| and the parts' at most 2^61.5 and 2^60.5 of them. */
struct LineUnit {
    int A, F;
};
template <int R1, int R2, class Part>
SH_HD LineUnit line_unit(Part part) {
    int A = 0;
#pragma unroll
    for (int n = 0; n < R2; ++n) {
        const int e = part(n).e;
        A = e > A ? e : A;
    }
    unsigned sum = 0, top = 0;
#pragma unroll
    for (int n = 0; n < R2; ++n) {
        const LinePart p = part(n);
        const unsigned m = shift_right(p.m, (unsigned)(A - p.e)) + 1u;
        sum += m;
        top = m > top ? m : top;
    }
    const unsigned need = sum > 2u * top ? sum : 2u * top;
    /* need 2^(F - 20) <= 2^61.5; sqrt(2) rounded up by 1e-6, which leaves room
     * for the roundings */
    const unsigned long long n = ((unsigned long long)need * 46341ull >> 15) + 1ull;
    const int F = 81 - (63 - sledgehamr::utils::fixed::clz64(n));
    constexpr int least = frac_bits(R1 * R2);
    return LineUnit{A, F > 61 ? 61 : (F > least ? F : least)};
}

/* The value with bits (hi, lo) in units of 2^(A - 1022 - F), F <= 61 and A at
 * least its biased exponent: rounded to nearest (halves away from zero). */
SH_HD i64 to_units(double v, int A, int F) {
    namespace fx = sledgehamr::utils::fixed;
    const int hi = fx::hi_word(v);
    const unsigned long long m = fx::shift_right(fx::significand<10>(hi, fx::lo_word(v)),
                                                 (unsigned)(A + 62 - F - fx::expo(hi)));
    const i64 r = (i64)((m + 1) >> 1); /* m: twice the units */
    return hi < 0 ? -r : r;
}
template <int F>
SH_HD i64 to_units(double v, int A) {
    namespace fx = sledgehamr::utils::fixed;
    const int hi = fx::hi_word(v);
    const unsigned d = (unsigned)(A - fx::expo(hi));
    const unsigned long long m =
        fx::shift_right(fx::significand<F - 52>(hi, fx::lo_word(v)), d); /* twice the units */
    const i64 r = (i64)((m + 1) >> 1);
    return hi < 0 ? -r : r;
}
/* Back to FP64, rounded to nearest, by the conversion instruction: it takes
 * the FP64 pipe for 16 clocks of an SM, but that pipe is idle here while the
 * integer ones bound the transforms (256^3, three arrays, per axis, all with
 * frac_bits(P): 504 us against 568 with the conversion in integers).  to_units
 * by conversions as well makes the FP64 pipe the bound: 600 us. */
SH_HD double from_units(i64 u, int A, int F) {
    namespace fx = sledgehamr::utils::fixed;
    const int pw = A - 1022 - F;
    const long long b = fx::bits((double)u);
    const int e = (int)((b >> 52) & 0x7FF) + pw;
    if (u != 0 && e >= 1 && e <= 2046) return fx::from_bits(b + ((long long)pw << 52));
    return fx::to_double(u, pw);
}
template <int F>
SH_HD double from_units(i64 u, int A) {
    return from_units(u, A, F);
}

} // namespace fft
} // namespace sh

#endif // SH_FFT_CUH_
