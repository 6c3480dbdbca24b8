/* Gravitational-wave spectrum (GravitationalWaves::ComputeSpectrum,
 * source/gravitational_waves.cpp:52-322) and the spectrum binning data
 * (Sledgehamr::ReadSpectrumKs/ReadProj, sledgehamr.cpp:554-615, whose
 * arrays pySledgehamr/Sledgehamr.py:7-27 generates).
 *
 * Pipeline on the device, per call:
 *   1. pack each of the six selected tensor components of time level NEW
 *      into a (pN)^3 real array, zero padded (utils::Fft, fft.h:143-262);
 *   2. unnormalised transforms of the components in pairs (sh_fft.cuh, or
 *      cuFFT Z2Z), the spectra of the halved x index taken from each pair;
 *   3. projection kernel: for every k-cell the TT-projected power
 *        multpl * sum_{ijlm} L_ijlm (Re u_ij Re u_lm + Im u_ij Im u_lm),
 *        L_ijlm = P_il P_jm - 1/2 P_ij P_lm,  P_ij = delta_ij - k_i k_j/|k|^2
 *      with k_i = index_to_k[index] and multpl = 1 for a in {0, pN/2}, else
 *      2, the 81-term sum in an equivalent form, mostly in integers
 *      (gw_project_kernel);
 *   4. deterministic binning: every bin sums its cells in ascending cell
 *      order with a fixed warp tree (bin lists built once per grid size and
 *      cached), then divides by (pN)^6.  Binned mode uses bin
 *      round(|n|); unbinned mode the position of |n|^2 in the sorted list of
 *      unique k^2.
 */
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <functional>
#include <new>

#include "sh_fft.cuh"
#include "sh_gw.h"
#include "sh_gw_bins.h"
#include "sledgehamr_gb300.h"

namespace sh {

std::vector<double> index_to_k_host(int N, int type) {
    std::vector<double> r(N);
    for (int a = 0; a < N; ++a) {
        double nt = (double)a;
        if ((double)a - N > -N / 2.0 - 1) nt -= N;
        const double x = 2. * M_PI / N * nt;
        if (type == 1) r[a] = std::sin(x);
        else if (type == 2) r[a] = (8. * std::sin(x) - std::sin(2. * x)) / 6.;
        else r[a] = (45. * std::sin(x) - 9. * std::sin(2. * x) + std::sin(3. * x)) / 30.;
    }
    return r;
}

namespace {

/* Pack components ca (real part) and cb (imaginary part) of a level buffer
 * (valid cells, any box layout covering [0,N)^3) into the first N^3 block of a
 * zero-initialised complex (pN)^3 array, a block per stage tile.  A tile knows
 * its box and gives a thread its column, so that no cell searches the boxes
 * and divides by their extents: 132 -> 94 us at 256^3 in boxes of 128 (79 for
 * the bytes). */
__global__ void __launch_bounds__(kThreads)
    gw_pack_kernel(const TileDev *__restrict__ tiles, const BoxDev *__restrict__ boxes, int ncomp,
                   int ca, int cb, const double *__restrict__ buf, double2 *__restrict__ dst, int P,
                   int dlo0, int dlo1, int dlo2) {
    const TileDev t = tiles[blockIdx.x];
    const BoxDev b = boxes[t.box];
    const int ty = threadIdx.x / t.nx;
    const int i = t.x0 + ((int)threadIdx.x - ty * t.nx);
    const int j = t.y0 + ty;
    if (ty >= kThreads / t.nx || i > b.hi[0] || j > b.hi[1]) return;
    const int kend = min(t.z0 + t.nz - 1, b.hi[2]);
    const long long gx = b.gdim[0], gxy = gx * b.gdim[1], PP = (long long)P * P;
    const double *s = buf + b.off * ncomp + (i - b.glo[0]) + (long long)(j - b.glo[1]) * gx +
                      (long long)(t.z0 - b.glo[2]) * gxy;
    const double *re = s + ca * b.gvol, *im = s + cb * b.gvol;
    double2 *d = dst + (long long)(t.z0 - dlo2) * PP + (long long)(j - dlo1) * P + (i - dlo0);
    for (int k = t.z0; k <= kend; ++k, re += gxy, im += gxy, d += PP)
        *d = make_double2(__ldg(re), __ldg(im));
}

/* Per k-cell TT power, four times unnormalised; layout ((c*P + b)*H + a).
 *
 * The six real components arrive in pairs, each pair transformed as one
 * complex field Z = u + i u' (a complex-to-complex transform costs what the
 * two real-to-complex ones cost together); with conj Z(-k) the conjugate of
 * the transform's value at -k,
 *     2 U(k) = Z(k) + conj Z(-k),   2 U'(k) = -i (Z(k) - conj Z(-k)),
 * and the factor 2 (4 in the power) is taken out by the bins' scale.
 *
 * The reference sums Lambda_ijlm(k) u_lm conj(u_ij) over i,j,l,m
 * (gravitational_waves.cpp:251-276) with Lambda_ijlm = P_il P_jm -
 * 1/2 P_ij P_lm and P = 1 - k k^T / k^2 (gravitational_waves.h:101-133).  As
 * Lambda is the TT projector this equals |W|^2 - 1/2 |tr W|^2 with
 * W = P U P. */
template <class C>
__device__ __forceinline__ void split_pair(C z, C m, C &u, C &v) {
    u.x = z.x + m.x;
    u.y = z.y - m.y;
    v.x = z.y + m.y;
    v.y = m.x - z.x;
}

/* FP32: W itself, with v = U k, s = k.v and w = v - s/2 k for the unit vector
 * k / |k| (near the Nyquist planes |k| is ~1e-16, and powers of it would
 * leave the range): W = U - k w^T - w k^T, about 100 operations. */
__device__ __forceinline__ float tt_power32(const float2 (&s6)[6], float kx, float ky, float kz) {
    float k[3] = {kx, ky, kz};
    const float rn = rsqrtf(k[0] * k[0] + k[1] * k[1] + k[2] * k[2]);
    k[0] *= rn;
    k[1] *= rn;
    k[2] *= rn;
    const int slot[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    float2 v[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        v[i].x = s6[slot[i][0]].x * k[0] + s6[slot[i][1]].x * k[1] + s6[slot[i][2]].x * k[2];
        v[i].y = s6[slot[i][0]].y * k[0] + s6[slot[i][1]].y * k[1] + s6[slot[i][2]].y * k[2];
    }
    const float sx = k[0] * v[0].x + k[1] * v[1].x + k[2] * v[2].x;
    const float sy = k[0] * v[0].y + k[1] * v[1].y + k[2] * v[2].y;
    const float h = 0.5f;
    float2 w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        w[i].x = v[i].x - h * sx * k[i];
        w[i].y = v[i].y - h * sy * k[i];
    }
    float first = 0, tr_re = 0, tr_im = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = i; j < 3; ++j) {
            const float2 u = s6[slot[i][j]];
            const float re = u.x - (k[i] * w[j].x + w[i].x * k[j]);
            const float im = u.y - (k[i] * w[j].y + w[i].y * k[j]);
            const float wt = i == j ? 1.f : 2.f;
            first += wt * (re * re + im * im);
            if (i == j) {
                tr_re += re;
                tr_im += im;
            }
        }
    return first - 0.5f * (tr_re * tr_re + tr_im * tr_im);
}

/* FP32 transforms (the per-cell value is widened to FP64 for the bin sums). */
__global__ void gw_project32_kernel(const float2 *__restrict__ Z0, const float2 *__restrict__ Z1,
                                    const float2 *__restrict__ Z2,
                                    const float *__restrict__ index_to_k, int P, double *out) {
    const int H = P / 2 + 1;
    const long long n = (long long)H * P * P;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        const int a = (int)(e % H);
        const int b = (int)((e / H) % P);
        const int c = (int)(e / ((long long)H * P));
        if (a == 0 && b == 0 && c == 0) {
            out[e] = 0.;
            continue;
        }
        const long long f = ((long long)c * P + b) * P + a;
        const long long g =
            ((long long)(c ? P - c : 0) * P + (b ? P - b : 0)) * P + (a ? P - a : 0);
        /* twice the transforms of the slots xx xy xz yy yz zz */
        float2 s6[6];
        split_pair(Z0[f], Z0[g], s6[0], s6[1]);
        split_pair(Z1[f], Z1[g], s6[2], s6[3]);
        split_pair(Z2[f], Z2[g], s6[4], s6[5]);
        const float multpl = (a == 0 || a == P / 2) ? 1.f : 2.f;
        out[e] = (double)(multpl * tt_power32(s6, index_to_k[a], index_to_k[b], index_to_k[c]));
    }
}

/* FP64 transforms: the power from the components of U across k.  With e1 and
 * e2 orthonormal and orthogonal to k, a = e1 U e1, b = e2 U e2, c = e1 U e2, it
 * is 1/2 |a - b|^2 + 2 |c|^2.  In the frame turned about z so that k = (rho, 0,
 * kz), e1 = y' and e2 = (kz, 0, -rho) / |k|, and with s = rho^2 / k^2
 *     a - b = s (xx' - zz) + 2 (rho kz / k^2) xz' - (xx' - yy'),
 *     |c|^2 = |kz xy' - rho yz'|^2 / k^2,
 *     (xx' - yy', 2 xy') = (xx - yy, 2 xy) turned by twice the angle of (kx, ky),
 *     (xz', yz') = (xz, yz) turned by that angle,
 *     2 xx' = xx + yy + (xx' - yy')
 * (any frame serves for k along z).
 *
 * As in the transforms (sh_fft.cuh), an FP64 instruction holds an SM for 16
 * clocks per warp, an integer one for a quarter of a clock: a cell's 12 values
 * are taken as integers in units of 2^-kProjBits of the power of two above the
 * largest, the pairs are split, turned and combined in integers with factors
 * of 62 fractional bits, and a - b and k c are rounded to FP64 once; the
 * squares, k^2 and the factors from it stay FP64 (about 20 instructions with
 * the division).  256^3: 1199 us in FP64 in a fixed basis, 1050 in the turned
 * frame (68 FP64 instructions, that pipe 88% busy), 376 in integers (8 blocks
 * per SM; 397 at 5); the bytes alone take 133.  128^3: 156 -> 81 us.
 *
 * Bounds, with |z| <= 2^56: pairs 2^57, xx - yy and 2 xy 2^58, turned 2^58.5,
 * 2 (xx' - zz) 2^59.8, within the 2^60 of a product's operands; a - b below
 * 2^60.  A product's partial sums need |c| + |d| <= 3/2 or c^2 + d^2 <= 1 of
 * its factors: s/2 <= 1/2 beside 2 rho kz / k^2 <= 1, kz and rho scaled below
 * 1/2. */
constexpr int kProjThreads = 128, kProjBits = 56;
using fft::i64;
struct Factor {
    int h, l;
};
/* v 2^-SHIFT in 62 fractional bits, |v 2^-SHIFT| <= 1 but for rounding */
template <int SHIFT>
__device__ __forceinline__ Factor factor(double v) {
    const i64 top = (1ll << 62) - 1;
    const i64 c = min(max(fft::to_units<63>(v, 1023 + SHIFT), -top), top);
    return Factor{fft::part_h(c), fft::part_l(c)};
}
/* x c + y d to the nearest unit (fft::mul) */
__device__ __forceinline__ i64 dot(i64 x, Factor c, i64 y, Factor d) {
    const int xh = (int)(x >> 31), xl = (int)(x & 0x7FFFFFFFll);
    const int yh = (int)(y >> 31), yl = (int)(y & 0x7FFFFFFFll);
    const i64 t =
        (i64)xh * c.l + ((i64)xl * c.h + ((i64)yh * d.l + ((i64)yl * d.h + fft::kRound)));
    return (i64)xh * c.h + ((i64)yh * d.h + (t >> 31));
}
/* v 2^e, v zero or with an exponent that stays in range */
__device__ __forceinline__ double times_pow2(double v, int e) {
    const int hi = __double2hiint(v);
    return (hi & 0x7FF00000) ? __hiloint2double(hi + (e << 20), __double2loint(v)) : 0.;
}

template <int PLANES>
__global__ void __launch_bounds__(kProjThreads, 8)
    gw_project_kernel(const double2 *__restrict__ Z0, const double2 *__restrict__ Z1,
                      const double2 *__restrict__ Z2, const double *__restrict__ index_to_k,
                      int P, double *__restrict__ out) {
    namespace fx = sledgehamr::utils::fixed;
    const int H = P / 2 + 1;
    const int col = blockIdx.x * kProjThreads + threadIdx.x;
    if (col >= H * P) return;
    const int b = col / H, a = col - b * H;
    const double kx = index_to_k[a], ky = index_to_k[b];
    const double kr2 = kx * kx + ky * ky, krho = sqrt(kr2);
    Factor cp{INT32_MAX, INT32_MAX}, sp{0, 0}, msp{0, 0}, c2p = cp, s2p = sp, ms2p = sp;
    if (kr2 != 0.) {
        cp = factor<0>(kx / krho);
        sp = factor<0>(ky / krho);
        msp = factor<0>(-ky / krho);
        const double s2 = 2. * kx * ky / kr2;
        c2p = factor<0>((kx - ky) * (kx + ky) / kr2);
        s2p = factor<0>(s2);
        ms2p = factor<0>(-s2);
    }
    /* half of the cell's weight: 1/2 (1 for a in {0, P/2}, else 2) */
    const double weight = (a == 0 || a == P / 2) ? 0.5 : 1.;
    const long long row = (long long)b * P + a;
    const long long mrow = (long long)(b ? P - b : 0) * P + (a ? P - a : 0);
    const long long plane = (long long)P * P;
    const int c0 = blockIdx.y * PLANES, c1 = min(c0 + PLANES, P);
    for (int c = c0; c < c1; ++c) {
        const long long f = c * plane + row, g = (c ? P - c : 0) * plane + mrow;
        const double2 zf[3] = {Z0[f], Z1[f], Z2[f]}, zg[3] = {Z0[g], Z1[g], Z2[g]};
        const double kc = index_to_k[c];
        int A = fx::kMinAnchor;
#pragma unroll
        for (int p = 0; p < 3; ++p)
            A = max(max(max(A, fx::expo(fx::hi_word(zf[p].x))), fx::expo(fx::hi_word(zf[p].y))),
                    max(fx::expo(fx::hi_word(zg[p].x)), fx::expo(fx::hi_word(zg[p].y))));
        /* twice the transforms of (xx, xy), (xz, yy), (yz, zz): [slot][re, im] */
        i64 u[3][2], v[3][2];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const i64 fr = fft::to_units<kProjBits>(zf[p].x, A);
            const i64 fi = fft::to_units<kProjBits>(zf[p].y, A);
            const i64 gr = fft::to_units<kProjBits>(zg[p].x, A);
            const i64 gi = fft::to_units<kProjBits>(zg[p].y, A);
            u[p][0] = fr + gr;
            u[p][1] = fi - gi;
            v[p][0] = fi + gi;
            v[p][1] = gr - fr;
        }
        /* kz and rho with the larger one in [1/4, 1/2) */
        const int up =
            1021 - max(fx::expo(fx::hi_word(kc)), fx::expo(fx::hi_word(krho)));
        const double kz = times_pow2(kc, up), rho = times_pow2(krho, up);
        const double r2 = rho * rho, w = 1. / (kz * kz + r2);
        const Factor hs = factor<1>(r2 * w), q = factor<-1>(rho * kz * w);
        const Factor fz = factor<0>(kz), fr = factor<0>(-rho);
        double ab[2], cc[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const i64 xx = u[0][r], xy = v[0][r], xz = u[1][r], yy = v[1][r], yz = u[2][r],
                      zz = v[2][r];
            const i64 d = xx - yy, xy2 = 2 * xy;
            const i64 e = dot(d, c2p, xy2, s2p);     /* xx' - yy' */
            const i64 xyt = dot(xy2, c2p, d, ms2p);  /* 2 xy' */
            const i64 xzt = dot(xz, cp, yz, sp);     /* xz' */
            const i64 yzt = dot(yz, cp, xz, msp);    /* yz' */
            const i64 y = xx + yy + e - 2 * zz;      /* 2 (xx' - zz) */
            ab[r] = fx::to_double(dot(y, hs, xzt, q) - e, A - 1022 - kProjBits);
            cc[r] = fx::to_double(dot(xyt, fz, 2 * yzt, fr), A - 1022 - kProjBits);
        }
        double res = weight * ((ab[0] * ab[0] + ab[1] * ab[1]) +
                               w * (cc[0] * cc[0] + cc[1] * cc[1]));
        if (A == 0x7FF) res = fx::from_bits(0x7FF8000000000000ll);
        out[(long long)c * H * P + col] = (col == 0 && c == 0) ? 0. : res;
    }
}

/* A column's angles (divisions by rho and rho^2, and a root) cost about two
 * of its cells: over 16 planes they fade, where that leaves the SMs 1024
 * threads each, otherwise over 4.  Where that is less than two warps per SM
 * the planes follow each other for nothing and a thread takes one: a spectrum
 * of 24^3 takes 71 us against 82, of 40^3 70 against 71.5, of 48^3 83.6 against
 * 81. */
template <int PLANES>
void launch_project_planes(const double2 *Z0, const double2 *Z1, const double2 *Z2,
                           const double *itk, int P, double *out, cudaStream_t stream) {
    const int H = P / 2 + 1;
    const dim3 grid((H * P + kProjThreads - 1) / kProjThreads, (P + PLANES - 1) / PLANES);
    gw_project_kernel<PLANES><<<grid, kProjThreads, 0, stream>>>(Z0, Z1, Z2, itk, P, out);
}
void launch_project(const double2 *Z0, const double2 *Z1, const double2 *Z2, const double *itk,
                    int P, double *out, cudaStream_t stream) {
    const long long cells = (P / 2 + 1LL) * P * P;
    if (cells / 16 >= 152LL * 1024)
        launch_project_planes<16>(Z0, Z1, Z2, itk, P, out, stream);
    else if (cells / 4 >= 152LL * 64)
        launch_project_planes<4>(Z0, Z1, Z2, itk, P, out, stream);
    else
        launch_project_planes<1>(Z0, Z1, Z2, itk, P, out, stream);
}

/* Deterministic sums of the bins' cells, scaled: a block of kBinThreads
 * threads per bin (blocks loop over bins), thread t summing the cells t,
 * t + kBinThreads, ... of the bin in order, then a fixed warp-shuffle and
 * shared-memory tree.  A whole block per bin keeps the 85 K-cell bins of a
 * 384^3 binned spectrum from running on a few hundred warps. */
constexpr int kBinThreads = 256;
__global__ void __launch_bounds__(kBinThreads)
    gw_bin_kernel(const double *val, const long long *bin_off, const int *bin_cells, int nbins,
                  double scale, double *bins) {
    __shared__ double part[kBinThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int bin = blockIdx.x; bin < nbins; bin += gridDim.x) {
        const long long o0 = bin_off[bin], o1 = bin_off[bin + 1];
        double s = 0.;
        for (long long q = o0 + threadIdx.x; q < o1; q += kBinThreads) s += val[bin_cells[q]];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) part[wid] = s;
        __syncthreads();
        if (wid == 0) {
            double t = lane < kBinThreads / 32 ? part[lane] : 0.;
            for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
            if (lane == 0) bins[bin] = t * scale;
        }
        __syncthreads();
    }
}

void launch_bins(const double *vals, const GwBins &g, double scale, double *bins_dev,
                 cudaStream_t stream) {
    const int nb = (int)g.ks.size();
    const int grid = std::max(1, std::min(nb, 152 * 8));
    gw_bin_kernel<<<grid, kBinThreads, 0, stream>>>(vals, g.d_off, g.d_cells, nb, scale,
                                                    bins_dev);
}

/* multpl |F|^2 per k-cell of a scalar field's R2C transform, with
 * |F| = sqrt(re^2 + im^2) as utils::Fft forms it (fft.h:244-250). */
__global__ void scalar_power_kernel(const double2 *F, int P, double *out) {
    const int H = P / 2 + 1;
    const long long n = (long long)H * P * P;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        const int a = (int)(e % H);
        /* the x planes that are their own mirror image count once */
        const double multpl = (a == 0 || 2 * a == P) ? 1. : 2.;
        const double2 z = F[e];
        const double absF = sqrt(__dadd_rn(__dmul_rn(z.x, z.x), __dmul_rn(z.y, z.y)));
        out[e] = multpl * absF * absF;
    }
}

template <class T>
bool upload(T *d, const std::vector<T> &h, cudaStream_t s) {
    return cudaMemcpyAsync(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s) ==
           cudaSuccess;
}
} // namespace

/* Builds (or reuses) the bin lists of a P^3 spectrum. */
void GwCache::prepare(int P, int unbinned, int projection_type, cudaStream_t s) {
    ++clock;
    for (GwBins &b : bins)
        if (b.P == P && b.unbinned == unbinned && b.projection_type == projection_type) {
            b.used = clock;
            cur = &b;
            return;
        }
    if ((int)bins.size() >= kMaxBins) { /* evict the least recently used */
        size_t lru = 0;
        for (size_t q = 1; q < bins.size(); ++q)
            if (bins[q].used < bins[lru].used) lru = q;
        cudaFree(bins[lru].d_off);
        cudaFree(bins[lru].d_cells);
        cudaFree(bins[lru].d_itk);
        cudaFree(bins[lru].d_itk32);
        bins.erase(bins.begin() + lru);
    }
    GwBins g;
    g.P = P;
    g.unbinned = unbinned;
    g.projection_type = projection_type;
    g.used = clock;
    const BinLists lists = bin_lists(P, unbinned != 0);
    g.ks = lists.ks;
    std::vector<double> itk = index_to_k_host(P, projection_type);
    std::vector<float> itk32(itk.begin(), itk.end());
    if (cudaMalloc(&g.d_off, lists.off.size() * sizeof(long long)) != cudaSuccess ||
        cudaMalloc(&g.d_cells, lists.cells.size() * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&g.d_itk, itk.size() * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&g.d_itk32, itk32.size() * sizeof(float)) != cudaSuccess ||
        !upload(g.d_off, lists.off, s) || !upload(g.d_cells, lists.cells, s) ||
        !upload(g.d_itk, itk, s) || !upload(g.d_itk32, itk32, s)) {
        cudaGetLastError();
        cudaFree(g.d_off);
        cudaFree(g.d_cells);
        cudaFree(g.d_itk);
        cudaFree(g.d_itk32);
        throw std::bad_alloc();
    }
    bins.push_back(std::move(g));
    cur = &bins.back();
}

bool GwCache::plan(int P, int kind, cufftHandle *out) {
    ++clock;
    for (Plan &p : plans)
        if (p.P == P && p.kind == kind) {
            p.used = clock;
            *out = p.h;
            return true;
        }
    if ((int)plans.size() >= kMaxPlans) {
        size_t lru = 0;
        for (size_t q = 1; q < plans.size(); ++q)
            if (plans[q].used < plans[lru].used) lru = q;
        cufftDestroy(plans[lru].h);
        plans.erase(plans.begin() + lru);
    }
    Plan p;
    p.P = P;
    p.kind = kind;
    p.used = clock;
    if (cufftCreate(&p.h) != CUFFT_SUCCESS) return false;
    long long n[3] = {P, P, P};
    const long long dist = (long long)P * P * P;
    size_t work = 0;
    const cufftResult r =
        kind == kPlanD2Z
            ? cufftMakePlanMany64(p.h, 3, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_D2Z, 1, &work)
            : cufftMakePlanMany64(p.h, 3, n, nullptr, 1, dist, nullptr, 1, dist,
                                  kind == kPlanZ2Z3 ? CUFFT_Z2Z : CUFFT_C2C, 3, &work);
    if (r != CUFFT_SUCCESS) {
        cufftDestroy(p.h);
        return false;
    }
    plans.push_back(p);
    *out = p.h;
    return true;
}

const fft::Twiddle *GwCache::table(int P, cudaStream_t s) {
    ++clock;
    for (Table &t : tables)
        if (t.P == P) {
            t.used = clock;
            return t.d;
        }
    if ((int)tables.size() >= kMaxPlans) {
        size_t lru = 0;
        for (size_t q = 1; q < tables.size(); ++q)
            if (tables[q].used < tables[lru].used) lru = q;
        cudaFree(tables[lru].d);
        tables.erase(tables.begin() + lru);
    }
    Table t;
    t.P = P;
    t.used = clock;
    t.d = fft::make_table(P, s);
    if (t.d) tables.push_back(t);
    return t.d;
}

void GwCache::release() {
    for (GwBins &b : bins) {
        cudaFree(b.d_off);
        cudaFree(b.d_cells);
        cudaFree(b.d_itk);
        cudaFree(b.d_itk32);
    }
    bins.clear();
    for (Plan &p : plans) cufftDestroy(p.h);
    plans.clear();
    for (Table &t : tables) cudaFree(t.d);
    tables.clear();
    cur = nullptr;
}

cudaError_t gw_spectrum_packed(GwCache &cache, cudaStream_t stream, int P, int N,
                               int projection_type, int unbinned, double *scratch,
                               double *bins_dev, int *nbins, long long *launches,
                               std::string &err,
                               const std::function<void(int, double2 *)> &pack) {
    cache.prepare(P, unbinned, projection_type, stream);
    const long long nfull = (long long)P * P * P;
    /* the library's own transforms at the sizes that they have, cuFFT's
     * otherwise (256^3, three arrays: 10.3 ms with cuFFT, which is bound by
     * the FP64 pipe, 1.6 ms in integers) */
    cufftHandle plan = 0;
    const fft::Twiddle *table = nullptr;
    if (fft::supported(P)) {
        table = cache.table(P, stream);
        if (!table) throw std::bad_alloc();
    } else {
        if (!cache.plan(P, GwCache::kPlanZ2Z3, &plan)) {
            err = "cuFFT plan of three P^3 complex transforms failed";
            return cudaErrorUnknown;
        }
        cufftSetStream(plan, stream);
    }
    /* scratch: three complex P^3 arrays (component pairs) | per-cell values */
    double2 *Z = (double2 *)scratch;
    double *vals = (double *)(Z + 3 * nfull);
    /* the pack covers all of P^3 without zero padding */
    if (P != N) cudaMemsetAsync(Z, 0, 3 * nfull * sizeof(double2), stream);
    for (int p = 0; p < 3; ++p) {
        pack(p, Z + p * nfull);
        (*launches)++;
    }
    if (table) {
        const cudaError_t e = fft::transform3(Z, 3, P, table, stream);
        if (e != cudaSuccess) return e;
        (*launches) += 3;
    } else if (cufftExecZ2Z(plan, (cufftDoubleComplex *)Z, (cufftDoubleComplex *)Z,
                            CUFFT_FORWARD) != CUFFT_SUCCESS) {
        err = "cufftExecZ2Z failed";
        return cudaErrorUnknown;
    }
    launch_project(Z, Z + nfull, Z + 2 * nfull, cache.cur->d_itk, P, vals, stream);
    (*launches)++;
    const int nb = (int)cache.ks().size();
    /* 1/P^6, and 1/4 for the pairs' factor 2 (exact) */
    const double scale = 0.25 / std::pow((double)P, 6);
    launch_bins(vals, *cache.cur, scale, bins_dev, stream);
    (*launches)++;
    *nbins = nb;
    return cudaGetLastError();
}

cudaError_t gw_spectrum_packed32(GwCache &cache, cudaStream_t stream, int P, int N,
                                 int projection_type, int unbinned, double *scratch,
                                 double *bins_dev, int *nbins, long long *launches,
                                 std::string &err,
                                 const std::function<void(int, float2 *)> &pack) {
    cache.prepare(P, unbinned, projection_type, stream);
    const int H = P / 2 + 1;
    const long long nfull = (long long)P * P * P;
    const long long nhalf = (long long)H * P * P;
    cufftHandle plan;
    if (!cache.plan(P, GwCache::kPlanC2C3, &plan)) {
        err = "cuFFT plan of three P^3 FP32 complex transforms failed";
        return cudaErrorUnknown;
    }
    cufftSetStream(plan, stream);
    /* scratch: three complex FP32 P^3 arrays (component pairs) | per-cell values */
    float2 *Z = (float2 *)scratch;
    double *vals = (double *)(Z + 3 * nfull);
    if (P != N) cudaMemsetAsync(Z, 0, 3 * nfull * sizeof(float2), stream);
    for (int p = 0; p < 3; ++p) {
        pack(p, Z + p * nfull);
        (*launches)++;
    }
    if (cufftExecC2C(plan, (cufftComplex *)Z, (cufftComplex *)Z, CUFFT_FORWARD) != CUFFT_SUCCESS) {
        err = "cufftExecC2C failed";
        return cudaErrorUnknown;
    }
    int g = (int)std::min<long long>((nhalf + 255) / 256, 152LL * 32);
    gw_project32_kernel<<<std::max(g, 1), 256, 0, stream>>>(
        Z, Z + nfull, Z + 2 * nfull, cache.cur->d_itk32, P, vals);
    (*launches)++;
    const int nb = (int)cache.ks().size();
    const double scale = 0.25 / std::pow((double)P, 6);
    launch_bins(vals, *cache.cur, scale, bins_dev, stream);
    (*launches)++;
    *nbins = nb;
    return cudaGetLastError();
}

cudaError_t scalar_spectrum_packed(GwCache &cache, cudaStream_t stream, int P, double pre,
                                   double *scratch, double *bins_dev, int *nbins,
                                   long long *launches, std::string &err,
                                   const std::function<void(double *)> &pack) {
    /* unbinned bins of k^2 (the k-map of the entry is not used) */
    cache.prepare(P, 1, 2, stream);
    const int H = P / 2 + 1;
    const long long nreal = (long long)P * P * P;
    const long long ncplx = (long long)H * P * P;
    cufftHandle plan;
    if (!cache.plan(P, GwCache::kPlanD2Z, &plan)) {
        err = "cuFFT plan of a P^3 real-to-complex transform failed";
        return cudaErrorUnknown;
    }
    cufftSetStream(plan, stream);
    double *real = scratch;
    double2 *cplx = (double2 *)(scratch + nreal + nreal % 2); /* 16-byte aligned */
    double *vals = (double *)(cplx + ncplx);
    cudaMemsetAsync(real, 0, nreal * sizeof(double), stream);
    pack(real);
    (*launches)++;
    if (cufftExecD2Z(plan, real, (cufftDoubleComplex *)cplx) != CUFFT_SUCCESS) {
        err = "cufftExecD2Z failed";
        return cudaErrorUnknown;
    }
    int g = (int)std::min<long long>((ncplx + 255) / 256, 152LL * 32);
    scalar_power_kernel<<<std::max(g, 1), 256, 0, stream>>>(cplx, P, vals);
    (*launches)++;
    const int nb = (int)cache.ks().size();
    launch_bins(vals, *cache.cur, pre, bins_dev, stream);
    (*launches)++;
    *nbins = nb;
    return cudaGetLastError();
}

cudaError_t gw_spectrum_device(GwCache &cache, cudaStream_t stream, const TileDev *tiles,
                               int ntiles, const BoxDev *boxes, int ncomp, const double *buf,
                               const int comps[6], int N, const int dlo[3], int zero_padding,
                               int projection_type, int unbinned, double *scratch,
                               double *bins_dev, int *nbins, long long *launches,
                               std::string &err) {
    const int P = N * zero_padding;
    return gw_spectrum_packed(
        cache, stream, P, N, projection_type, unbinned, scratch, bins_dev, nbins, launches, err,
        [&](int p, double2 *dst) {
            gw_pack_kernel<<<ntiles, kThreads, 0, stream>>>(tiles, boxes, ncomp, comps[2 * p],
                                                            comps[2 * p + 1], buf, dst, P, dlo[0],
                                                            dlo[1], dlo[2]);
        });
}

size_t gw_scratch_bytes(int N, int zero_padding) {
    const long long P = (long long)N * zero_padding;
    const long long H = P / 2 + 1;
    /* GW: three complex P^3 arrays + per-cell values; scalar spectra: a real
     * P^3 array + a half-spectrum + per-cell values (smaller) */
    return (size_t)(6 * P * P * P + H * P * P) * sizeof(double);
}

} // namespace sh

extern "C" {

int sh_spectrum_bins(int dim, long long *out, int capacity, int *nbins) {
    if (dim <= 0 || !nbins) return SH_ERR_ARG;
    std::vector<long long> v = sh::unique_k2_host(dim);
    *nbins = (int)v.size();
    if (!out) return SH_OK;
    if ((int)v.size() > capacity) return SH_ERR_ARG;
    std::copy(v.begin(), v.end(), out);
    return SH_OK;
}

int sh_index_to_k(int dim, int projection_type, double *out) {
    if (dim <= 0 || !out || projection_type < 1 || projection_type > 3) return SH_ERR_ARG;
    std::vector<double> v = sh::index_to_k_host(dim, projection_type);
    std::copy(v.begin(), v.end(), out);
    return SH_OK;
}

} /* extern "C" */
