/* One axis of a complex FP64 transform, a line of P = R1 R2 values at a time
 * in 64-bit integers (sh_fft.cuh).
 *
 * A block takes kLines lines.  A thread holds R1 values of a line, n = n2 +
 * R2 n1 with its own n2, and transforms them over n1; twiddled, they pass
 * through shared memory to the threads that hold the R2 values n2 of one k1
 * and transform those to k = k1 + R1 k2.  Every value is read and written
 * once.  Along x, neighbouring threads hold neighbouring values of a line;
 * along y and z neighbouring threads hold neighbouring lines, whose values
 * are contiguous.
 */
#ifndef SH_FFT_KERNEL_CUH_
#define SH_FFT_KERNEL_CUH_

#include "sh_fft.h"

namespace sh {
namespace fft {

constexpr int kLines = 16;

template <int R1, int R2>
constexpr int axis_threads() {
    return kLines * (R1 > R2 ? R1 : R2);
}
/* Shared memory [k1][n2][line]: an odd stride between lines of n2 and between
 * k1 keeps the 8-byte accesses of neighbouring n2, k1 and lines apart. */
template <int R2>
constexpr int k1_stride() {
    return R2 * (kLines + 1) | 1;
}
template <int R1, int R2>
constexpr size_t axis_smem() {
    return (size_t)R1 * k1_stride<R2>() * sizeof(Cx);
}

/* Axis 0, 1, 2: x, y, z.  Lines are numbered with x (axis 0: y) fastest. */
template <int R1, int R2>
__global__ void __launch_bounds__(axis_threads<R1, R2>(), axis_threads<R1, R2>() > 256 ? 1 : 2)
    axis_kernel(double2 *__restrict__ z, long long lines, int axis,
                const Twiddle *__restrict__ table) {
    constexpr int P = R1 * R2;
    namespace fx = sledgehamr::utils::fixed;
    extern __shared__ i64 sm[];
    constexpr int S = k1_stride<R2>();
    i64 *const sx = sm, *const sy = sm + R1 * S; /* real and imaginary parts */
    /* the parts of a line that its threads hold, and its unit */
    __shared__ LinePart parts[R2][kLines + 1];
    __shared__ LineUnit unit[kLines];

    const int tid = threadIdx.x;
    const long long l0 = (long long)blockIdx.x * kLines;
    const long long stride = axis == 0 ? 1 : (axis == 1 ? P : (long long)P * P);
    /* first element of line l */
    auto first = [&](long long l) -> long long {
        if (axis == 0) return l * P;
        const long long q = l / P;
        return axis == 1 ? q * P * P + (l - q * P)
                         : (q / P) * P * P * P + (q % P) * P + (l - q * P);
    };
    int line = axis == 0 ? tid / R2 : tid % kLines;
    const int n2 = axis == 0 ? tid % R2 : tid / kLines;
    bool in = line < kLines && n2 < R2 && l0 + line < lines;
    Cx v[R1];
    double2 a[R1];
    if (in) {
        const double2 *const p = z + first(l0 + line) + n2 * stride;
#pragma unroll
        for (int n = 0; n < R1; ++n) a[n] = p[(long long)(n * R2) * stride];
        parts[n2][line] =
            line_part<R1>([&](int n, int im) { return fx::hi_word(im ? a[n].y : a[n].x); });
    }
    __syncthreads();
    if (in) {
        const LineUnit u =
            line_unit<R1, R2>([&](int n) { return parts[n][line]; });
        if (n2 == 0) unit[line] = u;
#pragma unroll
        for (int n = 0; n < R1; ++n)
            v[n] = Cx{to_units(a[n].x, u.A, u.F), to_units(a[n].y, u.A, u.F)};
        dft<R1>(v);
#pragma unroll
        for (int k = 0; k < R1; ++k) {
            const Cx c = k == 0 ? v[0] : mul(v[k], table[n2 * k]);
            sx[k * S + n2 * (kLines + 1) + line] = c.x;
            sy[k * S + n2 * (kLines + 1) + line] = c.y;
        }
    }
    __syncthreads();
    line = axis == 0 ? tid / R1 : tid % kLines;
    const int k1 = axis == 0 ? tid % R1 : tid / kLines;
    in = line < kLines && k1 < R1 && l0 + line < lines;
    if (!in) return;
    Cx w[R2];
#pragma unroll
    for (int n = 0; n < R2; ++n)
        w[n] = Cx{sx[k1 * S + n * (kLines + 1) + line], sy[k1 * S + n * (kLines + 1) + line]};
    dft<R2>(w);
    const int A = unit[line].A, F = unit[line].F;
    double2 *const p = z + first(l0 + line) + k1 * stride;
    const bool finite = A != 0x7FF; /* a line holding NaN or infinity gives NaN */
#pragma unroll
    for (int k = 0; k < R2; ++k) {
        const double nan = fx::from_bits(0x7FF8000000000000ll);
        p[(long long)(k * R1) * stride] =
            finite ? make_double2(from_units(w[k].x, A, F), from_units(w[k].y, A, F))
                   : make_double2(nan, nan);
    }
}

/* A kernel's limit of dynamic shared memory belongs to the device that is
 * current when it is set, and a process may have contexts on several: it is
 * set at every launch that needs more than the 48 KB every device gives. */
template <int R1, int R2>
cudaError_t launch_axis(double2 *z, long long lines, int axis, const Twiddle *table,
                        cudaStream_t s) {
    constexpr size_t smem = axis_smem<R1, R2>();
    if constexpr (smem + (kLines + 1) * (R2 * sizeof(LinePart) + sizeof(LineUnit)) > 48 * 1024) {
        const cudaError_t e =
            cudaFuncSetAttribute(axis_kernel<R1, R2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem);
        if (e != cudaSuccess) return e;
    }
    axis_kernel<R1, R2><<<(int)((lines + kLines - 1) / kLines), axis_threads<R1, R2>(), smem, s>>>(
        z, lines, axis, table);
    return cudaGetLastError();
}

} // namespace fft
} // namespace sh

#endif // SH_FFT_KERNEL_CUH_
