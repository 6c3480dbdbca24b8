/* Host side of the FP64 three-dimensional transforms (sh_fft.h). */
#include "sh_fft.h"

#include <vector>

namespace sh {
namespace fft {

bool supported(int P) {
    static const int sizes[] = {32,  40,  48,  64,  72,  80,  96,  100, 120, 128,
                                144, 160, 192, 200, 240, 256, 288, 320, 384};
    for (int n : sizes)
        if (n == P) return true;
    return false;
}

Twiddle *make_table(int P, cudaStream_t s) {
    std::vector<Twiddle> h(P);
    for (int j = 0; j < P; ++j) h[j] = make_twiddle(j, P);
    Twiddle *d = nullptr;
    if (cudaMalloc(&d, P * sizeof(Twiddle)) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    /* in stream order: a copy on the default stream is not ordered with a
     * non-blocking one, and may end after its call returns */
    if (cudaMemcpyAsync(d, h.data(), P * sizeof(Twiddle), cudaMemcpyHostToDevice, s) !=
        cudaSuccess) {
        cudaGetLastError();
        cudaFree(d);
        return nullptr;
    }
    return d;
}

cudaError_t transform3(double2 *z, int n, int P, const Twiddle *table, cudaStream_t s) {
    const long long lines = (long long)n * P * P;
    for (int axis = 0; axis < 3; ++axis) {
        cudaError_t e = cudaErrorInvalidValue; /* P in none of the files */
        if (!launch_small(P, z, lines, axis, table, s, &e) &&
            !launch_medium(P, z, lines, axis, table, s, &e))
            launch_large(P, z, lines, axis, table, s, &e);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

} // namespace fft
} // namespace sh
