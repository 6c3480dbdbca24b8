/* Radix pairs of the FP64 transforms: 32, 40, 48, 64, 72, 80, 96. */
#include "sh_fft_kernel.cuh"

namespace sh {
namespace fft {

bool launch_small(int P, double2 *z, long long lines, int axis, const Twiddle *table,
                  cudaStream_t s, cudaError_t *e) {
    switch (P) {
    case 32: *e = launch_axis<8, 4>(z, lines, axis, table, s); break;
    case 48: *e = launch_axis<8, 6>(z, lines, axis, table, s); break;
    case 64: *e = launch_axis<8, 8>(z, lines, axis, table, s); break;
    case 80: *e = launch_axis<10, 8>(z, lines, axis, table, s); break;
    case 96: *e = launch_axis<12, 8>(z, lines, axis, table, s); break;
    case 40: *e = launch_axis<8, 5>(z, lines, axis, table, s); break;
    case 72: *e = launch_axis<12, 6>(z, lines, axis, table, s); break;
    default: return false;
    }
    return true;
}

} // namespace fft
} // namespace sh
