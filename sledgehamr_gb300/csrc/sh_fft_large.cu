/* Radix pairs of the FP64 transforms: 192, 200, 240, 256, 288, 320, 384. */
#include "sh_fft_kernel.cuh"

namespace sh {
namespace fft {

bool launch_large(int P, double2 *z, long long lines, int axis, const Twiddle *table,
                  cudaStream_t s, cudaError_t *e) {
    switch (P) {
    case 192: *e = launch_axis<16, 12>(z, lines, axis, table, s); break;
    case 256: *e = launch_axis<16, 16>(z, lines, axis, table, s); break;
    case 320: *e = launch_axis<16, 20>(z, lines, axis, table, s); break;
    case 384: *e = launch_axis<16, 24>(z, lines, axis, table, s); break;
    case 200: *e = launch_axis<20, 10>(z, lines, axis, table, s); break;
    case 240: *e = launch_axis<20, 12>(z, lines, axis, table, s); break;
    case 288: *e = launch_axis<24, 12>(z, lines, axis, table, s); break;
    default: return false;
    }
    return true;
}

} // namespace fft
} // namespace sh
