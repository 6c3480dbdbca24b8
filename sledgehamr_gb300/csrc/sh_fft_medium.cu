/* Radix pairs of the FP64 transforms: 100, 120, 128, 144, 160. */
#include "sh_fft_kernel.cuh"

namespace sh {
namespace fft {

bool launch_medium(int P, double2 *z, long long lines, int axis, const Twiddle *table,
                   cudaStream_t s, cudaError_t *e) {
    switch (P) {
    case 100: *e = launch_axis<10, 10>(z, lines, axis, table, s); break;
    case 120: *e = launch_axis<12, 10>(z, lines, axis, table, s); break;
    case 128: *e = launch_axis<16, 8>(z, lines, axis, table, s); break;
    case 144: *e = launch_axis<12, 12>(z, lines, axis, table, s); break;
    case 160: *e = launch_axis<16, 10>(z, lines, axis, table, s); break;
    default: return false;
    }
    return true;
}

} // namespace fft
} // namespace sh
