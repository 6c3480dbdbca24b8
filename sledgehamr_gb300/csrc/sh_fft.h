/* Interface of the FP64 three-dimensional transforms of sh_fft_kernel.cuh. */
#ifndef SH_FFT_H_
#define SH_FFT_H_

#include <cuda_runtime.h>

#include "sh_fft.cuh"

namespace sh {
namespace fft {

/* Whether transform3 takes P^3 arrays: P one of the 19 sizes instantiated in
 * sh_fft_small.cu, sh_fft_medium.cu and sh_fft_large.cu, up to 384. */
bool supported(int P);
/* Twiddle factors exp(-2 pi i j / P), j < P, on the device (cudaFree'd by the
 * caller), written in stream order; nullptr when the allocation fails. */
Twiddle *make_table(int P, cudaStream_t s);
/* In-place forward transforms of n complex FP64 P^3 arrays, one after the
 * other in z (element (x, y, z) of array q at ((q P + z) P + y) P + x),
 * unnormalised; table from make_table(P).  Three launches. */
cudaError_t transform3(double2 *z, int n, int P, const Twiddle *table, cudaStream_t s);

/* One axis of a radix pair (the instantiations live in several files, which
 * compile in parallel); false when the pair is not in that file, else *e is
 * the launch's error. */
bool launch_small(int P, double2 *z, long long lines, int axis, const Twiddle *table,
                  cudaStream_t s, cudaError_t *e);
bool launch_medium(int P, double2 *z, long long lines, int axis, const Twiddle *table,
                   cudaStream_t s, cudaError_t *e);
bool launch_large(int P, double2 *z, long long lines, int axis, const Twiddle *table,
                  cudaStream_t s, cudaError_t *e);

} // namespace fft
} // namespace sh

#endif // SH_FFT_H_
