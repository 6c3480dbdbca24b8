/* Periodic sources of the halo columns of an ensemble's tiles (host and
 * device). */
#ifndef SH_HALO_H_
#define SH_HALO_H_

#if defined(__CUDACC__)
#define SH_HALO_HD __host__ __device__ __forceinline__
#else
#define SH_HALO_HD inline
#endif

namespace sh {
namespace fast {

/* a in [-N, 2N) brought into [0, N) */
SH_HALO_HD int wrap(int a, int N) { return a < 0 ? a + N : (a >= N ? a - N : a); }

/* Cell that the plane element at a = (first cell of the tile - H + its place)
 * holds along one axis, or -1 for the places past the halo of an extent of N
 * cells.  Tiles are TX x TY places whatever N is, so that a tile of a small
 * realisation (N <= 16 along x) has places more than N beyond its last cell,
 * which nothing reads; one wrap leaves them outside the realisation, for the
 * last one outside the arrays. */
SH_HALO_HD int halo_source(int a, int N, int H) { return a < N + H ? wrap(a, N) : -1; }

} // namespace fast
} // namespace sh

#endif // SH_HALO_H_
