/* sh_halo.h over every place of every tile of realisations of 8 to 300 cells:
 * the places that a stencil reads hold the periodic cell, the others none,
 * and no place lies outside the realisation. */
#include "sh_halo.h"

#include <cstdio>
#include <initializer_list>

int main() {
    long long bad = 0;
    for (int N = 8; N <= 300; ++N)
        for (int H = 1; H <= 2; ++H)
            for (int T : {32, 8}) /* places of a tile along x and y */
                for (int x0 = 0; x0 < N; x0 += T)
                    for (int p = 0; p < T + 2 * H; ++p) {
                        const int a = x0 - H + p, s = sh::fast::halo_source(a, N, H);
                        const int want = a < N + H ? ((a % N) + N) % N : -1;
                        if (s != want || s < -1 || s >= N) {
                            if (bad++ == 0)
                                std::printf("N = %d, H = %d, tile at %d, place %d: cell %d\n", N, H,
                                            x0, p, s);
                        }
                    }
    std::printf("%lld places outside\n", bad);
    return bad != 0;
}
