/* The spectra's bin lists of even and odd grids: every cell of the
 * half-spectrum once, in the bin of its k^2, ascending within a bin.  Built
 * with range-checked vectors. */
#include "sh_gw_bins.h"

#include <cstdio>

static int check(int P, bool unbinned) {
    const sh::BinLists g = sh::bin_lists(P, unbinned);
    const long long H = P / 2 + 1, ncell = H * P * P;
    const int nb = (int)g.ks.size();
    if ((int)g.off.size() != nb + 1 || g.off[0] != 0 || g.off[nb] != ncell ||
        (long long)g.cells.size() != ncell)
        return 1;
    std::vector<char> seen((size_t)ncell, 0);
    for (int q = 0; q < nb; ++q)
        for (long long e = g.off[q]; e < g.off[q + 1]; ++e) {
            const long long cell = g.cells[(size_t)e];
            if (cell < 0 || cell >= ncell || seen[(size_t)cell]) return 2;
            if (e > g.off[q] && cell <= g.cells[(size_t)e - 1]) return 3;
            seen[(size_t)cell] = 1;
            long long k2 = 0;
            for (long long i : {cell % H, cell / H % P, cell / (H * P)}) {
                /* the residue of i modulo P that is nearest to zero */
                const long long k = 2 * i < P ? i : P - i;
                k2 += k * k;
            }
            if (unbinned ? k2 != g.ks[q] : q != (int)(std::sqrt((double)k2) + .5)) return 4;
        }
    return 0;
}

int main() {
    int bad = 0;
    for (int P = 1; P <= 41; ++P)
        for (int unbinned = 0; unbinned < 2; ++unbinned)
            if (const int e = check(P, unbinned)) {
                std::printf("P = %d, unbinned %d: %d\n", P, unbinned, e);
                ++bad;
            }
    return bad != 0 || check(99, true) || check(100, true);
}
