/* Bin lists of the spectra of P^3 grids (host code; any P, even or odd). */
#ifndef SH_GW_BINS_H_
#define SH_GW_BINS_H_

#include <algorithm>
#include <cmath>
#include <vector>

#ifdef _OPENMP
#include <omp.h>
#endif

namespace sh {

/* Wave number of index a: 0 .. (P - 1) / 2, then the negative ones from
 * -(P / 2) on. */
inline long long wave_index(long long a, int P) { return a < (P + 1) / 2 ? a : a - P; }

/* Sorted unique k^2 of a dim^3 grid. */
inline std::vector<long long> unique_k2_host(int dim) {
    std::vector<long long> sq;
    for (int a = 0; a < dim; ++a) sq.push_back(wave_index(a, dim) * wave_index(a, dim));
    std::sort(sq.begin(), sq.end());
    sq.erase(std::unique(sq.begin(), sq.end()), sq.end());
    const long long maxs = 3 * sq.back();
    std::vector<char> hit((size_t)maxs + 1, 0);
    for (long long x : sq)
        for (long long y : sq)
            for (long long z : sq) hit[(size_t)(x + y + z)] = 1;
    std::vector<long long> out;
    for (long long v = 0; v <= maxs; ++v)
        if (hit[(size_t)v]) out.push_back(v);
    return out;
}

/* The half-spectrum's cells ((c P + b) H + a, H = P / 2 + 1) sorted by bin,
 * ascending within a bin: bin q holds cells[off[q]] .. cells[off[q + 1] - 1]. */
struct BinLists {
    std::vector<long long> ks; /* k^2 of every bin */
    std::vector<long long> off;
    std::vector<int> cells;
};

inline BinLists bin_lists(int P, bool unbinned) {
    BinLists g;
    const int H = P / 2 + 1;
    const long long ncell = (long long)H * P * P;
    if (unbinned) {
        g.ks = unique_k2_host(P);
    } else {
        for (int k = 0; k <= std::sqrt(3.) / 2. * static_cast<double>(P) + .5; ++k)
            g.ks.push_back((long long)k * k);
    }
    const int nb = (int)g.ks.size();
    const long long maxsq = 3LL * (P / 2) * (P / 2); /* |wave_index| <= P / 2 */
    std::vector<int> lut((size_t)maxsq + 1, -1);
    if (unbinned) {
        for (int q = 0; q < nb; ++q) lut[(size_t)g.ks[q]] = q;
    } else {
        for (long long sq = 0; sq <= maxsq; ++sq) {
            long long r = (long long)std::llround(std::sqrt((double)sq));
            /* round(sqrt(sq)) == r  <=>  r^2 - r < sq <= r^2 + r */
            while (r * r + r < sq) ++r;
            while (r > 0 && r * r - r >= sq) --r;
            lut[(size_t)sq] = (int)r;
        }
    }
    auto bin_of = [&](long long e) {
        const int a = (int)(e % H), b = (int)((e / H) % P), c = (int)(e / ((long long)H * P));
        const long long li = wave_index(a, P), lj = wave_index(b, P), lk = wave_index(c, P);
        return lut[(size_t)(li * li + lj * lj + lk * lk)];
    };
    /* stable counting sort over contiguous chunks of cells, one per thread */
    int nt = 1;
#ifdef _OPENMP
    nt = std::max(1, std::min(omp_get_max_threads(), 64));
#endif
    const long long chunk = (ncell + nt - 1) / nt;
    std::vector<long long> cnt((size_t)nt * nb, 0);
#pragma omp parallel for num_threads(nt) schedule(static, 1)
    for (int t = 0; t < nt; ++t) {
        long long *c = cnt.data() + (size_t)t * nb;
        const long long e1 = std::min(ncell, (t + 1) * chunk);
        for (long long e = t * chunk; e < e1; ++e) c[bin_of(e)]++;
    }
    g.off.assign(nb + 1, 0);
    for (int q = 0; q < nb; ++q) {
        long long run = g.off[q];
        for (int t = 0; t < nt; ++t) {
            const long long c = cnt[(size_t)t * nb + q];
            cnt[(size_t)t * nb + q] = run; /* start of thread t's cells in bin q */
            run += c;
        }
        g.off[q + 1] = run;
    }
    g.cells.resize((size_t)ncell);
#pragma omp parallel for num_threads(nt) schedule(static, 1)
    for (int t = 0; t < nt; ++t) {
        long long *pos = cnt.data() + (size_t)t * nb;
        const long long e1 = std::min(ncell, (t + 1) * chunk);
        for (long long e = t * chunk; e < e1; ++e) g.cells[(size_t)pos[bin_of(e)]++] = (int)e;
    }
    return g;
}

} // namespace sh

#endif // SH_GW_BINS_H_
