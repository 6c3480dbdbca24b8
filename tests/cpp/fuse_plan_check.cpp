/* sh_fuse_plan.h against the search that it shortens: every depth's tiles
 * listed, sorted by cost and dealt to the SMs, the first depth that ends
 * earliest kept.  The same tiles in the same order, over mixes of members. */
#include "sh_fuse_plan.h"

#include <cstdio>
#include <random>

using namespace sh::fast;

static std::vector<FusedTile> exhaustive(const std::vector<FusedMember> &members, int nsm,
                                         int most) {
    auto cuts = [](int n, int most) { return (n + most - 1) / most; };
    std::vector<FusedTile> best;
    long long least = 0;
    int top = 0;
    for (const FusedMember &m : members) top = std::max(top, m.N);
    for (int parts = 1; parts <= 16 && top > 0; ++parts) {
        const int depth = cuts(top, parts);
        if (parts > 1 && depth < 8) break;
        std::vector<FusedTile> t;
        for (const FusedMember &m : members) {
            const int N = m.N;
            const int w = cuts(N, cuts(N, most)), nz = cuts(N, cuts(N, depth));
            for (int z = 0; z < N; z += nz)
                for (int y = 0; y < N; y += w)
                    for (int x = 0; x < N; x += w)
                        t.push_back(FusedTile{m.r, x, y, z, std::min(w, N - x),
                                              std::min(w, N - y), std::min(nz, N - z)});
        }
        std::stable_sort(t.begin(), t.end(), [](const FusedTile &a, const FusedTile &b) {
            return fused_cost(a.h, a.nz) > fused_cost(b.h, b.nz);
        });
        std::vector<long long> sm(nsm, 0);
        long long end = 0;
        for (const FusedTile &q : t) {
            auto first = std::min_element(sm.begin(), sm.end());
            *first += fused_cost(q.h, q.nz);
            end = std::max(end, *first);
        }
        if (best.empty() || end < least) {
            least = end;
            best.swap(t);
        }
    }
    return best;
}

int main() {
    std::mt19937 g(3);
    auto uniform = [&](int lo, int hi) { return std::uniform_int_distribution<int>(lo, hi)(g); };
    int bad = 0;
    for (int q = 0; q < 400; ++q) {
        std::vector<FusedMember> m;
        const int n = q == 0 ? 0 : uniform(1, q % 3 == 0 ? 40 : 6);
        const int top = q % 7 == 0 ? 12 : (q % 2 ? 160 : 70), same = q % 5 == 0 ? uniform(8, top) : 0;
        for (int r = 0; r < n; ++r) m.push_back(FusedMember{2 * r, same ? same : uniform(8, top)});
        const int nsm = q % 4 ? 152 : uniform(1, 152);
        const FusedPlan plan = plan_fused(m, nsm);
        /* blocks of 16 x 16 threads where every member fits one */
        int largest = 0;
        for (const FusedMember &r : m) largest = std::max(largest, r.N);
        const bool small = n > 0 && largest <= 10;
        const std::vector<FusedTile> &a = plan.tiles,
                                     b = exhaustive(m, nsm * (small ? 4 : 1), small ? 10 : 26);
        bool equal = a.size() == b.size() && plan.side == (small ? 16 : 32);
        for (size_t t = 0; equal && t < a.size(); ++t)
            equal = a[t].r == b[t].r && a[t].x0 == b[t].x0 && a[t].y0 == b[t].y0 &&
                    a[t].z0 == b[t].z0 && a[t].w == b[t].w && a[t].h == b[t].h &&
                    a[t].nz == b[t].nz;
        if (!equal) {
            std::printf("mix %d of %d members: %zu tiles against %zu\n", q, n, a.size(), b.size());
            ++bad;
        }
    }
    return bad != 0;
}
