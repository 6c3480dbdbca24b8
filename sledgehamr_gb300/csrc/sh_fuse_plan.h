/* Tiles of the one-pass RKN4 steps of FP32 axion ensembles (host code). */
#ifndef SH_FUSE_PLAN_H_
#define SH_FUSE_PLAN_H_

#include <algorithm>
#include <functional>
#include <map>
#include <queue>
#include <vector>

namespace sh {
namespace fast {

/* A block has side x side threads, one column each, of which the three stages
 * use up kFuseHalo on each side.  One block of side 32 fills an SM.  Members
 * of up to 10^3 cells leave most of such a block idle and take side 16, four
 * blocks per SM: 2000 members of 8^3 take 57 us per step against 140, FP32 + Kahan
 * (127 with the stages launched one by one). */
constexpr int kFuseSide = 32, kFuseSmall = 16, kFuseHalo = 3;
constexpr int fused_out(int side) { return side - 2 * kFuseHalo; } /* columns left */
constexpr int fused_blocks(int side) { return side == kFuseSmall ? 4 : 1; } /* per SM */

struct FusedTile {
    int r;
    int x0, y0, z0, w, h, nz;
};

/* A tile takes its rows with halo times its planes with halo and two more
 * for its start. */
inline long long fused_cost(int h, int nz) {
    return (long long)(h + 2 * kFuseHalo) * (nz + 2 * kFuseHalo + 2);
}

struct FusedMember {
    int r, N; /* slot and cells a side */
};

struct FusedPlan {
    int side = kFuseSide;
    std::vector<FusedTile> tiles;
};

/* Tiles of the members, longest first: every member cut into equal columns of
 * at most fused_out cells a side and into the depth (equal parts of the largest
 * member's planes) whose tiles end first when nsm SMs take them in order, as
 * many at a time as an SM holds blocks.  On a mix of 32^3 to 128^3 boxes the costs predict depths 16 /
 * 26 / 32 / 43 / 64 within 2 % (165 / 135 / 163 / 128 / 152 us per step).
 *
 * A pool plans at every admission and release, so a depth is tried on the
 * numbers of tiles of each cost, not on lists of tiles, and only when the SMs'
 * even share of its tiles ends before the best depth so far (deeper cuts add
 * halo, so that a pool of many tiles tries one or two of the sixteen): 24
 * members of 128^3 are planned in 0.02 ms, against 5.4 with every depth's
 * tiles listed and sorted. */
inline FusedPlan plan_fused(const std::vector<FusedMember> &members, int nsm) {
    auto cuts = [](int n, int most) { return (n + most - 1) / most; };
    std::map<int, int> sizes; /* members by size */
    for (const FusedMember &m : members) ++sizes[m.N];
    FusedPlan plan;
    if (sizes.empty()) return plan;
    const int top = sizes.rbegin()->first;
    if (top <= fused_out(kFuseSmall)) plan.side = kFuseSmall;
    const int most = fused_out(plan.side), slots = nsm * fused_blocks(plan.side);
    int best = 0;
    long long least = 0;
    for (int parts = 1; parts <= 16; ++parts) {
        const int depth = cuts(top, parts);
        if (parts > 1 && depth < 8) break;
        std::map<long long, long long, std::greater<long long>> tiles; /* number by cost */
        long long total = 0;
        for (const auto &size : sizes) {
            const int N = size.first, n = size.second;
            const int w = cuts(N, cuts(N, most)), nz = cuts(N, cuts(N, depth));
            const int cols = cuts(N, w), layers = cuts(N, nz);
            /* rows and planes of the last tile along y and z */
            const int hl = N - (cols - 1) * w, nl = N - (layers - 1) * nz;
            auto add = [&](int h, int planes, long long count) {
                if (count == 0) return;
                tiles[fused_cost(h, planes)] += count * cols * n;
                total += count * cols * n * fused_cost(h, planes);
            };
            add(w, nz, (long long)(cols - 1) * (layers - 1));
            add(hl, nz, layers - 1);
            add(w, nl, cols - 1);
            add(hl, nl, 1);
        }
        if (best != 0 && std::max((total + slots - 1) / slots, tiles.begin()->first) >= least) continue;
        std::priority_queue<long long, std::vector<long long>, std::greater<long long>> sm;
        for (int q = 0; q < slots; ++q) sm.push(0);
        long long end = 0;
        for (const auto &[cost, count] : tiles)
            for (long long q = 0; q < count; ++q) {
                const long long e = sm.top() + cost;
                sm.pop();
                sm.push(e);
                end = std::max(end, e);
            }
        if (best == 0 || end < least) {
            least = end;
            best = depth;
        }
    }
    std::vector<FusedTile> &t = plan.tiles;
    for (const FusedMember &m : members) {
        const int N = m.N;
        const int w = cuts(N, cuts(N, most)), nz = cuts(N, cuts(N, best));
        for (int z = 0; z < N; z += nz)
            for (int y = 0; y < N; y += w)
                for (int x = 0; x < N; x += w)
                    t.push_back(FusedTile{m.r, x, y, z, std::min(w, N - x), std::min(w, N - y),
                                          std::min(nz, N - z)});
    }
    std::stable_sort(t.begin(), t.end(), [](const FusedTile &a, const FusedTile &b) {
        return fused_cost(a.h, a.nz) > fused_cost(b.h, b.nz);
    });
    return plan;
}

} // namespace fast
} // namespace sh

#endif // SH_FUSE_PLAN_H_
