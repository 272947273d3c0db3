// How the single-token kernels' units are dealt out to warps and CTAs. Plain host arithmetic: no device code.
#pragma once
#include <algorithm>
#include <climits>

namespace oco {

// Warps per unit of the single-token kernels: as many as keep every warp of the grid busy.
inline int pick_ksplit(int units, int ctas, int warps_per_cta) {
    for (int k : {10, 8, 5, 4, 2})
        if (warps_per_cta % k == 0 && units * k <= ctas * warps_per_cta) return k;
    return 1;
}

// Blocks in a row for the busiest warp when `units` units of nkb blocks go round `ctas` CTAs, ksplit warps to a unit;
// `start`: blocks in whose time a unit begins (its first copies' latency, its sums and stores).
inline int blocks_in_a_row(int units, int nkb, int ctas, int warps_per_cta, int ksplit, int start = 0) {
    const int slots = ctas * (warps_per_cta / ksplit);
    return (units + slots - 1) / slots * ((nkb + ksplit - 1) / ksplit + start);
}

// Warps per unit where routed and always-on units share a launch (a Nemotron up launch): the split with the fewest
// blocks in a row for the busiest warp, several rounds of units allowed. At 928 units of 84 blocks on 148 x 20 warps
// two warps per unit leave a third of the warps without one (42 blocks in a row), five take 34.
inline int pick_ksplit_rounds(int units, int nkb, int ctas, int warps_per_cta) {
    int best = 1, least = INT_MAX;
    for (int k : {1, 2, 4, 5, 8, 10}) {
        if (warps_per_cta % k) continue;
        const int run = blocks_in_a_row(units, nkb, ctas, warps_per_cta, k);
        if (run < least) { least = run; best = k; }
    }
    return best;
}

// A down launch: CTAs go round K + shares places, one for each route and `shares` for the always-on expert (sh_nkb
// blocks per row; 0: there is none). turns: CTAs per place.
struct DownDeal { int shares, turns, ksplit, sh_ksplit; };

// Shares in proportion to the widths, unless another number leaves the busiest warp of either kind fewer blocks in a
// row: where the places don't divide the CTAs, some stay idle (75 places on 148 SMs use 75 of them), and next to very
// narrow routes the proportion asks for more shares than there are CTAs. A unit of such a route is one or two blocks
// long and costs its start, about a stage of 16 blocks. Hidden 4096, routes of 64, always-on expert of 4416, six routes:
// 69 shares 78.5 us, 43 shares 43.1, five 32.9; hidden 2688, 32 and 4800: one share 41.1 us, 142 shares 54.6, ten 26.8.
// For each number of turns only the largest number of shares is looked at; it leaves the fewest CTAs idle.
// turns == 0: more places than CTAs.
inline DownDeal deal_down(int K, int row_blocks, int nkb, int sh_nkb, int ctas, int warps_per_cta) {
    const int room = ctas - K;
    if (!sh_nkb || room < 1) {
        const int turns = sh_nkb ? 0 : ctas / K;
        return {0, turns, turns ? pick_ksplit(row_blocks, turns, warps_per_cta) : 1, 1};
    }
    DownDeal best{};
    int least = INT_MAX;
    auto look = [&](int shares) {
        const int turns = ctas / (K + shares);
        const DownDeal d{shares, turns, pick_ksplit(row_blocks, turns, warps_per_cta), pick_ksplit(row_blocks, turns * shares, warps_per_cta)};
        const int run = std::max(blocks_in_a_row(row_blocks, nkb, turns, warps_per_cta, d.ksplit, 16),
                                 blocks_in_a_row(row_blocks, sh_nkb, turns * shares, warps_per_cta, d.sh_ksplit, 16));
        if (run < least) { least = run; best = d; }
    };
    look(std::min(room, std::max(1, (sh_nkb + nkb / 2) / nkb)));
    for (int turns = ctas / (K + 1); turns >= 1; turns--) look(ctas / turns - K);
    return best;
}

}  // namespace oco
