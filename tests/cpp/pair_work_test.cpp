// pair_work (csrc/nvfp4_pair_work.h) over the launches that the command line asks for: every (tile, k block) is done exactly once;
// a part handed over is its pair's first item and the only one; the pairs that hand parts of a tile over are exactly those that the
// finishing pair waits for; no two pairs of those that share differ by more than two k blocks' cost, leaving the rounds aside.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>

#include "nvfp4_pair_work.h"

using namespace augur_sm100;

static bool check(uint32_t pairs, const PairShares& s) {
    std::vector<uint32_t> done(static_cast<size_t>(s.main + s.tail) * s.k_blocks, 0);
    std::map<uint32_t, std::vector<uint32_t>> givers, waits;
    uint64_t least = ~uint64_t(0), most = 0;
    for (uint32_t pair = 0; pair < pairs; ++pair) {
        const PairWork w = pair_work(pair, pairs, s);
        uint64_t cost = 0, blocks = 0;
        for (uint32_t i = 0; i < w.items; ++i) {
            const PairItem item = w.item(i, pair, pairs, s.k_blocks);
            if (item.tile >= s.main + s.tail || item.kb0 >= item.kb1 || item.kb1 > s.k_blocks) return false;
            for (uint32_t kb = item.kb0; kb < item.kb1; ++kb) ++done[static_cast<size_t>(item.tile) * s.k_blocks + kb];
            if (item.kind == 1) {
                if (i != 0) return false;
                givers[item.tile].push_back(pair);
            } else if (item.kb1 != s.k_blocks || (item.kind == 0 && item.kb0 != 0)) {
                return false;
            } else if (item.kind == 2) {
                if (item.first_giver >= pair || waits.count(item.tile)) return false;
                for (uint32_t giver = item.first_giver; giver < pair; ++giver) waits[item.tile].push_back(giver);
            }
            blocks += item.kb1 - item.kb0;
            cost += static_cast<uint64_t>(item.kb1 - item.kb0) * (item.tile < s.main ? s.cost_main : s.cost_tail);
        }
        if (blocks != w.blocks(s.k_blocks)) return false;
        if (s.sharers && pair < s.sharers) {
            least = cost < least ? cost : least;
            most = cost > most ? cost : most;
        }
    }
    for (uint32_t times : done) if (times != 1) return false;
    const uint32_t larger = s.cost_main > s.cost_tail ? s.cost_main : s.cost_tail;
    return givers == waits && (!s.sharers || most - least <= 2 * larger);
}

int main() {
    std::srand(5);
    uint32_t cut = 0;
    for (uint32_t round = 0; round < 20000; ++round) {
        const uint32_t all = 1 + std::rand() % (round % 2 ? 74 : 8), n_tiles = 1 + std::rand() % 140, token_pairs = 1 + std::rand() % 5;
        PairShares s{n_tiles * token_pairs, round % 3 ? n_tiles : 0, 1 + std::rand() % (round % 5 ? 12u : 70u), 0, 1 + std::rand() % 130u, 1 + std::rand() % 130u};
        const uint64_t cost = static_cast<uint64_t>(s.main % all) * s.k_blocks * s.cost_main + static_cast<uint64_t>(s.tail) * s.k_blocks * s.cost_tail;
        const uint64_t limit = cost / (s.cost_main > s.cost_tail ? s.cost_main : s.cost_tail);
        if (round % 7) s.sharers = static_cast<uint32_t>(limit < all ? limit : all);
        if (s.sharers > 1 && round % 4 == 0) s.sharers = 1 + std::rand() % s.sharers;
        uint32_t pairs = all;
        if (!s.sharers && s.main + s.tail < all) pairs = s.main + s.tail;
        cut += s.sharers != 0;
        if (!check(pairs, s)) {
            std::printf("pairs %u main %u tail %u k blocks %u sharers %u costs %u %u\n", pairs, s.main, s.tail, s.k_blocks, s.sharers, s.cost_main, s.cost_tail);
            return 1;
        }
    }
    std::puts(cut > 10000 ? "ok" : "too few launches share tiles");
    return 0;
}
