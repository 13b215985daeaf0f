// pair_work (csrc/nvfp4_pair_work.h) over random launches and over those that pair_plan (csrc/nvfp4_gemm_choice.h) makes of random GEMMs, both as the
// library includes them: every (tile, k block) is done exactly once;
// a part handed over is its pair's first item and the only one; the pairs that hand parts of a tile over are exactly those that the
// finishing pair waits for; no two pairs of those that share differ by more than two k blocks' cost, leaving the rounds aside.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>

#include "nvfp4_gemm_choice.h"
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

// Clusters of 1 .. 8 CTAs that a B200 holds, two CTAs on every SM, as two_cta_clusters counts them.
static const uint32_t kClusters[kNarrowMaxParts + 1] = {0, 296, 148, 88, 67, 53, 43, 35, 31};

static PairPlan plan_for(uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t terms, bool swiglu, uint32_t all, uint64_t slots, bool pairs_only) {
    return pair_plan(rows, cols, tokens, terms, swiglu, all, slots, pairs_only ? UINT32_MAX : narrow_cut(kClusters, rows, cols, tokens, terms).ns);
}
static PairShares shares_of(const PairPlan& plan, uint32_t rows, uint32_t cols, uint32_t terms) {
    const uint32_t n_tiles = (rows + 255) / 256;
    return PairShares{plan.token_pairs * n_tiles, plan.tail_columns ? n_tiles : 0, (cols + 255) / 256, plan.split.sharers,
                      pair_block_cost(terms, 0), pair_block_cost(terms, plan.tail_columns)};
}

static bool random_launches() {
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
            return false;
        }
    }
    if (cut <= 10000) std::puts("too few launches share tiles");
    return cut > 10000;
}

static bool chosen_launches() {
    uint32_t cut = 0, tails = 0, cut_tails = 0;
    for (uint32_t round = 0; round < 20000; ++round) {
        const uint32_t rows = 128 * (1 + std::rand() % 272), cols = 64 * (1 + std::rand() % (round % 3 ? 80 : 300)), terms = 1 + std::rand() % 3;
        const uint32_t tokens = 9 + std::rand() % (round % 2 ? 1100 : 4088), all = round % 4 ? 74 : 1 + std::rand() % 74;
        const uint64_t slots = round % 5 ? all : std::rand() % 80;
        const PairPlan plan = plan_for(rows, cols, tokens, terms, round % 3 == 0, all, slots, round % 8 == 0);
        if (!plan.token_pairs) continue;   // the narrow kernel's
        const uint32_t covered = plan.token_pairs * 256 + plan.tail_columns;
        const bool sound = plan.split.pairs <= all && plan.split.sharers <= plan.split.pairs && plan.split.sharers <= slots && covered >= tokens &&
                           (plan.tail_columns ? plan.tail_columns % 32 == 0 && plan.tail_columns <= 128 && tokens > plan.token_pairs * 256 : true);
        if (!sound || !check(plan.split.pairs, shares_of(plan, rows, cols, terms))) {
            std::printf("rows %u cols %u tokens %u terms %u pairs %u slots %llu: %u x 256 + %u on %u, shared by %u\n", rows, cols, tokens, terms, all,
                        static_cast<unsigned long long>(slots), plan.token_pairs, plan.tail_columns, plan.split.pairs, plan.split.sharers);
            return false;
        }
        cut += plan.split.sharers != 0;
        tails += plan.tail_columns != 0;
        cut_tails += plan.split.sharers && plan.tail_columns;
    }
    if (cut <= 2000 || tails <= 2000 || cut_tails <= 500) std::printf("cut %u, with tail tiles %u, both %u\n", cut, tails, cut_tails);
    return cut > 2000 && tails > 2000 && cut_tails > 500;
}

// Without arguments: the checks. With rows, cols, tokens, terms, 0 or 1 for gate|up and slots: what a B200's 74 pairs do of such a GEMM, as token pairs, tail columns and
// pairs that share tiles; of those, pairs that hand a part of a tail tile over, and tail tiles that are put together.
int main(int count, char** text) {
    if (count == 7) {
        uint32_t v[6];
        for (int i = 0; i < 6; ++i) v[i] = static_cast<uint32_t>(std::strtoul(text[1 + i], nullptr, 10));
        const PairPlan plan = plan_for(v[0], v[1], v[2], v[3], v[4] != 0, 74, v[5], false);
        uint32_t given = 0, finished = 0;
        if (plan.token_pairs) {
            const PairShares s = shares_of(plan, v[0], v[1], v[3]);
            for (uint32_t pair = 0; pair < plan.split.pairs; ++pair) {
                const PairWork w = pair_work(pair, plan.split.pairs, s);
                for (uint32_t i = 0; i < w.items; ++i) {
                    const PairItem item = w.item(i, pair, plan.split.pairs, s.k_blocks);
                    given += item.kind == 1 && item.tile >= s.main;
                    finished += item.kind == 2 && item.tile >= s.main;
                }
            }
        }
        std::printf("%u %u %u %u %u\n", plan.token_pairs, plan.tail_columns, plan.split.sharers, given, finished);
        return 0;
    }
    std::srand(5);
    if (!random_launches() || !chosen_launches()) return 1;
    std::puts("ok");
    return 0;
}
