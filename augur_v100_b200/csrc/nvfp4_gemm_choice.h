// Which kernel a prefill GEMM takes, and how the launch cuts its work, by what each would take: the estimates, the choice, the numbers of parts. On
// the host only, and plain C++, so that the choice can be looked at without a GPU.
#pragma once

#include <cstdint>

namespace augur_sm100 {

// ---- narrow kernel: 128 features x up to 128 tokens, `parts` CTAs (a cluster) per tile ----
constexpr uint32_t kNarrowMaxParts = 8;                               // portable cluster size
// How a launch cuts its work, and about how long it takes: the waves of clusters times the pipeline steps of a part, of the
// numbers of CTAs per item the one with the least. Fitted on a B200 with two CTAs on every SM, before a step's MMAs became one block of
// instructions and a cluster's sums were read where they are: a step (k block x term) 0.33 us at 16 tokens and 0.44 at 128, a launch about 6 us
// beyond its steps, a wave after the first 3, the parts' sums 4 us more at 128 tokens. Measured since, three terms, one part: 0.32 to 0.34 us
// a step at 16 tokens, 0.50 at 48, 0.55 at 128, and 5 to 9 us beyond. The number of parts chosen is 1.7 % off the best on average, 25 % at worst
// (1024 x 5120, 200 tokens). `clusters[parts]`: clusters of so many CTAs that a launch may count on to run at once.
struct NarrowCut {
    uint32_t token_tiles, tile_tokens, columns, parts, ns;
};
inline NarrowCut narrow_cut(const uint32_t (&clusters)[kNarrowMaxParts + 1], uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t terms) {
    constexpr uint32_t kTile = 128, kDepth = 256;
    NarrowCut cut{};
    cut.token_tiles = (tokens + kTile - 1) / kTile;
    cut.tile_tokens = tokens < kTile ? tokens : kTile;
    cut.columns = (cut.tile_tokens + 15) / 16 * 16;
    const uint64_t items = static_cast<uint64_t>(rows / kTile) * cut.token_tiles;
    const uint32_t k_blocks = (cols + kDepth - 1) / kDepth, step_ns = 320 + cut.columns * 120 / kTile;
    uint64_t least = ~uint64_t(0);
    for (uint32_t parts = 1; parts <= kNarrowMaxParts && parts <= k_blocks; ++parts) {
        const uint64_t waves = (items + clusters[parts] - 1) / clusters[parts];
        const uint64_t ns = waves * ((k_blocks + parts - 1) / parts * terms * step_ns + 3000) + 3000 + cut.columns * 4000 / kTile;
        if (ns < least) {
            least = ns;
            cut.parts = parts;
        }
    }
    // Against the pair kernel the estimate counts, not only the order: fitted as kPairBlockCost.
    const uint64_t ns = (items + clusters[cut.parts] - 1) / clusters[cut.parts] *
                            ((k_blocks + cut.parts - 1) / cut.parts * (terms * (350 + cut.columns) + 110) + 2900) +
                        2100 + cut.columns * 4000 / kTile;
    cut.ns = static_cast<uint32_t>(ns < UINT32_MAX / 2 ? ns : UINT32_MAX / 2);
    return cut;
}

// ---- pair kernel: 256 x 256 tiles on pairs of CTAs, tail tiles for up to 128 token rows past whole 256 ----
constexpr uint32_t kSplitWays = 8;              // a leftover tile is cut into this many parts at most

// How a launch of the pair kernel over `token_pairs` x 256 token rows shares its tiles out, and about how long it takes.
struct PairSplit {
    uint32_t pairs, sharers;     // sharers: pairs that share the leftover tiles (0: every tile is one pair's)
    uint32_t ns;
};

// In units of 10 ns, fitted on a B200 to 429 GEMMs (eleven weights from 1024 x 5120 to 34816 x 5120, 13 token counts from 48 to 1100, one to three terms),
// each with every choice forced in turn: what a k block of a whole tile costs and of a tail tile, handing the parts of leftover tiles over when nothing
// else is left to do (and per part) and when it happens under whole tiles, a launch beyond that. With the narrow kernel's estimate the
// choice is 0.1 % off the best on average, 14 % at worst (2432 x 2176, 160 to 256 tokens, one term, 9.0 against 10.2 us).
constexpr uint32_t kPairBlockCost[3] = {52, 93, 118};
constexpr uint32_t kSplitCost = 450, kSplitPartCost = 170, kSplitCoveredCost = 480, kSplitAddCost = 300, kPairLaunchNs = 5500;
inline uint32_t pair_block_cost(uint32_t terms, uint32_t tail_columns) {
    return tail_columns ? 30 + terms * 9 + terms * (tail_columns - 32) * 7 / 100 : kPairBlockCost[terms - 1];
}

// Tiles past the last full round of the pairs (all tiles, when there are fewer tiles than pairs) may be cut along k, in `ways`
// parts each at most and over all pairs at most, when the plan's scratch has a slot for the partial accumulator of each pair that
// shares them (`slots`). Of the numbers of parts up to kSplitWays the one with the least steps is taken: cut in eight, the 4 tiles of 1024
// rows and 256 tokens took 25 us, whole 15.
inline PairSplit pair_split(uint32_t token_pairs, uint32_t tail_columns, uint32_t rows, uint32_t cols, uint32_t terms, uint32_t all_pairs, uint64_t slots) {
    constexpr uint32_t kTile = 256, kDepth = 256;
    const uint32_t n_tiles = (rows + kTile - 1) / kTile, k_blocks = (cols + kDepth - 1) / kDepth;
    const uint32_t main = token_pairs * n_tiles, tail = tail_columns ? n_tiles : 0;
    const uint64_t cost_main = pair_block_cost(terms, 0), cost_tail = tail ? pair_block_cost(terms, tail_columns) : 0;
    const uint32_t rounds = main / all_pairs, left = main % all_pairs;
    PairSplit best{main + tail < all_pairs ? main + tail : all_pairs, 0, 0};
    // not cut: the first pair has the most tiles of either kind
    const uint64_t most_main = (main + all_pairs - 1) / all_pairs, most = (main + tail + all_pairs - 1) / all_pairs;
    uint64_t least = k_blocks * (most_main * cost_main + (most - most_main) * cost_tail);
    const uint64_t line = k_blocks * (left * cost_main + tail * cost_tail), largest = left ? cost_main : cost_tail;
    for (uint32_t ways = 2; line && ways <= kSplitWays; ++ways) {
        uint64_t sharers = line * ways / (k_blocks * largest);
        if (sharers > all_pairs) sharers = all_pairs;
        if (sharers > line / cost_main) sharers = line / cost_main;      // every range holds a k block
        if (sharers < 2 || (!tail && sharers <= left) || sharers > slots) break;
        const uint64_t parts = (sharers * k_blocks * largest + line - 1) / line;
        // Under whole tiles the finishing pair has one tile's time to add the parts, 3 us each; what that takes longer keeps its accumulator waiting (4096 x
        // 2688, 3584 tokens, two tiles left over, in eight parts each 61 us, three terms).
        const uint64_t adding = kSplitAddCost * (parts - 1), tile = k_blocks * cost_main;
        const uint64_t cost = k_blocks * rounds * cost_main + (line + sharers - 1) / sharers +
                              (rounds ? kSplitCoveredCost + (adding > tile ? adding - tile : 0) : kSplitCost + kSplitPartCost * parts);
        if (cost < least) {
            least = cost;
            best.sharers = static_cast<uint32_t>(sharers);
        }
    }
    if (best.pairs < best.sharers) best.pairs = best.sharers;
    best.ns = static_cast<uint32_t>(least * 10 > UINT32_MAX / 2 ? UINT32_MAX / 2 : least * 10) + kPairLaunchNs;
    return best;
}

// Which token rows the pair kernel takes, and how: all of them or none (the narrow kernel's then, which takes `narrow_ns`). The choice is the quickest
// by the estimates.
struct PairPlan {
    uint32_t token_pairs, tail_columns;
    PairSplit split;
};
inline PairPlan pair_plan(uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t terms, uint32_t all_pairs, uint64_t slots, uint32_t narrow_ns) {
    constexpr uint32_t kTile = 256;
    const uint32_t pairs = (tokens + kTile - 1) / kTile, rest = tokens % kTile;
    if (!all_pairs) return PairPlan{};
    PairPlan best{pairs, 0, pair_split(pairs, 0, rows, cols, terms, all_pairs, slots)};
    if (pairs > 1 && rest != 0 && rest <= kTile / 2) {
        const uint32_t columns = (rest + 31) / 32 * 32;
        const PairPlan tail{pairs - 1, columns, pair_split(pairs - 1, columns, rows, cols, terms, all_pairs, slots)};
        if (tail.split.ns < best.split.ns) best = tail;
    }
    return best.split.ns < narrow_ns ? best : PairPlan{};
}

}  // namespace augur_sm100
