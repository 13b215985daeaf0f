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
    // Against the pair kernel the time counts, not only the order, and it is an estimate of its own: fitted to 1660 GEMMs of 9 to 4096 tokens and 64 to 34816
    // rows and columns, each by both kernels, as the pair kernel's estimate (pair_split) and the difference of the two times. The meeting of a cluster is
    // 1.26 us per doubling of its CTAs. On 650 GEMMs more the choice between the kernels is 0.4 % off the best on average and 14 % at worst from 1024 rows
    // and columns on below 129 tokens, 22 % beyond; with constants fitted to 130 tokens and more and real layers alone 4.3 %, us now and then: 9600 x 64, 15 tokens, one term
    // 4.3 / 6.5, gate|up 18944 x 1088, 160 tokens, three terms 18.3 / 24.1.
    constexpr uint32_t kMeetNs[kNarrowMaxParts + 1] = {0, 0, 1264, 2003, 2528, 2935, 3267, 3549, 3792};
    const uint64_t waves = (items + clusters[cut.parts] - 1) / clusters[cut.parts], steps = (k_blocks + cut.parts - 1) / cut.parts;
    const uint64_t ns = waves * (2310 + cut.columns * 216 / 10 + kMeetNs[cut.parts] + steps * (112 + terms * (414 + cut.columns * 79 / 100)));
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

// What a k block of a whole tile and of a tail tile counts when leftover tiles are shared out: only the ratio matters.
constexpr uint32_t kPairBlockCost[3] = {52, 93, 118};
inline uint32_t pair_block_cost(uint32_t terms, uint32_t tail_columns) {
    return tail_columns ? 30 + terms * 9 + terms * (tail_columns - 32) * 7 / 100 : kPairBlockCost[terms - 1];
}

// The estimate, in ns, fitted on a B200 to 2560 GEMMs over the sizes of real layers (1024 to 17408 rows and columns, gate|up of twice that with their
// quantiser, 130 to 4096 tokens, one to three terms), each with every choice forced in turn. Tile after tile a pair takes the k blocks, or the epilogue
// where that is longer, which the last tile's follows; a last round of few tiles takes less of its time, since the board's power then goes to fewer SMs.
// A cut costs its pairs their share and a fixed time, more when a share is parts of two tiles, and some per part; the pair that puts a tile together keeps its
// accumulator waiting meanwhile, which a whole tile behind it hides only up to its own time. On 500 GEMMs more the choice is 1.0 % off the best on average
// and 5 % in one of twenty. (With constants fitted to up to 1100 tokens and a cut taken for hidden under whole tiles 4.0 % and 18 %, us now and then: 1536 x
// 6016, 3776 tokens, one term 27.5 / 32.8, gate|up 5120 x 1408, 810 tokens, two terms 13.0 / 22.0, 5376 x 4864, 2773 tokens, three terms 113 / 120.)
constexpr uint32_t kBlockNs[3] = {446, 793, 1134}, kStoreNs = 1180, kQuantiseNs[3] = {3790, 6360, 8360}, kTailStartNs = 980, kPairLaunchNs = 3800;
constexpr uint32_t kLastRoundShare[3] = {706, 857, 872};   // of 1000
constexpr uint32_t kCutNs = 4350, kCutPartNs = 1660, kCutCoveredNs = 800, kCutWaitNs = 9520, kCutWaitPartNs = 3190;
constexpr uint32_t kCutRaggedNs = 3420, kCutQuantiseNs = 3350, kCutTailNs = 4220, kNarrowQuantiseNs = 485;
inline uint64_t pair_tail_block_ns(uint32_t terms, uint32_t tail_columns) { return 169 + 115 * terms + terms * (tail_columns - 32) * 141 / 100; }

// Tiles past the last full round of the pairs (all tiles, when there are fewer tiles than pairs) may be cut along k, in `ways`
// parts each at most and over all pairs at most, when the plan's scratch has a slot for the partial accumulator of each pair that
// shares them (`slots`). `swiglu`: gate and up with the quantiser of as many terms behind them; a launch that stores its BF16 result instead is cut in the
// same way, so that both come to the same bits.
inline PairSplit pair_split(uint32_t token_pairs, uint32_t tail_columns, uint32_t rows, uint32_t cols, uint32_t terms, bool swiglu, uint32_t all_pairs,
                            uint64_t slots) {
    constexpr uint32_t kTile = 256, kDepth = 256;
    const uint32_t n_tiles = (rows + kTile - 1) / kTile, k_blocks = (cols + kDepth - 1) / kDepth;
    const uint32_t main = token_pairs * n_tiles, tail = tail_columns ? n_tiles : 0, rounds = main / all_pairs, left = main % all_pairs;
    const auto larger = [](uint64_t a, uint64_t b) { return a > b ? a : b; };
    const uint64_t out = swiglu ? kQuantiseNs[terms - 1] : kStoreNs, block = kBlockNs[terms - 1], last = k_blocks * block, tile = larger(last, out);
    const uint64_t tail_block = tail ? pair_tail_block_ns(terms, tail_columns) : 0, tail_tile = k_blocks * tail_block + kTailStartNs;
    // not cut: the first pair has the most tiles of either kind
    const uint64_t most_main = (main + all_pairs - 1) / all_pairs, most = (main + tail + all_pairs - 1) / all_pairs, share = kLastRoundShare[terms - 1];
    uint64_t least = most > most_main ? most_main * tile + (most - most_main) * tail_tile : (most - 1) * tile + last;
    if (!tail && left) least = rounds * tile + last * (share * all_pairs + (1000 - share) * left) / (1000 * all_pairs);
    PairSplit best{main + tail < all_pairs ? main + tail : all_pairs, 0, 0};
    const uint64_t cost_main = pair_block_cost(terms, 0), cost_tail = tail ? pair_block_cost(terms, tail_columns) : 0;
    const uint64_t line = k_blocks * (left * cost_main + tail * cost_tail), largest = left ? cost_main : cost_tail;
    uint64_t before = 0;
    for (uint32_t ways = 2; line && ways <= kSplitWays; ++ways) {
        uint64_t sharers = line * ways / (k_blocks * largest);
        if (sharers > all_pairs) sharers = all_pairs;
        if (sharers > line / cost_main) sharers = line / cost_main;      // every range holds a k block
        if (sharers < 2 || (!tail && sharers <= left) || sharers > slots || sharers == before) break;
        before = sharers;
        const uint64_t parts = (sharers * k_blocks * largest + line - 1) / line;
        uint64_t ns = tail ? k_blocks * (left * block + tail * tail_block) / sharers + kCutTailNs : (left * k_blocks + sharers - 1) / sharers * block;
        if (rounds == 0) ns += kCutNs + (parts - 1) * kCutPartNs;
        else ns += kCutCoveredNs + larger(rounds > 1 ? tile : last, kCutWaitNs + (parts - 1) * kCutWaitPartNs) + (rounds > 1 ? (rounds - 2) * tile + last : 0);
        if (!tail && sharers % left) ns += kCutRaggedNs;
        if (swiglu) ns += kCutQuantiseNs;
        if (ns < least) {
            least = ns;
            best.sharers = static_cast<uint32_t>(sharers);
        }
    }
    if (best.pairs < best.sharers) best.pairs = best.sharers;
    least += kPairLaunchNs + out;
    best.ns = static_cast<uint32_t>(least > UINT32_MAX / 2 ? UINT32_MAX / 2 : least);
    return best;
}

// Which token rows the pair kernel takes, and how: all of them or none (the narrow kernel's then, which takes `narrow_ns`). The choice is the quickest
// by the estimates.
struct PairPlan {
    uint32_t token_pairs, tail_columns;
    PairSplit split;
};
inline PairPlan pair_plan(uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t terms, bool swiglu, uint32_t all_pairs, uint64_t slots,
                          uint32_t narrow_ns) {
    constexpr uint32_t kTile = 256;
    const uint32_t pairs = (tokens + kTile - 1) / kTile, rest = tokens % kTile;
    if (!all_pairs) return PairPlan{};
    PairPlan best{pairs, 0, pair_split(pairs, 0, rows, cols, terms, swiglu, all_pairs, slots)};
    if (pairs > 1 && rest != 0 && rest <= kTile / 2) {
        const uint32_t columns = (rest + 31) / 32 * 32;
        const PairPlan tail{pairs - 1, columns, pair_split(pairs - 1, columns, rows, cols, terms, swiglu, all_pairs, slots)};
        if (tail.split.ns < best.split.ns) best = tail;
    }
    return best.split.ns < narrow_ns + (swiglu ? terms * kNarrowQuantiseNs : 0) ? best : PairPlan{};
}

}  // namespace augur_sm100
