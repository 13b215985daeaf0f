// How the pair GEMM's launch shares its work out between pairs of CTAs: what a pair does, in which order. In one place for the kernel
// and for the check on the host that every part of every tile is done once. Plain C++ outside nvcc.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define AUGUR_PAIR_FN __host__ __device__ __forceinline__
#else
#define AUGUR_PAIR_FN inline
#endif

namespace augur_sm100 {

// The work of one CTA pair, in the order it is done: the head or middle part of a leftover tile (its partial
// accumulator is handed to the pair that finishes the tile), the part that finishes a leftover tile, leftover tiles that are
// this pair's alone, then its full rounds of main tiles. A part handed over is its pair's first item and nothing waits
// in front of it; a finishing part follows, and only its epilogue warps wait (for first items of other pairs, about as long as
// its own), with the accumulator already released; the reads of the handed-over sums then run under the
// MMAs of the whole tiles that follow.
struct PairItem {
    uint32_t tile, kb0, kb1;
    uint32_t kind;           // 0: whole tile, 1: part handed over, 2: part that finishes the tile
    uint32_t first_giver;    // kind 2: the pairs first_giver .. this pair - 1 hand their parts over
};

// `main` tiles are numbered first, `tail` tiles after them. Whole rounds of main tiles go to pair p as p, p + pairs, ...; what is left,
// main tiles past the last full round and all tail tiles, is one line of k blocks, which the first `sharers` pairs cut into ranges of
// equal cost (cost_main or cost_tail a k block), each range at least the larger of the two. A range holds the tail of one tile, whole
// ones, the head of another, or the middle of one. Without sharers every tile is one pair's, the tail tiles last.
struct PairShares {
    uint32_t main, tail;              // tiles
    uint32_t k_blocks, sharers;
    uint32_t cost_main, cost_tail;
};

struct PairWork {
    uint32_t items, alone, first_alone;   // `alone`: whole leftover tiles from `first_alone` on
    PairItem given, finishing;
    bool gives, finishes;
    // k blocks of all items
    AUGUR_PAIR_FN uint32_t blocks(uint32_t k_blocks) const {
        const uint32_t parts = (gives ? 1u : 0u) + (finishes ? 1u : 0u);
        return (items - parts) * k_blocks + (gives ? given.kb1 - given.kb0 : 0) + (finishes ? finishing.kb1 - finishing.kb0 : 0);
    }
    AUGUR_PAIR_FN PairItem item(uint32_t index, uint32_t pair, uint32_t pairs, uint32_t k_blocks) const {
        const uint32_t parts = (gives ? 1u : 0u) + (finishes ? 1u : 0u);
        if (gives && index == 0) return given;
        if (finishes && index + 1 == parts) return finishing;
        if (index < parts + alone) return PairItem{first_alone + index - parts, 0, k_blocks, 0, 0};
        return PairItem{pair + (index - parts - alone) * pairs, 0, k_blocks, 0, 0};
    }
};

AUGUR_PAIR_FN PairWork pair_work(uint32_t pair, uint32_t pairs, const PairShares& s) {
    PairWork w{};
    if (!s.sharers) {
        const uint32_t tiles = s.main + s.tail;
        w.items = tiles > pair ? (tiles - pair + pairs - 1) / pairs : 0;
        return w;
    }
    const uint32_t rounds = s.main / pairs;
    w.items = rounds;
    if (pair >= s.sharers) return w;
    const uint32_t first_left = rounds * pairs, left_main = s.main - first_left;
    const uint64_t main_cost = static_cast<uint64_t>(left_main) * s.k_blocks * s.cost_main;
    const uint64_t cost = main_cost + static_cast<uint64_t>(s.tail) * s.k_blocks * s.cost_tail;
    // k blocks of the line that lie wholly before a point of the cost
    auto before = [&](uint64_t x) {
        return static_cast<uint32_t>(x < main_cost ? x / s.cost_main : static_cast<uint64_t>(left_main) * s.k_blocks + (x - main_cost) / s.cost_tail);
    };
    const uint32_t b0 = before(pair * cost / s.sharers), b1 = before((pair + 1) * cost / s.sharers);   // this pair's range, not empty
    const uint32_t a = b0 / s.k_blocks, b = (b1 - 1) / s.k_blocks, a_begin = a * s.k_blocks, b_begin = b * s.k_blocks;
    if (b1 >= a_begin + s.k_blocks) {
        // the range holds the tail of tile a: every pair from the one that owns the tile's first k block hands over
        const bool main_tile = a < left_main;
        const uint64_t first_done = main_tile ? (static_cast<uint64_t>(a_begin) + 1) * s.cost_main
                                              : main_cost + (static_cast<uint64_t>(a_begin - left_main * s.k_blocks) + 1) * s.cost_tail;
        w.finishes = true;
        w.finishing = PairItem{first_left + a, b0 - a_begin, s.k_blocks, 2, static_cast<uint32_t>((first_done * s.sharers - 1) / cost)};
        if (w.finishing.first_giver == pair) w.finishing.kind = 0;   // the whole tile
    } else {
        w.gives = true;
        w.given = PairItem{first_left + a, b0 - a_begin, b1 - a_begin, 1, 0};
    }
    if (b > a) {
        const bool ends = b1 == b_begin + s.k_blocks;   // the range ends with tile b
        w.first_alone = first_left + a + 1;
        w.alone = b - a - (ends ? 0u : 1u);
        if (!ends) {
            w.gives = true;
            w.given = PairItem{first_left + b, 0, b1 - b_begin, 1, 0};
        }
    }
    w.items = rounds + w.alone + (w.gives ? 1u : 0u) + (w.finishes ? 1u : 0u);
    return w;
}

}  // namespace augur_sm100
