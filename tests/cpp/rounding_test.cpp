// The quantiser's tie correction over every F32 quotient that can matter, and its block-scale quotient over many, against the rules
// they stand for. Prints "ok" last.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "nvfp4_rounding.h"

using namespace augur_sm100::tc;

static float as_float(uint32_t bits) {
    float f;
    memcpy(&f, &bits, 4);
    return f;
}

// The hardware converter's magnitude code: nearest level, a tie to the even code, 7 (6.0) for all above.
static int nearest_even(float a) {
    if (a <= 0.25f) return 0;
    if (a < 0.75f) return 1;
    if (a <= 1.25f) return 2;
    if (a < 1.75f) return 3;
    if (a <= 2.5f) return 4;
    if (a < 3.5f) return 5;
    if (a <= 5.0f) return 6;
    return 7;
}

// The rule: nearest level, a tie to the smaller magnitude.
static int nearest_toward_zero(float a) {
    return (a > 0.25f) + (a > 0.75f) + (a > 1.25f) + (a > 1.75f) + (a > 2.5f) + (a > 3.5f) + (a > 5.0f);
}

int main() {
    uint64_t wrong = 0;
    auto check = [&](float q) {
        const float moved = std::fma(q, kTieNudge, q);
        if (nearest_even(std::fabs(moved)) != nearest_toward_zero(std::fabs(q)) || std::signbit(moved) != std::signbit(q)) ++wrong;
    };
    for (uint32_t bits = 0x3c800000u; bits <= 0x41800000u; ++bits) check(as_float(bits));       // 2^-6 .. 16: every value
    for (uint32_t bits = 1; bits < 0x7f800000u; bits += 0x101u) {                                // the others, thinned, both signs
        check(as_float(bits));
        check(-as_float(bits));
    }
    if (wrong) {
        printf("ties: %llu codes differ\n", static_cast<unsigned long long>(wrong));
        return 1;
    }
    // maximum / (6 g): significands at random, the exponents of both over the whole range that the fast path takes
    uint64_t state = 0x9e3779b97f4a7c15ull, tried = 0;
    auto next = [&]() {
        state ^= state << 13;
        state ^= state >> 7;
        state ^= state << 17;
        return static_cast<uint32_t>(state >> 20);
    };
    for (uint32_t i = 0; i < 20000000u; ++i) {
        const float global = as_float(((62u + next() % 118u) << 23) | (next() & 0x7fffffu));
        uint32_t significand = next() & 0x7fffffu;
        if (i % 4 == 0) significand &= 0x7f0000u;                                                // a BF16 maximum
        const float maximum = as_float(((64u + next() % 127u) << 23) | significand);
        const QuantScale s = quant_scale(global);
        if (s.six_reciprocal == 0.0f) continue;
        ++tried;
        if (quotient_by_reciprocal(maximum, s.six_reciprocal, s.six) != maximum / s.six) ++wrong;
    }
    if (wrong || tried < 15000000u) {
        printf("block scale: %llu of %llu quotients differ\n", static_cast<unsigned long long>(wrong), static_cast<unsigned long long>(tried));
        return 1;
    }
    printf("ok\n");
    return 0;
}
