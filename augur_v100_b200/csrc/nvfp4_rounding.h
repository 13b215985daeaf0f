// The rounding steps of the activation quantiser that rest on exact arithmetic, in one place for the kernels and for the comparison of
// them, over every value or many, that runs on the host. Plain C++ outside nvcc.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define AUGUR_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define AUGUR_HOST_DEVICE inline
#endif

namespace augur_sm100 {
namespace tc {

// What every quotient is moved by, relative to itself, ahead of the hardware's E2M1 converter, so that its ties ("to even") come out as
// the rule has them ("toward zero"). At 0.75, 1.75 and 3.5 "even" is the larger level; at the other ties it is the smaller
// one. The three have a significand of 1.5 or 1.75, the others of 1 or 1.25. q - q * 1.457 * 2^-25 takes 0.364 m of an ulp off a
// quotient with significand m, which rounds to the neighbour nearer to zero once it exceeds half of one: for m above 1.37, and for
// exact powers of two, below which an ulp is half as large. A tie of the three then lies below itself, the value one ulp above
// it on the tie, which rounds up as it must; a power of two moves within the level that it belongs to (0.25 is a tie and goes to
// zero either way); and no other boundary has values so close.
constexpr float kTieNudge = -0x1.75p-25f;

// x / d, correctly rounded, from y = RN(1 / d): two steps of Newton's method on the quotient, each with an exact FMA residual
// (Markstein's theorem), for normal x, d and quotients well inside the range, d not of the all-ones significand.
AUGUR_HOST_DEVICE float quotient_by_reciprocal(float x, float y, float d) {
#ifdef __CUDA_ARCH__
    float q = __fmul_rn(x, y);
    q = __fmaf_rn(__fmaf_rn(q, -d, x), y, q);
    return __fmaf_rn(__fmaf_rn(q, -d, x), y, q);
#else
    float q = x * y;
    q = std::fma(std::fma(q, -d, x), y, q);
    return std::fma(std::fma(q, -d, x), y, q);
#endif
}

// What a quantiser knows about its global scale before it has seen an element: 6 g, and its rounded reciprocal where
// quotient_by_reciprocal is exact for a `maximum` from 2^-63 to 2^64 (0 where it need not be).
struct QuantScale {
    float global, six, six_reciprocal;
};
inline QuantScale quant_scale(float global_scale) {
    const float six = 6.0f * global_scale;
    uint32_t bits;
    memcpy(&bits, &six, 4);
    const uint32_t field = bits >> 23;
    return QuantScale{global_scale, six, field >= 64u && field <= 180u && (bits & 0x7fffffu) != 0x7fffffu ? 1.0f / six : 0.0f};
}

}  // namespace tc
}  // namespace augur_sm100
