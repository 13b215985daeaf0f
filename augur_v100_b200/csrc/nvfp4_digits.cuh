// BF16 activations of 1..8 token rows as eight NVFP4 terms, the digits of the value in radix 8: the layout of the split in
// memory and the device code that writes it, shared by the small-token kernels on tensor memory.
#pragma once

#include <cstdint>

#include "nvfp4_layout.cuh"
#include "nvfp4_tc.cuh"

namespace augur_sm100 {
namespace tc {

constexpr uint32_t kTerms = 8;                         // radix-8 digits of the activation split
constexpr uint32_t kCols = 8 * kTerms;                 // MMA n: column = term * 8 + token
constexpr uint32_t kStageK = 256;                      // k per ring stage = one 128-byte swizzled row of codes
constexpr uint32_t kStageCodeBytes = kTileM * 128;     // 16 KB of weight codes
constexpr uint32_t kStageSfBytes = 4 * kSfAtomBytes;   // 2 KB: the 4 scale atoms of a stage (weights; activations alike)
constexpr uint32_t kChunkBytes = kCols * 128;          // 8 KB: activation codes of one 256-k chunk, 64 rows x 128 bytes

// The split activations in global memory (plan scratch): the image the ring stages want, chunk by chunk.
//   [chunk = k / 256][64 rows][128 bytes]   codes, rows already in the 128-byte swizzle of a shared-memory operand tile
//   [k / 64][512 bytes]                     block-scale atoms (row n at byte (n % 32) * 16 + (n / 32) * 4 + (k / 16) % 4)
__host__ __device__ constexpr uint64_t split_code_bytes(uint32_t cols) { return static_cast<uint64_t>((cols + kStageK - 1) / kStageK) * kChunkBytes; }
__host__ __device__ constexpr uint64_t split_sf_bytes(uint32_t cols) { return static_cast<uint64_t>((cols + kStageK - 1) / kStageK) * kStageSfBytes; }
__host__ __device__ constexpr uint64_t split_bytes(uint32_t cols) { return split_code_bytes(cols) + split_sf_bytes(cols); }

// ---- activation split ----
// One lane per element, sixteen neighbouring lanes per 16-element group. With A the exponent field of the largest magnitude
// of the token row (of what is split together) and G that of the group's, the group's block scale is 2^q, q = G + 8 - A (the row's
// largest group gets 2^8; E4M3 holds powers of two down to 2^-9, smaller groups keep 2^-9 and lose low bits),
// term t has the global scale 2^(A - 155) * 8^t (times the level, half the digit), and the element is the integer I = |x| / 2^(q + A - 156): at
// most 255 * 2^14 for the group's largest element, exact for every element within 2^-14 of it, rounded to
// nearest below. I is written in radix 8 with digits -4..3: I plus 4 in every octal place has the digits plus 4
// as its octal digits (eight of them: 3 * (8^8 - 1) / 7 > 255 * 2^14). Digit t is the code of term t: level
// |digit| / 2, sign of digit times sign of x; all eight are formed at once in the nibbles of one word. The eight
// lanes of a half group transpose their words so that lane t holds the eight codes of term t, and store one
// word each.
struct SplitTarget {
    uint8_t* split;               // the phase's split activations
    uint32_t sf_offset;           // of its block-scale atoms
    uint32_t group0, groups;      // the job's groups of every token row
    uint32_t tokens;
};

// (Both halves are real functions, not inlined: the code that runs at the boundary between the two products is
// then the code the launch has already run for its input, and is still in the instruction cache.)
// First half of a group's split, before the row's anchor is known: the group's largest magnitude (returned), the
// digits relative to it (`drop` low bits fewer), the codes stored. Whole warps; `index` past the job is inactive.
static __device__ __noinline__ uint32_t split_codes(const SplitTarget to, uint2 where, uint32_t bits, uint32_t drop, uint32_t lane) {
    const bool active = where.x != ~0u;
    const uint32_t token = active ? where.x : 0, group = where.y;
    const uint32_t magnitude = bits & 0x7fffu, negative = (bits >> 15) & 1u;
    uint32_t largest = max(magnitude, __shfl_xor_sync(0xffffffffu, magnitude, 8));
    largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, 4));
    largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, 2));
    largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
    const int g = max(static_cast<int>(largest >> 7), 1);           // a subnormal has the exponent of field 1
    const uint32_t field = magnitude >> 7;
    const uint32_t significand = field ? 128u + (magnitude & 127u) : magnitude;
    // |x| = significand * 2^(max(field, 1) - 134); I = |x| * 2^(156 - q - A) = significand * 2^(field - G + 14) with q = G + 8 - A
    const int shift = max(static_cast<int>(max(field, 1u)) - g + 14 - static_cast<int>(drop), -16);
    const uint32_t value = shift >= 0 ? significand << shift : (significand + (1u << (-shift - 1))) >> -shift;
    // octal digits of I + 44444444 (octal), one per nibble: d = digit + 4 in 0..7
    uint32_t d = (value + 0x924924u) & 0xffffffu;
    d = (d & 0x00000fffu) | ((d & 0x00fff000u) << 4);
    d = (d & 0x003f003fu) | ((d & 0x0fc00fc0u) << 2);
    d = (d & 0x07070707u) | ((d & 0x38383838u) << 1);
    // level = |d - 4|: d & 3 where d >= 4, else 4 - d = (~d & 3) + 1; the digit is negative where d < 4
    const uint32_t upper = (d >> 2) & 0x11111111u, upper_mask = upper * 15u;
    const uint32_t level = ((d & 0x33333333u) & upper_mask) | (((~d & 0x33333333u) + 0x11111111u) & ~upper_mask);
    const uint32_t nonzero = (level | (level >> 1) | (level >> 2)) & 0x11111111u;
    const uint32_t minus = ((upper ^ 0x11111111u) ^ (negative * 0x11111111u)) & nonzero;
    uint32_t digits = level | (minus << 3);    // code of term t in bits 4t .. 4t + 3
    // 8 lanes x 8 nibbles, transposed: lane t of the eight ends up with nibble t of all eight, in lane order
    uint32_t other = __shfl_xor_sync(0xffffffffu, digits, 4);
    digits = (lane & 4) ? (other >> 16) | (digits & 0xffff0000u) : (digits & 0x0000ffffu) | (other << 16);
    other = __shfl_xor_sync(0xffffffffu, digits, 2);
    digits = (lane & 2) ? ((other & 0xff00ff00u) >> 8) | (digits & 0xff00ff00u) : (digits & 0x00ff00ffu) | ((other & 0x00ff00ffu) << 8);
    other = __shfl_xor_sync(0xffffffffu, digits, 1);
    digits = (lane & 1) ? ((other & 0xf0f0f0f0u) >> 4) | (digits & 0xf0f0f0f0u) : (digits & 0x0f0f0f0fu) | ((other & 0x0f0f0f0fu) << 4);
    // lanes t and t + 8 hold the two words of the group's eight bytes in row n = t * 8 + token
    other = __shfl_xor_sync(0xffffffffu, digits, 8);
    if (active && (lane & 8) == 0) {
        const uint32_t n = (lane & 7) * 8 + token, chunk = group >> 4, unit = (group & 15) >> 1, half = group & 1;
        uint8_t* codes = to.split + static_cast<uint64_t>(chunk) * kChunkBytes + (n >> 3) * 1024 + (n & 7) * 128 + ((unit ^ (n & 7)) << 4);
        *reinterpret_cast<uint2*>(codes + half * 8) = make_uint2(digits, other);
    }
    return largest;
}

// Second half, with the row's anchor: the group's block scale 2^q, q = G + 8 - A. A group more than 2^17 below its
// row's largest magnitude keeps 2^-9 and has its codes redone with that many low bits fewer (rare). True if the
// group is larger than the anchor provides for (an anchor that was guessed).
static __device__ __noinline__ bool split_scales(const SplitTarget to, const uint32_t* anchor, uint2 where, uint32_t bits, uint32_t largest,
                                          uint32_t lane) {
    const bool active = where.x != ~0u;
    const uint32_t token = active ? where.x : 0, group = where.y;
    const int q = max(static_cast<int>(largest >> 7), 1) + 8 - static_cast<int>(anchor[token]);
    const uint32_t drop = active && q < -9 ? static_cast<uint32_t>(-9 - q) : 0u;
    if (__any_sync(0xffffffffu, drop != 0)) split_codes(to, where, bits, drop, lane);
    if (active && (lane & 8) == 0) {
        const int clamped = min(max(q, -9), 8);
        const uint32_t scale_code = clamped >= -6 ? static_cast<uint32_t>(clamped + 7) << 3 : 1u << (clamped + 9);
        const uint32_t n = (lane & 7) * 8 + token;
        uint8_t* sf = to.split + to.sf_offset + static_cast<uint64_t>(group >> 2) * kSfAtomBytes + (group & 3);
        sf[(n & 31) * 16 + (n >> 5) * 4] = static_cast<uint8_t>(scale_code);
    }
    return active && q > 8;   // the group is larger than the anchor allows for
}

}  // namespace tc
}  // namespace augur_sm100
