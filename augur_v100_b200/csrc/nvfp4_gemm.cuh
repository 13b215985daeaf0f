// What the prefill GEMM kernels share: launch parameters, accumulator conversion and the tensor map of packed codes.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "nvfp4_internal.h"
#include "nvfp4_layout.cuh"
#include "nvfp4_tc.cuh"

namespace augur_sm100 {

struct GemmParams {
    const uint8_t* weight_sf;      // scale region of the weight tensor
    const uint8_t* act_sf;         // scale region of term 0; terms are `act_term_stride` bytes apart
    uint64_t act_term_stride;
    __nv_bfloat16* out;
    uint32_t* status_word;
    uint32_t rows, cols, tokens, terms;
    uint32_t token_pairs;          // 256-token row pairs of the pair kernel's launch
    uint32_t tail_columns;         // tokens past them, in steps of 32 (0: none), on tail tiles
    uint32_t cost_main, cost_tail; // of a k block of a whole tile and of a tail tile, for the balance of the leftover tiles
    uint32_t padded_tokens;        // tokens rounded up to whole 128-row tiles: row stride of the staged activation planes
    float scale;                   // g_w * g_a
    float scale_b;                 // SwiGLU: g_w of the up rows * g_a
    uint32_t swiglu;               // weight rows alternate 16 gate / 16 up; output is bf16(silu(gate) * up), rows / 2 wide
    // SwiGLU: the intermediate is also (or only, if `out` is null) quantised for the next GEMM
    uint8_t* quant_out;            // staged activations: [terms] code planes of whole tiles, then the scale regions
    uint32_t quant_terms;
    tc::QuantScale quant_scale;
    // Pair tiles whose count is not a multiple of the pairs: the tiles left over are cut along k between all pairs
    // (null: whole tiles only). Partial accumulators pass through `split_slots`, announced by `split_flags`.
    float* split_slots;            // [pair][CTA of the pair][epilogue warp][128 columns / 4][lane] x float4
    uint32_t* split_flags;         // [pair][CTA of the pair][epilogue warp], zero between launches
    uint32_t split_sharers;        // pairs that share the leftover tiles (0: whole tiles only)
};

__host__ __device__ constexpr uint32_t padded_tokens(uint32_t tokens) { return (tokens + tc::kTileM - 1) / tc::kTileM * tc::kTileM; }
// Bytes of the staged activations of one term: code plane of whole tiles, then the scale atoms.
__host__ __device__ constexpr uint64_t staged_term_bytes(uint32_t tokens, uint32_t cols) {
    return tcgen05_extent_bytes(padded_tokens(tokens), cols);
}


// 32 accumulator columns of one token row -> packed BF16. Plain: 32 outputs. SwiGLU: the weight rows
// alternate 16 gate / 16 up, so columns 0..15 are gate sums and 16..31 the matching up sums of 16
// intermediate columns; the 16 outputs bf16(silu(gate) * up) fill packed[0..8).
__device__ __forceinline__ void convert_chunk(const uint32_t (&v)[32], float scale, float scale_b, bool swiglu, uint32_t (&packed)[16]) {
    if (!swiglu) {
#pragma unroll
        for (uint32_t i = 0; i < 16; ++i) {
            const __nv_bfloat162 two = __floats2bfloat162_rn(__uint_as_float(v[2 * i]) * scale, __uint_as_float(v[2 * i + 1]) * scale);
            packed[i] = *reinterpret_cast<const uint32_t*>(&two);
        }
        return;
    }
    float h[16];
#pragma unroll
    for (uint32_t i = 0; i < 16; ++i) {
        const float gate = __uint_as_float(v[i]) * scale, up = __uint_as_float(v[16 + i]) * scale_b;
        // fast exponential and reciprocal (a few 1e-7 relative): this runs between the accumulator read and
        // its release, in front of the next tile's MMAs. A gate below -87 gives exp = inf and h = -0.
        h[i] = __fdividef(gate, 1.0f + __expf(-gate)) * up;
    }
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const __nv_bfloat162 two = __floats2bfloat162_rn(h[2 * i], h[2 * i + 1]);
        packed[i] = *reinterpret_cast<const uint32_t*>(&two);
    }
}

// Packed codes as a 2-D byte tensor [rows][cols/2]; boxes of `box_rows` rows x 128 bytes, 128-byte swizzle. A host-side
// computation: no allocation and no device access.
bool make_code_map(CUtensorMap* map, uint64_t address, uint64_t rows, uint32_t cols, uint32_t box_rows = 128);

// The GEMM for token counts that are narrow next to the weights (csrc/nvfp4_gemm_narrow.cu). `map_weight`: boxes of 128 rows.
augur_cuda_result_v1 launch_gemm_narrow(augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_plan_v1* plan, const CUtensorMap& map_weight,
                                        uint64_t activation, const GemmParams& p);
// About how long it takes.
uint32_t gemm_narrow_ns(int32_t ordinal, uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t terms);

}  // namespace augur_sm100
