// Prefill NVFP4 linear for sm_100a: BF16 -> NVFP4 activation quantiser and a
// warp-specialised tcgen05 block-scaled GEMM (kind::mxf4nvf4, scale_vec::4X) with
// TMA-fed shared-memory stages and the accumulator in tensor memory.
//
// D[token][feature] = g_w * g_a * sum_terms sum_k A_term[token][k] * W[feature][k]
//   A operand: quantised activations, 256 token rows per tile on two CTAs
//   B operand: weights, 256 feature rows per tile (128 in a half tile at the end)
//   both K-major, packed two E2M1 codes per byte, 128-byte swizzled rows of 256 k
//   block scales: 512-byte atoms (128 rows x 4 scales) copied smem -> TMEM by tcgen05.cp
//
// Every mbarrier wait is bounded: a wait that runs out records a code in the plan's status word, raises a CTA-wide
// abort flag, and all roles fall through to the common exit where tensor memory is released.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>


#include "nvfp4_gemm.cuh"
#include "nvfp4_gemm_choice.h"
#include "nvfp4_internal.h"
#include "nvfp4_layout.cuh"
#include "nvfp4_pair_work.h"
#include "nvfp4_tc.cuh"

namespace augur_sm100 {
namespace {
using namespace tc;

static_assert(sizeof(augur_cuda_nvfp4_sm100_act_quant_args_v1) == 56, "act_quant ABI");
static_assert(sizeof(augur_cuda_nvfp4_sm100_gemm_args_v1) == 80, "gemm ABI");

constexpr uint32_t kTileN = 256;          // features per tile (128 for a half tile at the end)
constexpr uint32_t kBlockK = 256;         // k per shared-memory stage = one 128-byte swizzled row
constexpr uint32_t kBytesA = kTileM * 128;            // 16 KB
constexpr uint32_t kBytesSfA = 4 * kSfAtomBytes;      // 2 KB: 4 atoms (k) of one 128-row block
constexpr uint32_t kBytesSfB = 8 * kSfAtomBytes;      // 4 KB: 2 row blocks x 4 atoms
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTmemAcc = 0;          // 256 accumulator columns

constexpr uint32_t kErrProducerWait = 0x101, kErrMmaWaitTokens = 0x102, kErrMmaWaitTmem = 0x103,
                   kErrEpilogueWait = 0x104, kErrCopyWait = 0x105, kErrMmaWaitWeights = 0x106,
                   kErrSplitWait = 0x107;

// ---- two-CTA tiles ------------------------------------------------------------------------------
// A 128 x 256 tile on one CTA pulls 54 KB through L2 -> shared memory per 256-deep k block, and that
// path, not the tensor pipe, would bound it. Here two CTAs of a cluster (a pair of SMs) share one
// 256 x 256 tile with tcgen05 cta_group::2: each CTA loads its own 128 token rows (A), its own
// half of the 256 weight rows (B) and the scales of both, 38 KB per k block for the same
// 128 x 256 x 256 of arithmetic per SM. The even CTA of the pair (the leader) issues the MMAs for
// both; each CTA's accumulator half sits in its own tensor memory and is drained by its own
// epilogue warps.
//
// Two rings per CTA: a weight stage (20 KB) holds a k block's weight rows and their scales for all activation terms, a token
// slot (18 KB) one term of it. What bounds the kernel is the board's power (SM clock 1.5 to 1.65 GHz under it) and, within it,
// about 150 cycles per MMA: so bytes that need not move into shared memory are time. With one ring, whose stages brought the
// weights again for every term, three terms of 17408 x 5120 x 4096 took 434 us (GEMM alone; 457 in a long loop), with two
// 384 (418), two terms 291 -> 272; 5120 x 17408 x 777, three terms, 114 -> 97.
//
// Barriers per slot of a ring (same offsets in both CTAs):
//   landed  leader's only: the slot's block-scale atoms of both CTAs have landed (loaded before the operand tiles);
//   full    leader's only: two arrivals, the leader's producer (expecting the operand bytes of both CTAs; both producers' TMA
//           loads complete on it: cta_group::2 loads, leader's address) and the commit behind the copy warp's shared -> tensor
//           memory copies of the slot's scales, which says that they are done;
//   empty   token slots only, one per CTA, arrived by the leader's tcgen05.commit multicast to both CTAs.
// And: tmem_full one per CTA, same multicast;   tmem_empty leader's only, one arrival per epilogue warp of either CTA (the
// peer's through a cluster-scope arrive).
constexpr uint32_t kPairBytesB = 128 * 128;                          // this CTA's 128 weight rows
constexpr uint32_t kPairWeightStage = kPairBytesB + kBytesSfB;       // 20480
constexpr uint32_t kPairTokenSlot = kBytesA + kBytesSfA;             // 18432
constexpr uint32_t kPairMaxDepth = 8;                                // slots of either ring
// Ring depths by activation terms: about as many k blocks ahead on either ring as shared memory holds. A weight stage is
// free when the last term's step of its k block is complete, which the wait for a token slot of a later step says (no barrier and no
// commit of its own: a second commit per step, and scales that queue behind codes, took one term from 157 to 178 us): the slot of
// term `weight_term` of block b was last used by that step of block b - weights, or by a later one.
struct PairDepths {
    uint32_t weights, tokens;
};
__host__ __device__ constexpr PairDepths pair_depths(uint32_t terms) {
    return terms == 1 ? PairDepths{5, 5} : terms == 2 ? PairDepths{4, 6} : PairDepths{3, 8};
}
__host__ __device__ constexpr uint32_t pair_weight_term(uint32_t terms) {
    const uint32_t before = (pair_depths(terms).weights - 1) * terms + 1;
    return pair_depths(terms).tokens > before ? pair_depths(terms).tokens - before : 0;
}
static_assert(pair_weight_term(1) < 1 && pair_weight_term(2) < 2 && pair_weight_term(3) < 3, "a freed weight stage shows in the token ring");
__host__ __device__ constexpr uint32_t pair_ring_bytes(uint32_t terms) {
    return pair_depths(terms).weights * kPairWeightStage + pair_depths(terms).tokens * kPairTokenSlot;
}
constexpr uint32_t kPairRingBytes = pair_ring_bytes(3);              // the largest: 208896
static_assert(pair_ring_bytes(1) <= kPairRingBytes && pair_ring_bytes(2) <= kPairRingBytes, "space for the rings");
// Tensor memory of the pair kernel: 256 accumulator columns, then one set of weight-row scale columns per weight stage
// (32 each) and one set of token-row scale columns per token slot (16 each).
constexpr uint32_t kTmemPairScales = 256;
constexpr uint32_t pair_tmem_columns(uint32_t terms) { return kTmemPairScales + pair_depths(terms).weights * 32 + pair_depths(terms).tokens * 16; }
static_assert(pair_tmem_columns(1) <= kTmemCols && pair_tmem_columns(2) <= kTmemCols && pair_tmem_columns(3) <= kTmemCols,
              "scale columns of both rings fit beside the accumulator");
// Epilogue transposition rows: an epilogue warp holds one accumulator row per lane; to store row pieces that are
// contiguous in global memory it parks one 32-column chunk (64 bytes of BF16 per row, rows padded by 16 bytes so
// that the row-per-lane writes spread over all banks) and reads it back with 4 lanes per row.
constexpr uint32_t kPairEpilogueWarps = 8;      // two per tensor-memory lane quadrant
constexpr uint32_t kPairOutRowBytes = 64 + 16;
constexpr uint32_t kPairOutBytes = kPairEpilogueWarps * 32 * kPairOutRowBytes;         // 20480
constexpr uint32_t kPairBarriers = 5 * kPairMaxDepth + 2;
constexpr uint32_t kPairSmemBytes = kPairRingBytes + kPairOutBytes + 1024 + 512;
static_assert(kPairSmemBytes <= 227 * 1024, "shared memory of a CTA");
constexpr uint32_t kPairCopyWarp = 2 + kPairEpilogueWarps;    // token-row scales; the warp after it copies the weight-row scales
constexpr uint32_t kPairThreads = 32 * (kPairCopyWarp + 2);   // TMA warp, MMA warp, epilogue warps, two scale-copy warps
static_assert(kPairBarriers * 8 + 8 + kPairThreads / 32 * 4 + sizeof(PairWork) <= 512, "barriers, tensor-memory base, abort flag, the warps' counters and the pair's work fit behind the rings");
constexpr uint32_t kSplitWaitLimit = 1u << 20;  // polls of a handed-over part's flag (each a round trip to L2) before giving up
constexpr uint64_t kSplitSlotBytes = 2ull * kPairEpilogueWarps * 32 * 128 * 4;   // one pair's accumulator: 256 x 256 f32
constexpr uint32_t kLeaderMask = 0xFEFFFFFFu;   // clears the CTA-rank bit of a shared::cluster address within a pair

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The TMA loads of a converged warp for one slot of the token ring, and for one stage of the weight ring: block scales first, on a
// barrier of their own, then operand rows, all counted on barriers of the pair's leader CTA (cta_group::2), whose producer (`leader`)
// announces the bytes of both CTAs. As predicated instructions in one block, for the reason given at tc_step.
__device__ __forceinline__ void tma_token_step(bool leader, uint32_t landed, uint32_t scales, const CUtensorMap* map_scales, uint32_t scale_y,
                                               uint32_t scale_z, uint32_t full, uint32_t bytes, uint32_t codes, const CUtensorMap* map_codes, uint32_t x, uint32_t y) {
    asm volatile(
        "{\n.reg .pred e, l;\nelect.sync _|e, 0xffffffff;\nsetp.ne.and.b32 l, %0, 0, e;\n"
        "@l mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %2;\n"
        "@e cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%3], [%4, {%5, %6, %7}], [%8];\n"
        "@l mbarrier.arrive.expect_tx.shared::cta.b64 _, [%9], %10;\n"
        "@e cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%11], [%12, {%13, %14}], [%15];\n}"
        ::"r"(leader ? 1u : 0u), "r"(landed), "r"(2 * kBytesSfA), "r"(scales), "l"(map_scales), "r"(0u), "r"(scale_y), "r"(scale_z), "r"(landed & kLeaderMask),
          "r"(full), "r"(bytes), "r"(codes), "l"(map_codes), "r"(x), "r"(y), "r"(full & kLeaderMask)
        : "memory");
}
__device__ __forceinline__ void tma_weight_step(bool leader, uint32_t landed, uint32_t scales, const CUtensorMap* map_scales, uint32_t scale_y,
                                                uint32_t scale_z, uint32_t full, uint32_t codes, const CUtensorMap* map_codes, uint32_t x, uint32_t y) {
    asm volatile(
        "{\n.reg .pred e, l;\nelect.sync _|e, 0xffffffff;\nsetp.ne.and.b32 l, %0, 0, e;\n"
        "@l mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %2;\n"
        "@e cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%3], [%4, {%5, %6, %7}], [%8];\n"
        "@l mbarrier.arrive.expect_tx.shared::cta.b64 _, [%9], %10;\n"
        "@e cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%11], [%12, {%13, %14}], [%15];\n}"
        ::"r"(leader ? 1u : 0u), "r"(landed), "r"(2 * kBytesSfB), "r"(scales), "l"(map_scales), "r"(0u), "r"(scale_y), "r"(scale_z), "r"(landed & kLeaderMask),
          "r"(full), "r"(2 * kPairBytesB), "r"(codes), "l"(map_codes), "r"(x), "r"(y), "r"(full & kLeaderMask)
        : "memory");
}
// Arrives on the barrier at this offset in both CTAs of the pair once the MMAs issued so far are done.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(static_cast<uint16_t>(3))
                 : "memory");
}
// A step of a converged warp, as tc_step: the one to four MMAs of a k block (64 k each: 32 bytes further in every operand row,
// `step_a` and `step_b` scale columns further) and the commit that frees what they read. `a` and `b` are the low words of operand
// descriptors, whose high words are all alike.
__device__ __forceinline__ void tc_step_pair(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t step_a,
                                             uint32_t step_b, uint32_t accumulate, uint32_t k_steps, uint32_t done) {
    constexpr uint32_t kHigh = (1024 >> 4) | (1u << 14) | (2u << 29);
    asm volatile(
        "{\n.reg .pred e, p, q, e1, e2, e3;\n.reg .b64 a0, a1, a2, a3, b0, b1, b2, b3;\n.reg .b32 l1, l2, l3, m1, m2, m3, s1, s2, s3, t1, t2, t3;\n"
        "tcgen05.fence::after_thread_sync;\nelect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %8, 0;\nsetp.eq.u32 q, 0, 0;\n"
        "setp.gt.and.u32 e1, %9, 1, e;\nsetp.gt.and.u32 e2, %9, 2, e;\nsetp.gt.and.u32 e3, %9, 3, e;\n"
        "add.s32 l1, %1, 2;\nadd.s32 l2, %1, 4;\nadd.s32 l3, %1, 6;\nadd.s32 m1, %2, 2;\nadd.s32 m2, %2, 4;\nadd.s32 m3, %2, 6;\n"
        "mov.b64 a0, {%1, %11};\nmov.b64 a1, {l1, %11};\nmov.b64 a2, {l2, %11};\nmov.b64 a3, {l3, %11};\n"
        "mov.b64 b0, {%2, %11};\nmov.b64 b1, {m1, %11};\nmov.b64 b2, {m2, %11};\nmov.b64 b3, {m3, %11};\n"
        "add.s32 s1, %4, %6;\nadd.s32 s2, s1, %6;\nadd.s32 s3, s2, %6;\nadd.s32 t1, %5, %7;\nadd.s32 t2, t1, %7;\nadd.s32 t3, t2, %7;\n"
        "@e tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], a0, b0, %3, [%4], [%5], p;\n"
        "@e1 tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], a1, b1, %3, [s1], [t1], q;\n"
        "@e2 tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], a2, b2, %3, [s2], [t2], q;\n"
        "@e3 tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], a3, b3, %3, [s3], [t3], q;\n"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%10], %12;\n}"
        ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(step_a), "r"(step_b), "r"(accumulate), "r"(k_steps), "r"(done), "r"(kHigh),
          "h"(static_cast<uint16_t>(3))
        : "memory");
}
// The scale atoms of a slot, four k steps of one 128-row block or of two (2 KB apart), on their way to both CTAs' tensor memory, four columns an
// atom, those of one k step side by side; and the arrival that says so.
template <uint32_t kBlocks>
__device__ __forceinline__ void tc_copy_step_pair(uint32_t columns, uint64_t desc, uint32_t ready) {
    static_assert(kSfAtomBytes >> 4 == 32, "steps of the descriptors below");
    if (kBlocks == 1) {
        asm volatile(
            "{\n.reg .pred e;\n.reg .b64 a1, a2, a3;\n.reg .b32 c1, c2, c3;\ntcgen05.fence::after_thread_sync;\nelect.sync _|e, 0xffffffff;\n"
            "add.s64 a1, %1, 32;\nadd.s64 a2, %1, 64;\nadd.s64 a3, %1, 96;\nadd.s32 c1, %0, 4;\nadd.s32 c2, %0, 8;\nadd.s32 c3, %0, 12;\n"
            "@e tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;\n@e tcgen05.cp.cta_group::2.32x128b.warpx4 [c1], a1;\n"
            "@e tcgen05.cp.cta_group::2.32x128b.warpx4 [c2], a2;\n@e tcgen05.cp.cta_group::2.32x128b.warpx4 [c3], a3;\n"
            "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%2];\n}"
            ::"r"(columns), "l"(desc), "r"(ready)
            : "memory");
    } else {
        asm volatile(
            "{\n.reg .pred e;\n.reg .b64 a1, a2, a3, b0, b1, b2, b3;\n.reg .b32 c1, c2, c3, d0, d1, d2, d3;\n"
            "tcgen05.fence::after_thread_sync;\nelect.sync _|e, 0xffffffff;\n"
            "add.s64 a1, %1, 32;\nadd.s64 a2, %1, 64;\nadd.s64 a3, %1, 96;\nadd.s64 b0, %1, 128;\nadd.s64 b1, %1, 160;\nadd.s64 b2, %1, 192;\nadd.s64 b3, %1, 224;\n"
            "add.s32 c1, %0, 8;\nadd.s32 c2, %0, 16;\nadd.s32 c3, %0, 24;\nadd.s32 d0, %0, 4;\nadd.s32 d1, %0, 12;\nadd.s32 d2, %0, 20;\nadd.s32 d3, %0, 28;\n"
            "@e tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;\n@e tcgen05.cp.cta_group::2.32x128b.warpx4 [d0], b0;\n"
            "@e tcgen05.cp.cta_group::2.32x128b.warpx4 [c1], a1;\n@e tcgen05.cp.cta_group::2.32x128b.warpx4 [d1], b1;\n"
            "@e tcgen05.cp.cta_group::2.32x128b.warpx4 [c2], a2;\n@e tcgen05.cp.cta_group::2.32x128b.warpx4 [d2], b2;\n"
            "@e tcgen05.cp.cta_group::2.32x128b.warpx4 [c3], a3;\n@e tcgen05.cp.cta_group::2.32x128b.warpx4 [d3], b3;\n"
            "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%2];\n}"
            ::"r"(columns), "l"(desc), "r"(ready)
            : "memory");
    }
}
template <bool kTail>
struct PairTail {
    __device__ constexpr operator bool() const { return kTail; }
};
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar & kLeaderMask) : "memory");
}

// A tile of the pair kernel: 256 token rows on the MMA's row dimension and 256 features on its n (128 in a half tile at the end), or,
// for the token rows past the last whole 256, a tail tile: the operands change places, 256 features are the rows (128 on either
// CTA) and the tokens, in steps of 32, n. So 9 token rows cost the weights' way into shared memory and 32 columns, not 256 rows of
// padding; and in one launch with the others the tail shares their balance over the pairs.
struct PairTile {
    uint32_t n_tile, token0;   // 256-feature tile; first token row
    bool tail;
};
__device__ __forceinline__ PairTile pair_tile(uint32_t tile, uint32_t main_tiles, uint32_t m_pairs) {
    if (tile >= main_tiles) return PairTile{tile - main_tiles, m_pairs * 2 * kTileM, true};
    return PairTile{tile / m_pairs, tile % m_pairs * 2 * kTileM, false};
}

// 16 BF16 values of one token, one quantisation group, as the next GEMM's activations.
__device__ __forceinline__ void quantise_row(const GemmParams& p, uint32_t token, uint32_t group, const uint32_t (&packed)[8]) {
    const uint32_t width = p.rows / 2;
    const uint64_t code_bytes = tcgen05_codes_bytes(p.padded_tokens, width), scale_bytes = tcgen05_scale_bytes(p.padded_tokens, width);
    float2 residual[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) residual[i] = make_float2(__uint_as_float(packed[i] << 16), __uint_as_float(packed[i] & 0xffff0000u));
#pragma unroll 1
    for (uint32_t term = 0; term < p.quant_terms; ++term) {
        uint32_t codes[2], scale_code;
        quantise_term(residual, p.quant_scale, term + 1 < p.quant_terms, codes, &scale_code);
        *reinterpret_cast<uint2*>(p.quant_out + term * code_bytes + static_cast<uint64_t>(token) * (width / 2) + group * 8) = make_uint2(codes[0], codes[1]);
        p.quant_out[p.quant_terms * code_bytes + term * scale_bytes + tcgen05_scale_offset(token, group, width)] = static_cast<uint8_t>(scale_code);
    }
}

// The first look at a barrier is in line, the rest suspended: what does not poll leaves the board's power to the MMAs (17408 x 5120 x 4096 with its
// quantiser, one term 195.8 -> 194.4 us, MLP block of 4096 tokens 1328 -> 1322).
__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* status_word, uint32_t code) {
    return mbar_test(bar, parity) || warp_wait_suspended(bar, parity, abort_flag, status_word, code);
}
// Where the sums that a pair hands over pass through: a slot per epilogue warp of either CTA (`place` 0 .. 15).
__device__ __forceinline__ uint32_t pair_slot(uint32_t giver, uint32_t place) { return giver * 2 * kPairEpilogueWarps + place; }
__device__ __forceinline__ float4* pair_slot_sums(const GemmParams& p, uint32_t slot, uint32_t lane) {
    return reinterpret_cast<float4*>(p.split_slots) + static_cast<uint64_t>(slot) * (32 * 32) + lane;
}
// The part that finishes a leftover tile waits for the parts handed over, which are then added in pair order.
static __device__ __noinline__ bool pair_parts_arrived(const GemmParams& p, const PairItem& item, uint32_t pair, uint32_t place, volatile uint32_t* abort_flag) {
    bool arrived = true;
    for (uint32_t giver = item.first_giver; giver < pair; ++giver) {
        const uint32_t slot = pair_slot(giver, place);
        if ((threadIdx.x & 31) == 0) {
            uint32_t spin = 0;
            while (atomicAdd(p.split_flags + slot, 0u) == 0u) {
                if (++spin > kSplitWaitLimit || ((spin & 255u) == 255u && *abort_flag)) {
                    arrived = false;
                    *abort_flag = 1;
                    atomicCAS(p.status_word, 0u, kErrSplitWait);
                    break;
                }
            }
            // The flags read zero again when the launch is over, unless a part was given up on and came late: that launch has failed and says so, and
            // reading the plan's status clears what it left.
            p.split_flags[slot] = 0;
        }
    }
    __threadfence();
    return __all_sync(0xffffffffu, arrived) != 0;
}
// 32 weight rows (one per lane) of 32 tokens of a tail tile on their way out: turned through shared memory, so that a row of it
// is one token's.
__device__ __forceinline__ void pair_store_tail(const GemmParams& p, uint8_t* rows, uint32_t token0, uint32_t row0, uint32_t lane, const uint32_t (&sums)[32]) {
    if (!p.swiglu) {
#pragma unroll
        for (uint32_t i = 0; i < 32; ++i) {
            *reinterpret_cast<__nv_bfloat16*>(rows + i * kPairOutRowBytes + lane * 2) = __float2bfloat16_rn(__uint_as_float(sums[i]) * p.scale);
        }
    } else {
        // Lanes 0..15 hold gate rows and lanes 16..31 the matching up rows: the former finish the even tokens, the latter the odd ones.
        const bool upper = lane >= 16;
#pragma unroll
        for (uint32_t i = 0; i < 32; i += 2) {
            const float other = __uint_as_float(__shfl_xor_sync(0xffffffffu, upper ? sums[i] : sums[i + 1], 16));
            const float gate = (upper ? other : __uint_as_float(sums[i])) * p.scale, up = (upper ? __uint_as_float(sums[i + 1]) : other) * p.scale_b;
            *reinterpret_cast<__nv_bfloat16*>(rows + (i + (lane >> 4)) * kPairOutRowBytes + (lane & 15) * 2) =
                __float2bfloat16_rn(__fdividef(gate, 1.0f + __expf(-gate)) * up);   // as in convert_chunk
        }
    }
    __syncwarp();
    if (p.quant_out && token0 + lane < p.tokens) {
        const uint4 low = *reinterpret_cast<const uint4*>(rows + lane * kPairOutRowBytes), high = *reinterpret_cast<const uint4*>(rows + lane * kPairOutRowBytes + 16);
        const uint32_t packed[8] = {low.x, low.y, low.z, low.w, high.x, high.y, high.z, high.w};
        quantise_row(p, token0 + lane, row0 / 32, packed);
    }
    if (p.out) {
        const uint32_t lanes = p.swiglu ? 2 : 4, width = p.swiglu ? p.rows / 2 : p.rows;   // 16 bytes a lane
        uint8_t* out_base = reinterpret_cast<uint8_t*>(p.out + static_cast<uint64_t>(token0) * width + (p.swiglu ? row0 / 2 : row0));
        for (uint32_t r = lane / lanes; r < 32 && token0 + r < p.tokens; r += 32 / lanes) {
            const uint32_t piece = lane % lanes;
            *reinterpret_cast<uint4*>(out_base + static_cast<uint64_t>(r) * width * 2 + piece * 16) =
                *reinterpret_cast<const uint4*>(rows + r * kPairOutRowBytes + piece * 16);
        }
    }
    __syncwarp();   // the rows are rewritten for the next chunk
}
// The epilogue of a tail tile, a function of its own so that it costs the main tiles' no registers: lanes are weight rows and columns tokens, at
// most 64 of them per warp. Releases the accumulator; false if a part that was to be handed over did not come.
static __device__ __noinline__ bool pair_tail_epilogue(const GemmParams& p, const PairItem& item, uint32_t accumulator, uint8_t* rows, uint32_t first_token,
                                                       uint32_t row0, uint32_t pair, uint32_t place, uint32_t tmem_empty, volatile uint32_t* abort_flag) {
    const uint32_t lane = threadIdx.x & 31;
    const bool second = first_token + 32 < p.tokens;
    uint32_t v[2][32];
    tc_load32(accumulator, v[0]);
    tc_load32(accumulator + 32, v[1]);   // past the tile's columns: never used
    tc_wait_ld();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive_leader(tmem_empty);
    if (item.kind == 1) {
        float4* own = pair_slot_sums(p, pair_slot(pair, place), lane);
#pragma unroll
        for (uint32_t c = 0; c < 2; ++c) {
            if (c && !second) break;
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                own[(c * 8 + i) * 32] = make_float4(__uint_as_float(v[c][4 * i]), __uint_as_float(v[c][4 * i + 1]),
                                                    __uint_as_float(v[c][4 * i + 2]), __uint_as_float(v[c][4 * i + 3]));
            }
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicExch(p.split_flags + pair_slot(pair, place), 1u);
        return true;
    }
    if (item.kind == 2) {
        if (!pair_parts_arrived(p, item, pair, place, abort_flag)) return false;
        for (uint32_t giver = item.first_giver; giver < pair; ++giver) {
            const float4* src = pair_slot_sums(p, pair_slot(giver, place), lane);
#pragma unroll
            for (uint32_t c = 0; c < 2; ++c) {
                if (c && !second) break;
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    const float4 part = __ldcg(src + (c * 8 + i) * 32);
                    v[c][4 * i] = __float_as_uint(__uint_as_float(v[c][4 * i]) + part.x);
                    v[c][4 * i + 1] = __float_as_uint(__uint_as_float(v[c][4 * i + 1]) + part.y);
                    v[c][4 * i + 2] = __float_as_uint(__uint_as_float(v[c][4 * i + 2]) + part.z);
                    v[c][4 * i + 3] = __float_as_uint(__uint_as_float(v[c][4 * i + 3]) + part.w);
                }
            }
        }
    }
    pair_store_tail(p, rows, first_token, row0, lane, v[0]);
    if (second) pair_store_tail(p, rows, first_token + 32, row0, lane, v[1]);
    return true;
}

// One instantiation per number of activation terms (the ring depths as constants are worth 1.5 %), with and without the fused quantiser, whose
// registers the other epilogues need not pay for.
template <uint32_t kTerms, bool kQuantised>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_act, const __grid_constant__ CUtensorMap map_weight,
                 const __grid_constant__ CUtensorMap map_act_sf, const __grid_constant__ CUtensorMap map_weight_sf,
                 const __grid_constant__ CUtensorMap map_tail, const __grid_constant__ GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* out_stage = smem + kPairRingBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_stage + kPairOutBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kPairBarriers);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();            // 0 = leader
    const uint32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    constexpr PairDepths depth = pair_depths(kTerms);
    const uint32_t smem_base = smem_u32(smem), tokens_base = smem_base + depth.weights * kPairWeightStage;
    const uint32_t bar0 = smem_u32(bars);
    const uint32_t w_full = bar0, w_landed = bar0 + 8 * kPairMaxDepth;
    const uint32_t t_full = bar0 + 16 * kPairMaxDepth, t_landed = bar0 + 24 * kPairMaxDepth, t_empty = bar0 + 32 * kPairMaxDepth;
    const uint32_t bar_tmem_full = bar0 + 40 * kPairMaxDepth, bar_tmem_empty = bar_tmem_full + 8;

    // An odd number of 128-row token tiles leaves the second CTA of the last pair without rows of its own: it
    // loads whatever follows (the next term's rows, or the fill value past the tensor) and stores nothing.
    const uint32_t m_pairs = p.token_pairs;
    // With an odd number of 128-row blocks of weights the last tile is half as wide (MMA n = 128): each CTA brings 64 of
    // its rows, and the epilogue warps of the second column half have nothing to do.
    const uint32_t n_tiles = (p.rows + kTileN - 1) / kTileN;
    const uint32_t half_tile = p.rows % kTileN ? n_tiles - 1 : n_tiles;
    const uint32_t main_tiles = m_pairs * n_tiles;
    // A last k block that is only partly inside the tensor is loaded like the others (the TMA fills what lies past
    // the edge); the MMA issuer only consumes the k steps inside.
    const uint32_t k_blocks = (p.cols + kBlockK - 1) / kBlockK;
    // What this pair does is kept in shared memory: fourteen registers less in every role (the epilogue holds 128 sums a thread).
    PairWork& work = *reinterpret_cast<PairWork*>(tmem_slot + 2 + kPairThreads / 32);
    if (threadIdx.x == 32 * 2) {
        work = pair_work(pair, pairs, PairShares{main_tiles, p.tail_columns ? n_tiles : 0, k_blocks, p.split_sharers, p.cost_main, p.cost_tail});
    }
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kPairMaxDepth; ++s) {
            mbar_init(w_full + 8 * s, 2);
            mbar_init(w_landed + 8 * s, 1);
            mbar_init(t_full + 8 * s, 2);
            mbar_init(t_empty + 8 * s, 1);
            mbar_init(t_landed + 8 * s, 1);
        }
        mbar_init(bar_tmem_full, 1);
        mbar_init(bar_tmem_empty, 2 * kPairEpilogueWarps);   // one arrival per epilogue warp of either CTA
        *abort_flag = 0;
        for (uint32_t w = 0; w < kPairThreads / 32; ++w) abort_flag[1 + w] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // the peer's barriers exist before anything can signal them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_weights = tmem_base + kTmemPairScales, tmem_tokens = tmem_weights + depth.weights * 32;

    // The weights are constant, so the first ring of them, `ahead` k blocks of the first item, is under way while the launch before
    // this one, whose results the token rows are, still drains. What a role waits for on a barrier must not include that launch,
    // whose time would count against the bound of the wait: a role that depends on it waits for its end first.
    uint32_t ahead = 0;
    if (work.items) {
        const PairItem first = work.item(0, pair, pairs, k_blocks);
        ahead = min(depth.weights, first.kb1 - first.kb0);
    }

    if (warp == 0) {
        // ---------------- TMA producer (both CTAs) ----------------
        // The block scales of a slot go first, on a barrier of their own: they are small and land early, so the copy warps have
        // them in tensor memory by the time the operand tiles arrive.
        uint32_t w_stage = 0, slot = 0, t_phase = 1;
        bool alive = true;
        // As n operand the scales of all 256 features go to both CTAs, as row operand those of a CTA's own 128 (and the block behind, unused).
        auto load_weights = [&](const PairTile& t, uint32_t kb, uint32_t stage) {
            const uint32_t codes = smem_base + stage * kPairWeightStage;
            tma_weight_step(rank == 0, w_landed + 8 * stage, codes + kPairBytesB, &map_weight_sf, kb * 4, t.n_tile * 2 + (t.tail ? rank : 0),
                            w_full + 8 * stage, codes, &map_weight, kb * 128, t.n_tile * kTileN + rank * (!t.tail && t.n_tile == half_tile ? 64 : 128));
        };
        if (work.items) {
            const PairItem first = work.item(0, pair, pairs, k_blocks);
            const PairTile tile = pair_tile(first.tile, main_tiles, m_pairs);
            for (uint32_t stage = 0; stage < ahead; ++stage) {
                load_weights(tile, first.kb0 + stage, stage);
            }
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (lane == 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        uint32_t blocks = 0;
        for (uint32_t index = 0; alive && index < work.items; ++index) {
            const PairItem item = work.item(index, pair, pairs, k_blocks);
            const PairTile tile = pair_tile(item.tile, main_tiles, m_pairs);
            // a tail tile's tokens are the n operand: half of them on either CTA, the scales of their one 128-row block on both
            const CUtensorMap* map_tokens = tile.tail ? &map_tail : &map_act;
            const uint32_t pair_bytes = tile.tail ? p.tail_columns * 128 : 2 * kBytesA;
            const uint32_t token_row = tile.token0 + rank * (tile.tail ? p.tail_columns / 2 : kTileM);
            const uint32_t scale_block = (tile.tail ? tile.token0 : token_row) / 128;
            for (uint32_t kb = item.kb0; alive && kb < item.kb1; ++kb, ++blocks) {
#pragma unroll
                for (uint32_t term = 0; term < kTerms; ++term) {
                    if (!pair_wait(t_empty + 8 * slot, t_phase, abort_flag, p.status_word, kErrProducerWait)) {
                        alive = false;
                        break;
                    }
                    if (term == pair_weight_term(kTerms) && blocks >= ahead) load_weights(tile, kb, w_stage);
                    const uint32_t base = tokens_base + slot * kPairTokenSlot;
                    tma_token_step(rank == 0, t_landed + 8 * slot, base + kBytesA, &map_act_sf, kb * 4, term * (p.padded_tokens / 128) + scale_block,
                                   t_full + 8 * slot, pair_bytes, base, map_tokens, kb * 128, term * p.padded_tokens + token_row);
                    if (++slot == depth.tokens) { slot = 0; t_phase ^= 1; }
                }
                if (++w_stage == depth.weights) w_stage = 0;
            }
        }
    } else if (warp == 1 && rank == 0) {
        // ---------------- MMA issuer (leader only) ----------------
        // Issuing a tcgen05 operation keeps a warp busy for tens of cycles, and one warp issuing the 12 scale copies and
        // the 4 MMAs of every step could not keep the tensor pipe fed; the copies are issued by two warps of their own
        // (below) into the slots' scale columns, this one issues only the MMAs, a step's as one block of predicated instructions. Descriptors advance by
        // additions (their low bits hold address >> 4).
        uint32_t w_stage = 0, w_phase = 0, slot = 0, t_phase = 0, tmem_phase = 0, behind = 0, behind_phase = 0, ahead_steps = 0;
        bool alive = true;
        constexpr uint32_t kWideTile = (1u << 7) | (1u << 10) | ((kTileN >> 3) << 17) | (((2 * kTileM) >> 4) << 24);
        constexpr uint32_t kHalfTile = (1u << 7) | (1u << 10) | ((kTileN / 2 >> 3) << 17) | (((2 * kTileM) >> 4) << 24);
        const uint32_t w_desc0 = static_cast<uint32_t>(operand_desc(smem_base)), t_desc0 = static_cast<uint32_t>(operand_desc(tokens_base));
        const uint32_t last_k_steps = (p.cols - (k_blocks - 1) * kBlockK) / 64;   // 1..4 k steps of 64 in the last k block
        asm volatile("griddepcontrol.wait;" ::: "memory");   // the token rows
        for (uint32_t index = 0; alive && index < work.items; ++index) {
            const PairItem item = work.item(index, pair, pairs, k_blocks);
            // The epilogues of both CTAs must have drained the previous tile's accumulator: the one wait that polls, since the tensor pipe
            // stands still meanwhile.
            if (!warp_look_wait(bar_tmem_empty, tmem_phase ^ 1, abort_flag, p.status_word, kErrMmaWaitTmem)) break;
            const PairTile tile = pair_tile(item.tile, main_tiles, m_pairs);
            uint32_t accumulate = 0;
            // `Tail`: the weights are the row operand
            auto multiply = [&](auto tail, uint32_t idesc) {
                for (uint32_t kb = item.kb0; kb < item.kb1; ++kb) {
                    if (!pair_wait(w_full + 8 * w_stage, w_phase, abort_flag, p.status_word, kErrMmaWaitWeights)) return false;
                    const uint32_t w_desc = w_desc0 + w_stage * (kPairWeightStage >> 4), sf_w = tmem_weights + w_stage * 32;
                    const uint32_t k_steps = kb + 1 < k_blocks ? 4u : last_k_steps;
                    if (++w_stage == depth.weights) { w_stage = 0; w_phase ^= 1; }
#pragma unroll
                    for (uint32_t term = 0; term < kTerms; ++term) {
                        // codes in shared memory (TMA) and block scales on their way to tensor memory (copy warp)
                        if (!pair_wait(t_full + 8 * slot, t_phase, abort_flag, p.status_word, kErrMmaWaitTokens)) return false;
                        // No more than two steps of a whole tile are issued ahead of the pipe: the scale copies of later slots queue behind the MMAs and are
                        // announced when they are done, too late for the next steps otherwise (18944 x 5120, 512 tokens, three terms 53.3 -> 51.6 us). At
                        // one term, and in tail tiles, whose steps are short, nothing is gained.
                        if (kTerms > 1 && ahead_steps == 2) {
                            if (!tail && !pair_wait(t_empty + 8 * behind, behind_phase, abort_flag, p.status_word, kErrMmaWaitTokens)) return false;
                            if (++behind == depth.tokens) { behind = 0; behind_phase ^= 1; }
                        } else {
                            ++ahead_steps;
                        }
                        const uint32_t t_desc = t_desc0 + slot * (kPairTokenSlot >> 4), sf_t = tmem_tokens + slot * 16, t_done = t_empty + 8 * slot;
                        // Each MMA consumes 64 k = 32 bytes of every row: start address + 2; only k steps inside the tensor. The commit frees
                        // the slot, and with it the slot's scale columns, in both CTAs.
                        if (tail) tc_step_pair(tmem_base + kTmemAcc, w_desc, t_desc, idesc, sf_w, sf_t, 8, 4, accumulate, k_steps, t_done);
                        else tc_step_pair(tmem_base + kTmemAcc, t_desc, w_desc, idesc, sf_t, sf_w, 4, 8, accumulate, k_steps, t_done);
                        if (++slot == depth.tokens) { slot = 0; t_phase ^= 1; }
                        accumulate = 1;
                    }
                }
                return true;
            };
            alive = tile.tail ? multiply(PairTail<true>(), kHalfTile - (((kTileN / 2 - p.tail_columns) >> 3) << 17))
                              : multiply(PairTail<false>(), tile.n_tile == half_tile ? kHalfTile : kWideTile);
            if (alive && elect_one()) tc_commit_pair(bar_tmem_full);     // both accumulator halves complete
            __syncwarp();
            tmem_phase ^= 1;
        }
    } else if ((warp == kPairCopyWarp || warp == kPairCopyWarp + 1) && rank == 0) {
        // ---------------- scale-copy issuers (leader only): shared memory -> tensor memory, both CTAs ----------------
        // One warp copies the token rows' scales of every step, the other the weight rows' scales, which are the same for all
        // activation terms of a k block. (One thread issuing all twelve copies of a one-term step needed longer
        // than the step's MMAs: 193 us for 4096 tokens on 17408 x 5120.)
        // A slot's scale atoms have landed. The producer refilled the slot only after the MMAs that used it last were
        // complete, so the slot's scale columns are free. The MMA warp waits for a commit behind the copies: with a plain arrival, on the strength of copies and
        // later MMAs executing in the order of their issue, most launches of 17408 x 5120, 1024 tokens, three terms multiplied some k block's last 64 k
        // before the scales of its second 128 features were there, once a step of the MMA warp was as short as it is.
        // Slots are taken as they come, whatever tile they belong to, and whole: what a last k block or a tile does not have is not read.
        const uint32_t blocks = work.blocks(k_blocks);
        if (warp == kPairCopyWarp) {
            asm volatile("griddepcontrol.wait;" ::: "memory");   // the token rows
            const uint64_t desc0 = sf_desc(tokens_base + kBytesA);
            uint32_t slot = 0, phase = 0;
            for (uint32_t left = blocks * kTerms; left; --left) {
                if (!pair_wait(t_landed + 8 * slot, phase, abort_flag, p.status_word, kErrCopyWait)) break;
                tc_copy_step_pair<1>(tmem_tokens + slot * 16, desc0 + slot * (kPairTokenSlot >> 4), t_full + 8 * slot);
                if (++slot == depth.tokens) { slot = 0; phase ^= 1; }
            }
        } else {
            const uint64_t desc0 = sf_desc(smem_base + kPairBytesB);
            uint32_t stage = 0, phase = 0;
            for (uint32_t block = 0; block < blocks; ++block) {
                // stages beyond the first ring are free when the token rows have been multiplied with
                if (block == ahead) asm volatile("griddepcontrol.wait;" ::: "memory");
                if (!pair_wait(w_landed + 8 * stage, phase, abort_flag, p.status_word, kErrCopyWait)) break;
                tc_copy_step_pair<2>(tmem_weights + stage * 32, desc0 + stage * (kPairWeightStage >> 4), w_full + 8 * stage);
                if (++stage == depth.weights) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp >= 2 && warp < 2 + kPairEpilogueWarps) {
        // ---------------- epilogue (both CTAs): own TMEM half -> BF16 -> global ----------------
        // The wait for the tile is a suspended one: eight polling warps cost 2 to 3 % of the time at the board's power cap.
        // Two warps per lane quadrant, 128 accumulator columns each. A warp reads its columns into registers
        // in one go and releases the accumulator at once; conversion, staging and the stores to global memory
        // run while the next tile's MMAs are already under way.
        const uint32_t quadrant = warp & 3, half = (warp - 2) >> 2;
        uint32_t tmem_phase = 0;
        asm volatile("griddepcontrol.wait;" ::: "memory");   // nothing is written while an earlier kernel may still read it
        // this warp's transposition rows (lane = row): one 32-column chunk at a time
        uint8_t* my_rows = out_stage + (warp - 2) * 32 * kPairOutRowBytes;
        for (uint32_t index = 0; index < work.items; ++index) {
            const PairItem item = work.item(index, pair, pairs, k_blocks);
            const PairTile tile = pair_tile(item.tile, main_tiles, m_pairs);
            const uint32_t n_tile = tile.n_tile;
            if (!warp_wait_suspended(bar_tmem_full, tmem_phase, abort_flag, p.status_word, kErrEpilogueWait)) break;
            tc_fence_after();
            const uint32_t accumulator = tmem_base + kTmemAcc + ((quadrant * 32) << 16) + half * (tile.tail ? 64 : 128);
            auto release = [&]() {   // the accumulator is free for the next tile's MMAs from here on
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_leader(bar_tmem_empty);
                tmem_phase ^= 1;
            };
            // Rows past the tokens, and the columns a half tile does not have: nothing to store, hand over or add. (Padding rows
            // hold whatever the staging buffer held; converting them cost more than real ones, since zeros and non-finite
            // values leave the quantiser's fast path.)
            const uint32_t first_token = tile.token0 + (tile.tail ? half * 64 : rank * kTileM + quadrant * 32);
            const uint32_t tail_row = n_tile * kTileN + rank * kTileM + quadrant * 32;   // of a tail tile: this warp's weight rows
            if (first_token >= p.tokens || (tile.tail ? tail_row >= p.rows : half && n_tile == half_tile)) {
                release();
                continue;
            }

            const uint32_t out_width = kQuantised || p.swiglu ? p.rows / 2 : p.rows, token = first_token + lane;
            uint32_t scale_words[3] = {0, 0, 0};   // SwiGLU, quantised: the scale bytes of this row's 4 groups, per term: one word of an atom
            uint32_t held[8];
            // The BF16 values this lane holds, quantised for the next GEMM while the next tile's MMAs run: groups c (`held`) and c + 1. Eight warps
            // do not hide the latencies of one group's chain of three terms: two side by side, and stores of 16 bytes.
            auto quantise_two = [&](uint32_t c, const uint32_t (&second)[16]) {
                if (token >= p.tokens) return;
                const uint64_t code_bytes = tcgen05_codes_bytes(p.padded_tokens, out_width);
                const uint32_t group = n_tile * (kTileN / 32) + half * 4 + c;
                float2 residual[2][8];
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    residual[0][i] = make_float2(__uint_as_float(held[i] << 16), __uint_as_float(held[i] & 0xffff0000u));
                    residual[1][i] = make_float2(__uint_as_float(second[i] << 16), __uint_as_float(second[i] & 0xffff0000u));
                }
#pragma unroll
                for (uint32_t term = 0; term < 3; ++term) {
                    if (term >= p.quant_terms) break;
                    uint32_t codes[2][2], scale_code[2];
                    if (term + 1 < p.quant_terms) quantise_groups_as<true>(residual, p.quant_scale, codes, scale_code);
                    else quantise_groups_as<false>(residual, p.quant_scale, codes, scale_code);
                    scale_words[term] |= scale_code[0] << (8 * c) | scale_code[1] << (8 * c + 8);
                    *reinterpret_cast<uint4*>(p.quant_out + term * code_bytes + static_cast<uint64_t>(token) * (out_width / 2) + group * 8) =
                        make_uint4(codes[0][0], codes[0][1], codes[1][0], codes[1][1]);
                }
                if (c == 2) {
                    const uint64_t scale_bytes = tcgen05_scale_bytes(p.padded_tokens, out_width);
#pragma unroll
                    for (uint32_t term = 0; term < 3; ++term) {
                        if (term >= p.quant_terms) break;
                        *reinterpret_cast<uint32_t*>(p.quant_out + p.quant_terms * code_bytes + term * scale_bytes +
                                                     tcgen05_scale_offset(token, n_tile * (kTileN / 32) + half * 4, out_width)) = scale_words[term];
                    }
                }
            };
            // One 32-column chunk of sums on its way out.
            auto store_chunk = [&](uint32_t c, const uint32_t (&sums)[32]) {
                uint32_t packed[16];
                if (kQuantised || p.swiglu) {
                    // 32 accumulator columns = gate and up sums of 16 intermediate columns = one quantisation group per row
                    convert_chunk(sums, p.scale, p.scale_b, true, packed);
                    if (kQuantised) {
                        if (c & 1) quantise_two(c - 1, packed);
#pragma unroll
                        for (uint32_t i = 0; i < 8; ++i) held[i] = packed[i];
                    }
                    if (p.out) {
                        // transpose through shared memory: 32 bytes of every row, written out as 2 lanes per row
                        uint4* dst = reinterpret_cast<uint4*>(my_rows + lane * kPairOutRowBytes);
                        dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                        dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
                        __syncwarp();
                        uint8_t* out_base = reinterpret_cast<uint8_t*>(p.out + static_cast<uint64_t>(first_token) * out_width +
                                                                       n_tile * (kTileN / 2) + half * 64 + c * 16);
#pragma unroll
                        for (uint32_t r16 = 0; r16 < 32; r16 += 16) {
                            const uint32_t r = r16 + (lane >> 1), piece = lane & 1;
                            if (first_token + r >= p.tokens) continue;   // padding rows of the last tile are computed, never stored
                            const uint4 value = *reinterpret_cast<const uint4*>(my_rows + r * kPairOutRowBytes + piece * 16);
                            *reinterpret_cast<uint4*>(out_base + static_cast<uint64_t>(r) * out_width * 2 + piece * 16) = value;
                        }
                        __syncwarp();   // the rows are rewritten for the next chunk
                    }
                    return;
                }
                convert_chunk(sums, p.scale, p.scale_b, false, packed);
                // transpose through shared memory: 64 bytes of every row, written out as 4 lanes per row
                uint4* dst = reinterpret_cast<uint4*>(my_rows + lane * kPairOutRowBytes);
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    dst[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
                }
                __syncwarp();
                uint8_t* out_base = reinterpret_cast<uint8_t*>(p.out + static_cast<uint64_t>(first_token) * p.rows + n_tile * kTileN +
                                                               half * 128 + c * 32);
#pragma unroll
                for (uint32_t r8 = 0; r8 < 32; r8 += 8) {
                    const uint32_t r = r8 + (lane >> 2), piece = lane & 3;
                    if (first_token + r >= p.tokens) continue;   // padding rows of the last tile are computed, never stored
                    const uint4 value = *reinterpret_cast<const uint4*>(my_rows + r * kPairOutRowBytes + piece * 16);
                    *reinterpret_cast<uint4*>(out_base + static_cast<uint64_t>(r) * p.rows * 2 + piece * 16) = value;
                }
                __syncwarp();   // the rows are rewritten for the next chunk
            };
            auto slot_of = [&](uint32_t giver) { return pair_slot(giver, rank * kPairEpilogueWarps + warp - 2); };
            auto slot_sums = [&](uint32_t slot) { return pair_slot_sums(p, slot, lane); };
            auto parts_arrived = [&]() { return pair_parts_arrived(p, item, pair, rank * kPairEpilogueWarps + warp - 2, abort_flag); };
            if (tile.tail) {
                if (!pair_tail_epilogue(p, item, accumulator, my_rows, first_token, tail_row, pair, rank * kPairEpilogueWarps + warp - 2, bar_tmem_empty, abort_flag)) break;
                tmem_phase ^= 1;
                continue;
            }
            if (item.kind == 2 && index + 1 == work.items) {
                if (!parts_arrived()) break;
                // Nothing follows that waits for the accumulator: a chunk at a time stays in registers, and the same chunk of several
                // parts is in flight at once (one part after the other, all 128 columns each, cost 3 us per part).
#pragma unroll 1
                for (uint32_t c = 0; c < 4; ++c) {
                    uint32_t sums[32];
                    tc_load32(accumulator + c * 32, sums);
                    tc_wait_ld();
                    for (uint32_t giver = item.first_giver; giver < pair; giver += 3) {
                        float4 part[3][8];
#pragma unroll
                        for (uint32_t q = 0; q < 3; ++q) {
                            const float4* src = slot_sums(slot_of(giver + q));
#pragma unroll
                            for (uint32_t i = 0; i < 8; ++i) {
                                part[q][i] = giver + q < pair ? __ldcg(src + (c * 8 + i) * 32) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            }
                        }
#pragma unroll
                        for (uint32_t q = 0; q < 3; ++q) {
                            if (giver + q >= pair) break;
#pragma unroll
                            for (uint32_t i = 0; i < 8; ++i) {
                                sums[4 * i] = __float_as_uint(__uint_as_float(sums[4 * i]) + part[q][i].x);
                                sums[4 * i + 1] = __float_as_uint(__uint_as_float(sums[4 * i + 1]) + part[q][i].y);
                                sums[4 * i + 2] = __float_as_uint(__uint_as_float(sums[4 * i + 2]) + part[q][i].z);
                                sums[4 * i + 3] = __float_as_uint(__uint_as_float(sums[4 * i + 3]) + part[q][i].w);
                            }
                        }
                    }
                    store_chunk(c, sums);
                }
                release();
                continue;
            }

            uint32_t v[4][32];
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) tc_load32(accumulator + c * 32, v[c]);
            tc_wait_ld();
            release();
            if (item.kind == 1) {
                // a part of a leftover tile: the sums go, as they are, to the pair that finishes the tile
                const uint32_t slot = slot_of(pair);
                float4* dst = slot_sums(slot);
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c) {
#pragma unroll
                    for (uint32_t i = 0; i < 8; ++i) {
                        dst[(c * 8 + i) * 32] = make_float4(__uint_as_float(v[c][4 * i]), __uint_as_float(v[c][4 * i + 1]),
                                                            __uint_as_float(v[c][4 * i + 2]), __uint_as_float(v[c][4 * i + 3]));
                    }
                }
                __threadfence();
                __syncwarp();
                if (lane == 0) atomicExch(p.split_flags + slot, 1u);
                continue;
            }
            if (item.kind == 2) {
                if (!parts_arrived()) break;
                for (uint32_t giver = item.first_giver; giver < pair; ++giver) {
                    const float4* src = slot_sums(slot_of(giver));
#pragma unroll
                    for (uint32_t c = 0; c < 4; ++c) {
#pragma unroll
                        for (uint32_t i = 0; i < 8; ++i) {
                            const float4 part = __ldcg(src + (c * 8 + i) * 32);
                            v[c][4 * i] = __float_as_uint(__uint_as_float(v[c][4 * i]) + part.x);
                            v[c][4 * i + 1] = __float_as_uint(__uint_as_float(v[c][4 * i + 1]) + part.y);
                            v[c][4 * i + 2] = __float_as_uint(__uint_as_float(v[c][4 * i + 2]) + part.z);
                            v[c][4 * i + 3] = __float_as_uint(__uint_as_float(v[c][4 * i + 3]) + part.w);
                        }
                    }
                }
            }
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) store_chunk(c, v[c]);
        }
    }

    // Neither CTA may release tensor memory while the other can still be written by an MMA or read
    // by an epilogue: every thread of the pair meets here (all waits above are bounded).
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

using PairKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, GemmParams);
constexpr PairKernel kPairKernels[6] = {gemm_pair_kernel<1, false>, gemm_pair_kernel<2, false>, gemm_pair_kernel<3, false>,
                                        gemm_pair_kernel<1, true>, gemm_pair_kernel<2, true>, gemm_pair_kernel<3, true>};

// ---- activation quantiser kernel ---------------------------------------------------------------
// One thread per (token, 16-element group). Destination: the code planes of all terms
// stacked ([terms][tokens][cols/2], one TMA tensor of terms*tokens rows), then the scale
// regions of all terms.
constexpr uint32_t kQuantThreads = 128;
// `x` is read by coherent loads: the launch before this one may still be writing it when this grid starts, so it is not
// constant for the life of the grid, which is what __ldg (and a compiler's choice of it) would promise.
__global__ void __launch_bounds__(kQuantThreads) act_quant_kernel(const uint16_t* x, uint8_t* destination, uint32_t tokens, uint32_t cols,
                                                                  uint32_t terms, const QuantScale scale) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");   // x may come from the launch before this one, and the destination may still be read by it
    const uint32_t groups = cols / 16;
    // tokens * cols fits 32 bits, so the group index does too
    const uint32_t index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= tokens * groups) return;
    const uint32_t token = index / groups, group = index - token * groups;
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<uint64_t>(token) * cols + group * 16);
    const uint4 lo = __ldcg(src), hi = __ldcg(src + 1);
    const uint32_t words[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    float2 residual[8];   // pairs of neighbouring elements, as the two-wide F32 instructions take them
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        residual[i] = make_float2(__uint_as_float(words[i] << 16), __uint_as_float(words[i] & 0xffff0000u));
    }
    // every term's code plane has whole 128-row tiles (the rows past `tokens` are never written and
    // only ever feed output rows that are not stored)
    const uint64_t code_bytes = tcgen05_codes_bytes(padded_tokens(tokens), cols), scale_bytes = tcgen05_scale_bytes(tokens, cols);
    for (uint32_t term = 0; term < terms; ++term) {
        uint32_t packed[2], scale_code;
        quantise_term(residual, scale, term + 1 < terms, packed, &scale_code);
        *reinterpret_cast<uint2*>(destination + term * code_bytes + static_cast<uint64_t>(token) * (cols / 2) + group * 8) =
            make_uint2(packed[0], packed[1]);
        // The scales of four consecutive groups of a token are four consecutive bytes of an atom: lanes are
        // consecutive groups (cols / 16 is a multiple of 4, so a quad of lanes never straddles a token or the
        // end of the grid), and the first lane of every quad stores the four as one word.
        const uint32_t active = __activemask();
        uint32_t quad = scale_code;
        quad |= __shfl_down_sync(active, scale_code, 1) << 8;
        quad |= __shfl_down_sync(active, scale_code, 2) << 16;
        quad |= __shfl_down_sync(active, scale_code, 3) << 24;
        if ((group & 3u) == 0) {
            *reinterpret_cast<uint32_t*>(destination + terms * code_bytes + term * scale_bytes + tcgen05_scale_offset(token, group, cols)) = quad;
        }
    }
}

// ---- tensor maps --------------------------------------------------------------------------------
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_entry() {
    static EncodeTiled cached = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult query = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &query) != cudaSuccess ||
            query != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            fn = nullptr;
        }
        return reinterpret_cast<EncodeTiled>(fn);
    }();
    return cached;
}

}  // namespace

bool make_code_map(CUtensorMap* map, uint64_t address, uint64_t rows, uint32_t cols, uint32_t box_rows) {
    const EncodeTiled encode = encode_entry();
    if (!encode) return false;
    const cuuint64_t dims[2] = {cols / 2, rows};
    const cuuint64_t strides[1] = {cols / 2};
    const cuuint32_t box[2] = {128, box_rows};
    const cuuint32_t element_strides[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, reinterpret_cast<void*>(address), dims, strides, box,
                  element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

namespace {
// Block-scale atoms as a tensor [128-row blocks][atoms of a block along k][256 x u16] (512 bytes an atom); a box is the 4 atoms of
// `box_blocks` row blocks and one 256-deep k block.
bool make_scale_map(CUtensorMap* map, uint64_t address, uint64_t row_blocks, uint64_t atoms, uint32_t box_blocks) {
    const EncodeTiled encode = encode_entry();
    if (!encode) return false;
    const cuuint64_t dims[3] = {256, atoms, row_blocks};
    const cuuint64_t strides[2] = {kSfAtomBytes, atoms * kSfAtomBytes};
    const cuuint32_t box[3] = {256, 4, box_blocks};
    const cuuint32_t element_strides[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, reinterpret_cast<void*>(address), dims, strides, box,
                  element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---- validation ------------------------------------------------------------------------------------
bool act_shape_ok(uint32_t tokens, uint32_t cols, uint32_t terms) {
    return tokens && cols && tokens <= (1u << 24) && cols % 64 == 0 && terms >= 1 && terms <= 3 &&
           static_cast<uint64_t>(padded_tokens(tokens)) * cols <= UINT32_MAX;
}

bool check_act_quant(int32_t d, augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_act_quant_args_v1* a, bool full,
                     augur_cuda_result_v1* failure) {
    *failure = invalid();
    if (!header_ok(d, s, a)) {
        if (a && s && d >= 0 && s->ordinal == d && a->abi_version != AUGUR_CUDA_ABI_VERSION_V1) {
            *failure = make_result(AUGUR_CUDA_STATUS_ABI_VERSION_MISMATCH);
        }
        return false;
    }
    if (!act_shape_ok(a->tokens, a->cols, a->terms) || !std::isfinite(a->global_scale) || a->global_scale <= 0.0f) {
        return false;
    }
    if (a->input_len_bytes != static_cast<uint64_t>(a->tokens) * a->cols * 2 ||
        a->destination_len_bytes != a->terms * staged_term_bytes(a->tokens, a->cols)) {
        return false;
    }
    const Range r[2] = {{a->input_bf16, a->input_len_bytes, 16}, {a->destination, a->destination_len_bytes, 256}};
    if (!all_disjoint(r, 2)) return false;
    return !full || inspect_device_ranges(d, r, 2, failure);
}

// What `output_bf16` of a GEMM descriptor is: [tokens][rows], [tokens][rows / 2] (fused SwiGLU), or absent.
enum class GemmOutput { kFull, kHalfWidth, kNone };

bool check_gemm(int32_t d, augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_plan_v1* plan,
                const augur_cuda_nvfp4_sm100_gemm_args_v1* a, bool full, augur_cuda_result_v1* failure,
                GemmOutput output = GemmOutput::kFull) {
    *failure = invalid();
    if (!header_ok(d, s, a)) {
        if (a && s && d >= 0 && s->ordinal == d && a->abi_version != AUGUR_CUDA_ABI_VERSION_V1) {
            *failure = make_result(AUGUR_CUDA_STATUS_ABI_VERSION_MISMATCH);
        }
        return false;
    }
    if (!plan_ok(plan, d, s) || !act_shape_ok(a->tokens, a->cols, a->activation_terms)) return false;
    if (!a->rows || a->rows % 128 != 0 || static_cast<uint64_t>(a->rows) * a->cols > UINT32_MAX) return false;
    if (!scale_ok(a->weight_global_scale) || !std::isfinite(a->activation_global_scale) ||
        a->activation_global_scale <= 0.0f) {
        return false;
    }
    if (a->weight_len_bytes != tcgen05_extent_bytes(a->rows, a->cols) ||
        a->activation_len_bytes != a->activation_terms * staged_term_bytes(a->tokens, a->cols)) {
        return false;
    }
    Range r[4] = {{a->weight, a->weight_len_bytes, 256}, {a->activation, a->activation_len_bytes, 256}, plan_scratch_range(plan), {}};
    size_t count = 3;
    if (output != GemmOutput::kNone) {
        const uint64_t width = output == GemmOutput::kHalfWidth ? a->rows / 2 : a->rows;
        if (a->output_len_bytes != static_cast<uint64_t>(a->tokens) * width * 2) return false;
        r[count++] = {a->output_bf16, a->output_len_bytes, 16};
    } else if (a->output_bf16 || a->output_len_bytes) {
        return false;
    }
    if (!all_disjoint(r, count)) return false;
    if (!full) return true;
    // the plan's scratch was inspected when the plan was made
    if (!inspect_device_ranges(d, r, 2, failure)) return false;
    return output == GemmOutput::kNone || inspect_device_ranges(d, r + 3, 1, failure);
}

}  // namespace

// How many two-CTA clusters of the pair kernel fit the current device at once. The leftover-tile split lets
// a pair wait for parts that lower-numbered pairs produce, so every pair of the grid has to be resident:
// the grid is capped with this number (it can be below SMs / 2 when cluster placement leaves SMs unused).
uint32_t gemm_pair_resident_clusters() {
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(2);
    config.blockDim = dim3(kPairThreads);
    config.dynamicSmemBytes = kPairSmemBytes;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = 2;
    attribute.val.clusterDim.y = 1;
    attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    int fewest = INT_MAX;
    for (PairKernel kernel : kPairKernels) {
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) != cudaSuccess || clusters < 1) {
            cudaGetLastError();
            return 0;
        }
        if (clusters < fewest) fewest = clusters;
    }
    return static_cast<uint32_t>(fewest);
}

cudaError_t gemm_configure_device() {
    for (PairKernel kernel : kPairKernels) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemBytes);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace augur_sm100

using namespace augur_sm100;

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_gemm_plan_scratch_extent_host_v1(
    uint32_t sm_count, uint64_t* out_bytes) {
    if (!out_bytes || !sm_count || sm_count > 4096) return invalid();
    *out_bytes = kCounterBytes + static_cast<uint64_t>(sm_count / 2) * kSplitSlotBytes;
    return ok();
}

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_gemm_scratch_extent_host_v1(
    uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t activation_terms, uint64_t* out_bytes) {
    if (!out_bytes || !rows || rows % 128 != 0 || !act_shape_ok(tokens, cols, activation_terms)) return invalid();
    // The GEMM itself needs no scratch; a caller that lets the plan stage the quantised
    // activations needs this much.
    *out_bytes = activation_terms * staged_term_bytes(tokens, cols);
    return ok();
}

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_act_quant_preflight_v1(
    int32_t d, augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_act_quant_args_v1* a) {
    augur_cuda_result_v1 failure;
    return check_act_quant(d, s, a, true, &failure) ? ok() : failure;
}

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_act_quant_prevalidated_submit_v1(
    int32_t d, augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_act_quant_args_v1* a) {
    augur_cuda_result_v1 failure;
    if (!check_act_quant(d, s, a, false, &failure)) return failure;
    if (consume_injected_fault()) return make_result(AUGUR_CUDA_STATUS_DIAGNOSTIC_FAULT_INJECTED);
    const cudaError_t e = cudaSetDevice(d);
    if (e != cudaSuccess) return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE, e);
    const uint64_t groups = static_cast<uint64_t>(a->tokens) * (a->cols / 16);
    // Rows past `tokens` in the last 128-row tile (codes and scale bytes) are left as they are: they only
    // feed output rows that the GEMM never stores.
    // Spread: 6144 x 5120, three terms, 48 tokens 18.5 -> 17.2 us; 256 tokens 30.7 -> 30.4.
    launch_dependent_spread(s->stream, act_quant_kernel, static_cast<uint32_t>((groups + kQuantThreads - 1) / kQuantThreads), kQuantThreads,
                            reinterpret_cast<const uint16_t*>(a->input_bf16), reinterpret_cast<uint8_t*>(a->destination), a->tokens, a->cols,
                            a->terms, quant_scale(a->global_scale));
    count_launch();
    return submitted();
}

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_gemm_bf16_preflight_v1(
    int32_t d, augur_cuda_stream_t s, augur_cuda_nvfp4_sm100_plan_v1* plan,
    const augur_cuda_nvfp4_sm100_gemm_args_v1* a) {
    augur_cuda_result_v1 failure;
    if (!check_gemm(d, s, plan, a, true, &failure)) return failure;
    CUtensorMap probe;
    return make_code_map(&probe, a->weight, a->rows, a->cols) ? ok() : make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE);
}

namespace {
// Enqueues the GEMM of a validated descriptor. `swiglu`: a->rows counts the physical weight rows
// (gate and up interleaved), the output is a->rows / 2 wide.
struct QuantTarget {
    uint64_t destination = 0;
    uint32_t terms = 0;
    float global_scale = 0.0f;
};

// The choice of nvfp4_gemm_choice.h for this plan: a pair that hands a part over needs a slot of its scratch behind the counter regions, whose first words
// serve as the flags.
PairPlan plan_pairs(const augur_cuda_nvfp4_sm100_plan_v1* plan, uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t terms, bool swiglu) {
    const uint64_t slots = plan->scratch_bytes > kCounterBytes ? (plan->scratch_bytes - kCounterBytes) / kSplitSlotBytes : 0;
    return pair_plan(rows, cols, tokens, terms, swiglu, plan->pair_clusters, slots, gemm_narrow_ns(plan->ordinal, rows, cols, tokens, terms));
}

augur_cuda_result_v1 launch_gemm(augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_plan_v1* plan,
                                 const augur_cuda_nvfp4_sm100_gemm_args_v1* a, bool swiglu, float up_global_scale,
                                 QuantTarget quant = QuantTarget()) {
    // Tensor maps are encoded on the host into kernel parameter space: no allocation, no driver query.
    // The activation map spans the stacked code planes of all terms (terms * padded tokens rows).
    CUtensorMap map_weight;
    if (!make_code_map(&map_weight, a->weight, a->rows, a->cols)) return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE);
    GemmParams p{};
    p.weight_sf = reinterpret_cast<const uint8_t*>(a->weight) + tcgen05_codes_bytes(a->rows, a->cols);
    const uint32_t padded = padded_tokens(a->tokens);
    p.act_sf = reinterpret_cast<const uint8_t*>(a->activation) + a->activation_terms * tcgen05_codes_bytes(padded, a->cols);
    p.act_term_stride = tcgen05_scale_bytes(a->tokens, a->cols);
    p.out = reinterpret_cast<__nv_bfloat16*>(a->output_bf16);
    p.status_word = plan->status_word;
    p.rows = a->rows; p.cols = a->cols; p.tokens = a->tokens; p.terms = a->activation_terms;
    p.padded_tokens = padded;
    p.scale = a->weight_global_scale * a->activation_global_scale;
    p.scale_b = up_global_scale * a->activation_global_scale;
    p.swiglu = swiglu ? 1u : 0u;
    p.quant_out = reinterpret_cast<uint8_t*>(quant.destination);
    p.quant_terms = quant.terms;
    p.quant_scale = quant_scale(quant.global_scale);
    const PairPlan pairs = plan_pairs(plan, a->rows, a->cols, a->tokens, a->activation_terms, swiglu);
    p.token_pairs = pairs.token_pairs;
    if (p.token_pairs) {
        // 256 x 256 tiles on pairs of CTAs (clusters of two); the grid is a whole number of pairs.
        CUtensorMap map_act, map_act_sf, map_weight_sf;
        const uint64_t atoms = a->cols / 64;
        if (!make_code_map(&map_act, a->activation, static_cast<uint64_t>(a->activation_terms) * padded, a->cols) ||
            !make_scale_map(&map_weight_sf, reinterpret_cast<uint64_t>(p.weight_sf), a->rows / 128, atoms, 2) ||
            !make_scale_map(&map_act_sf, reinterpret_cast<uint64_t>(p.act_sf),
                            static_cast<uint64_t>(a->activation_terms) * (padded / 128), atoms, 1)) {
            return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE);
        }
        p.tail_columns = pairs.tail_columns;
        CUtensorMap map_tail = map_act;
        if (p.tail_columns && !make_code_map(&map_tail, a->activation, static_cast<uint64_t>(a->activation_terms) * padded, a->cols, p.tail_columns / 2)) {
            return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE);
        }
        p.cost_main = pair_block_cost(a->activation_terms, 0);
        p.cost_tail = pair_block_cost(a->activation_terms, p.tail_columns);
        if (pairs.split.sharers) {
            p.split_sharers = pairs.split.sharers;
            p.split_flags = reinterpret_cast<uint32_t*>(plan->scratch);
            p.split_slots = reinterpret_cast<float*>(plan->scratch + kCounterBytes);
        }
        launch_dependent(s->stream, kPairKernels[a->activation_terms - 1 + (p.quant_out ? 3 : 0)], 2 * pairs.split.pairs, kPairThreads, kPairSmemBytes, map_act, map_weight, map_act_sf, map_weight_sf, map_tail, p);
        count_launch();
        return submitted();
    }
    return launch_gemm_narrow(s, plan, map_weight, a->activation, p);
}

static_assert(sizeof(augur_cuda_nvfp4_sm100_gemm_swiglu_args_v1) == 88, "gemm_swiglu ABI");

// The fused form as a plain GEMM descriptor over the physical (interleaved) weight rows; false if the
// descriptor's own fields are bad. Output extent is checked here (it is half as wide).
bool swiglu_as_gemm(const augur_cuda_nvfp4_sm100_gemm_swiglu_args_v1* a, augur_cuda_nvfp4_sm100_gemm_args_v1* g) {
    if (a->reserved || !a->rows || a->rows % 64 != 0 || a->rows > (1u << 30) || !scale_ok(a->up_global_scale)) return false;
    if (a->output_len_bytes != static_cast<uint64_t>(a->tokens) * a->rows * 2) return false;
    *g = augur_cuda_nvfp4_sm100_gemm_args_v1{};
    g->abi_version = a->abi_version;
    g->struct_size = sizeof(*g);
    g->weight = a->weight; g->weight_len_bytes = a->weight_len_bytes;
    g->activation = a->activation; g->activation_len_bytes = a->activation_len_bytes;
    g->output_bf16 = a->output_bf16;
    g->rows = 2 * a->rows; g->cols = a->cols; g->tokens = a->tokens; g->activation_terms = a->activation_terms;
    g->output_len_bytes = static_cast<uint64_t>(a->tokens) * g->rows * 2;   // what check_gemm expects for 2*rows columns
    g->weight_global_scale = a->gate_global_scale; g->activation_global_scale = a->activation_global_scale;
    return true;
}
}  // namespace

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_gemm_bf16_prevalidated_submit_v1(
    int32_t d, augur_cuda_stream_t s, augur_cuda_nvfp4_sm100_plan_v1* plan,
    const augur_cuda_nvfp4_sm100_gemm_args_v1* a) {
    augur_cuda_result_v1 failure;
    if (!check_gemm(d, s, plan, a, false, &failure)) return failure;
    if (consume_injected_fault()) return make_result(AUGUR_CUDA_STATUS_DIAGNOSTIC_FAULT_INJECTED);
    const cudaError_t e = cudaSetDevice(d);
    if (e != cudaSuccess) return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE, e);
    return launch_gemm(s, plan, a, false, 0.0f);
}

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_gemm_swiglu_bf16_preflight_v1(
    int32_t d, augur_cuda_stream_t s, augur_cuda_nvfp4_sm100_plan_v1* plan,
    const augur_cuda_nvfp4_sm100_gemm_swiglu_args_v1* a) {
    if (!header_ok(d, s, a)) {
        if (a && s && d >= 0 && s->ordinal == d && a->abi_version != AUGUR_CUDA_ABI_VERSION_V1) {
            return make_result(AUGUR_CUDA_STATUS_ABI_VERSION_MISMATCH);
        }
        return invalid();
    }
    augur_cuda_nvfp4_sm100_gemm_args_v1 g;
    if (!swiglu_as_gemm(a, &g)) return invalid();
    augur_cuda_result_v1 failure;
    // the output range handed to the range checks is the real (half-width) one
    g.output_len_bytes = a->output_len_bytes;
    if (!check_gemm(d, s, plan, &g, true, &failure, GemmOutput::kHalfWidth)) return failure;
    CUtensorMap probe;
    return make_code_map(&probe, g.weight, g.rows, g.cols) ? ok() : make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE);
}

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_gemm_swiglu_bf16_prevalidated_submit_v1(
    int32_t d, augur_cuda_stream_t s, augur_cuda_nvfp4_sm100_plan_v1* plan,
    const augur_cuda_nvfp4_sm100_gemm_swiglu_args_v1* a) {
    if (!header_ok(d, s, a)) {
        if (a && s && d >= 0 && s->ordinal == d && a->abi_version != AUGUR_CUDA_ABI_VERSION_V1) {
            return make_result(AUGUR_CUDA_STATUS_ABI_VERSION_MISMATCH);
        }
        return invalid();
    }
    augur_cuda_nvfp4_sm100_gemm_args_v1 g;
    if (!swiglu_as_gemm(a, &g)) return invalid();
    augur_cuda_result_v1 failure;
    g.output_len_bytes = a->output_len_bytes;
    if (!check_gemm(d, s, plan, &g, false, &failure, GemmOutput::kHalfWidth)) return failure;
    if (consume_injected_fault()) return make_result(AUGUR_CUDA_STATUS_DIAGNOSTIC_FAULT_INJECTED);
    const cudaError_t e = cudaSetDevice(d);
    if (e != cudaSuccess) return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE, e);
    return launch_gemm(s, plan, &g, true, a->up_global_scale);
}

namespace {
static_assert(sizeof(augur_cuda_nvfp4_sm100_gemm_swiglu_quant_args_v1) == 112, "gemm_swiglu_quant ABI");

// An intermediate size that is a multiple of 128: its rows of gate and up fill whole 256-row tiles.
bool check_swiglu_quant(int32_t d, augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_plan_v1* plan,
                        const augur_cuda_nvfp4_sm100_gemm_swiglu_quant_args_v1* a, bool full,
                        augur_cuda_nvfp4_sm100_gemm_args_v1* g, augur_cuda_result_v1* failure) {
    *failure = invalid();
    if (!header_ok(d, s, a)) {
        if (a && s && d >= 0 && s->ordinal == d && a->abi_version != AUGUR_CUDA_ABI_VERSION_V1) {
            *failure = make_result(AUGUR_CUDA_STATUS_ABI_VERSION_MISMATCH);
        }
        return false;
    }
    if (a->reserved || !a->rows || a->rows % 128 != 0 || a->rows > (1u << 30) || !scale_ok(a->up_global_scale) ||
        a->destination_terms < 1 || a->destination_terms > 3 || !std::isfinite(a->destination_global_scale) ||
        a->destination_global_scale <= 0.0f || !a->tokens || !plan ||
        plan->sm_count < 2) {
        return false;
    }
    const bool writes_bf16 = a->output_bf16 != 0;
    if (!act_shape_ok(a->tokens, a->rows, a->destination_terms) ||
        a->destination_len_bytes != a->destination_terms * staged_term_bytes(a->tokens, a->rows)) {
        return false;
    }
    // the members it shares with the plain GEMM, over the physical (interleaved) weight rows
    *g = augur_cuda_nvfp4_sm100_gemm_args_v1{};
    g->abi_version = a->abi_version;
    g->struct_size = sizeof(*g);
    g->weight = a->weight; g->weight_len_bytes = a->weight_len_bytes;
    g->activation = a->activation; g->activation_len_bytes = a->activation_len_bytes;
    g->output_bf16 = a->output_bf16; g->output_len_bytes = a->output_len_bytes;
    g->rows = 2 * a->rows; g->cols = a->cols; g->tokens = a->tokens; g->activation_terms = a->activation_terms;
    g->weight_global_scale = a->gate_global_scale; g->activation_global_scale = a->activation_global_scale;
    if (!check_gemm(d, s, plan, g, full, failure, writes_bf16 ? GemmOutput::kHalfWidth : GemmOutput::kNone)) return false;
    *failure = invalid();
    // the staged destination against every other range
    const Range destination = {a->destination, a->destination_len_bytes, 256};
    const Range others[4] = {{a->weight, a->weight_len_bytes, 256}, {a->activation, a->activation_len_bytes, 256},
                             plan_scratch_range(plan), {a->output_bf16, a->output_len_bytes, 16}};
    for (size_t i = 0; i < (writes_bf16 ? 4u : 3u); ++i) {
        if (!disjoint(destination, others[i])) return false;
    }
    return !full || inspect_device_ranges(d, &destination, 1, failure);
}
}  // namespace

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_gemm_swiglu_quant_preflight_v1(
    int32_t d, augur_cuda_stream_t s, augur_cuda_nvfp4_sm100_plan_v1* plan,
    const augur_cuda_nvfp4_sm100_gemm_swiglu_quant_args_v1* a) {
    augur_cuda_nvfp4_sm100_gemm_args_v1 g;
    augur_cuda_result_v1 failure;
    if (!check_swiglu_quant(d, s, plan, a, true, &g, &failure)) return failure;
    CUtensorMap probe;
    return make_code_map(&probe, g.weight, g.rows, g.cols) ? ok() : make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE);
}

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_gemm_swiglu_quant_prevalidated_submit_v1(
    int32_t d, augur_cuda_stream_t s, augur_cuda_nvfp4_sm100_plan_v1* plan,
    const augur_cuda_nvfp4_sm100_gemm_swiglu_quant_args_v1* a) {
    augur_cuda_nvfp4_sm100_gemm_args_v1 g;
    augur_cuda_result_v1 failure;
    if (!check_swiglu_quant(d, s, plan, a, false, &g, &failure)) return failure;
    if (consume_injected_fault()) return make_result(AUGUR_CUDA_STATUS_DIAGNOSTIC_FAULT_INJECTED);
    const cudaError_t e = cudaSetDevice(d);
    if (e != cudaSuccess) return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE, e);
    QuantTarget quant;
    quant.destination = a->destination;
    quant.terms = a->destination_terms;
    quant.global_scale = a->destination_global_scale;
    return launch_gemm(s, plan, &g, true, a->up_global_scale, quant);
}
