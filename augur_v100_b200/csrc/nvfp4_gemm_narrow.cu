// Prefill NVFP4 GEMM for token counts that are narrow next to the weights (sm_100a): short prompts, and batched decode of
// more users than the small-token kernels take.
//
// The pair kernel of nvfp4_gemm.cu puts 256 token rows on its tile, so 9 tokens cost what 256 do. Here the weights are the
// 128-row operand and the tokens sit on the MMA n dimension, whose size follows their number in steps of 16 (at most
// 128): the work is that of the tokens there are, and what is left is streaming the weights once. What bounds a launch is a
// chain of latencies, a pipeline step (k block x term) behind the other, not HBM or the tensor pipe alone: with two CTAs on every SM and
// three terms a step takes 0.32 us at 16 tokens, 0.50 at 48 and 0.55 at 128, where the MMAs of the two CTAs occupy the pipe for 0.19 to 0.31 us
// (at 1.65 GHz) and HBM delivers the weights in 0.28; 6144 x 5120 at 48 tokens, five parts, has them 13 % and 9 % busy.
//
//   D[feature][token] = sum over k blocks of 256, terms, k steps of 64:  W[128 x 64] * A_term[tokens x 64]^T
//
// Two rings in shared memory, because a weight stage (16 KB of codes, 2 KB of block scales) serves all terms of its k block
// while an activation slot (tokens x 128 bytes of codes, 2 KB of scales) serves one term.
//
// An item is (128-row tile, token tile of at most 128), one per CTA. Two CTAs share an SM (112 KB of shared and half of tensor
// memory each): while one waits for its rings or stores its results the other feeds the tensor pipe (one CTA per SM with
// deeper rings took 30.4 us where this takes 22 for 17408 x 5120, 128 tokens, three terms). With fewer tiles than
// places a cluster of up to 8 CTAs shares an item, each CTA an equal range of its k blocks; when all are done every CTA
// reads the partial sums of its share of the columns from all of them over distributed shared memory and adds them in CTA
// order: no scratch, no fences to global memory, no atomics, and results that do not depend on scheduling. (The pair
// kernel's hand-over of leftover tiles through global memory is what most of its time goes to at these sizes.)
//
// Roles: warp 0 TMA and scale copies of the weights, 1 MMA, 2 TMA of the activations, 3 their scale copies to tensor memory,
// 4..11 epilogue. What a step costs beyond its bytes is the time its warps take to issue it: each waits on as few barriers
// as possible, and what it issues is one block of predicated instructions (tc_step, tc_copy_step, tma_step), one instantiation per number of
// terms: 9 tokens, three terms, quantiser included, 34816 x 5120 27.3 -> 24.0 us, 17408 x 5120 18.5 -> 16.8, 5120 x 17408 20.3 -> 18.5; 6144 x 5120 at 48
// 14.15 -> 13.7. From 96 tokens on nothing changed: there the bytes into shared memory are the bound, 24 KB a step and CTA, 80 a ns and SM.
// Every wait is bounded; a wait that runs out records a code in the plan's status word, raises a CTA-wide abort flag, and
// all roles fall through to the common exits. What a role waits for on a barrier never includes the launch before: a role that
// depends on it waits for its end first, so that its time does not count against the bound.
#include "nvfp4_gemm.cuh"
#include "nvfp4_gemm_choice.h"

namespace augur_sm100 {
namespace {
using namespace tc;

constexpr uint32_t kNarrowK = 256;                                    // k per stage = one 128-byte swizzled row of codes
constexpr uint32_t kNarrowCodes = kTileM * 128;                       // 16 KB
constexpr uint32_t kNarrowScales = 4 * kSfAtomBytes;                  // 2 KB: the 4 atoms of 128 rows
constexpr uint32_t kNarrowStage = kNarrowCodes + kNarrowScales;       // one weight stage
constexpr uint32_t kNarrowMaxDepth = 8;                               // slots of either ring
constexpr uint32_t kNarrowEpilogueWarps = 8;                          // two per tensor-memory lane quadrant
constexpr uint32_t kNarrowThreads = 32 * (4 + kNarrowEpilogueWarps);   // 12 warps: registers are handed out to warps by fours
// As if CTAs had 14 warps: 72 registers a thread instead of 80, no spills. Two CTAs of 12 warps with 80 take all but 4 K of an SM's
// 64 K registers and a quantiser CTA (5 K) fits beside one of them only, so half the CTAs began to load weights after the quantiser
// instead of under it (6144 x 5120, three terms, quantiser included: 256 tokens 31.8 -> 29.4 us, 128 tokens 24.2 -> 23.0).
constexpr uint32_t kNarrowBound = 32 * 14;
constexpr uint32_t kNarrowState = 1024;                               // barriers, tensor-memory base, abort flag, a counter per warp
constexpr uint32_t kNarrowTurnPitch = 36;                             // floats between columns of the transposition area: 16-byte reads hit all banks
constexpr uint32_t kNarrowSumPitch = 129;                             // 16-byte rows between groups of four columns of the partial sums, likewise
constexpr uint32_t kNarrowRowPitch = kTileM + 4;                      // floats between columns of finished sums on their way to SwiGLU, likewise
// Of two CTAs per SM. At 113 KB they took all of an SM's shared memory with what the system reserves for each, so that no quantiser
// CTA found room beside two of them: 17408 x 5120, three terms, 128 tokens 33.8 -> 30.8 us, 48 tokens 26.1 -> 24.4.
constexpr uint32_t kNarrowSmem = 112 * 1024;
constexpr uint32_t kNarrowTmemColumns = 256;
static_assert((6 * kNarrowMaxDepth + 1) * 8 + 8 + kNarrowThreads / 32 * 4 <= kNarrowState, "the small state fits");
static_assert(kTileM / 4 * kNarrowSumPitch * 16 + kTileM / 2 * kNarrowRowPitch * 4 <= kNarrowSmem - 1024 - kNarrowState,
              "partial sums of all columns and finished ones of half of them in the space of the rings");

constexpr uint32_t kErrNarrowWeights = 0x111, kErrNarrowTokens = 0x112, kErrNarrowFull = 0x113, kErrNarrowScales = 0x114,
                   kErrNarrowCopy = 0x115, kErrNarrowAccFull = 0x116;

struct NarrowParams {
    GemmParams g;
    uint32_t tile_tokens, token_tiles, columns;   // columns: MMA n, tile_tokens rounded up to 16
    uint32_t parts;                                       // CTAs per item (the cluster size)
    uint32_t weight_depth, token_depth, slot_bytes;       // ring slots, size of an activation slot
    uint32_t sf_weight, sf_token;                         // first tensor-memory columns of either ring's scales
};

// A row of 32 accumulator values of one token (weight rows row0 .. row0 + 31) -> output, quantised output.
__device__ __forceinline__ void narrow_store(const GemmParams& g, uint32_t token, uint32_t row0, const uint32_t (&v)[32]) {
    uint32_t packed[16];
    convert_chunk(v, g.scale, g.scale_b, g.swiglu != 0, packed);
    if (!g.swiglu) {
        uint4* dst = reinterpret_cast<uint4*>(g.out + static_cast<uint64_t>(token) * g.rows + row0);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) dst[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
        return;
    }
    const uint32_t out_width = g.rows / 2;
    if (g.out) {
        uint4* dst = reinterpret_cast<uint4*>(g.out + static_cast<uint64_t>(token) * out_width + row0 / 2);
        dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
    }
    if (g.quant_out) {
        // the 16 outputs are one quantisation group of the next GEMM's activations
        const uint32_t group = row0 / 32;
        const uint64_t code_bytes = tcgen05_codes_bytes(g.padded_tokens, out_width), scale_bytes = tcgen05_scale_bytes(g.padded_tokens, out_width);
        float2 residual[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) residual[i] = make_float2(__uint_as_float(packed[i] << 16), __uint_as_float(packed[i] & 0xffff0000u));
#pragma unroll 1
        for (uint32_t term = 0; term < g.quant_terms; ++term) {
            uint32_t codes[2], scale_code;
            quantise_term(residual, g.quant_scale, term + 1 < g.quant_terms, codes, &scale_code);
            *reinterpret_cast<uint2*>(g.quant_out + term * code_bytes + static_cast<uint64_t>(token) * (out_width / 2) + group * 8) = make_uint2(codes[0], codes[1]);
            g.quant_out[g.quant_terms * code_bytes + term * scale_bytes + tcgen05_scale_offset(token, group, out_width)] = static_cast<uint8_t>(scale_code);
        }
    }
}

// 16 bytes at this offset of another CTA's shared memory.
__device__ __forceinline__ float4 narrow_read_cluster(uint32_t offset, uint32_t cta) {
    uint32_t at;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(offset), "r"(cta));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

__device__ __forceinline__ void narrow_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <uint32_t kTerms>
__global__ void __launch_bounds__(kNarrowBound, 2)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap map_weight, const __grid_constant__ CUtensorMap map_act, const NarrowParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const GemmParams& g = p.g;
    uint8_t* slots = smem + p.weight_depth * kNarrowStage;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kNarrowSmem - 1024 - kNarrowState);
    const uint32_t bar0 = smem_u32(bars);
    // per slot of either ring: landed, free, scales in tensor memory (and with them the codes in shared memory)
    const uint32_t w_full = bar0, w_empty = bar0 + 8 * kNarrowMaxDepth, w_ready = bar0 + 16 * kNarrowMaxDepth;
    const uint32_t t_full = bar0 + 24 * kNarrowMaxDepth, t_empty = bar0 + 32 * kNarrowMaxDepth, t_ready = bar0 + 40 * kNarrowMaxDepth;
    const uint32_t acc_full = bar0 + 48 * kNarrowMaxDepth;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6 * kNarrowMaxDepth + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // The next kernel of the stream may become resident from here on (it waits for this one's end before it reads).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (uint32_t b = 0; b < 6 * kNarrowMaxDepth + 1; ++b) mbar_init(bar0 + 8 * b, 1);
        *abort_flag = 0;
        for (uint32_t w = 0; w < kNarrowThreads / 32; ++w) abort_flag[1 + w] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kNarrowTmemColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const uint32_t part = blockIdx.x % p.parts, item = blockIdx.x / p.parts;
    const uint32_t row_tile = item / p.token_tiles, token_row = item % p.token_tiles * p.tile_tokens;
    const uint32_t token_end = min(token_row + p.tile_tokens, g.tokens);
    const uint32_t k_blocks = (g.cols + kNarrowK - 1) / kNarrowK, atoms = g.cols / 64;      // scale atoms of a 128-row block along k
    const uint32_t kb0 = part * k_blocks / p.parts, kb1 = (part + 1) * k_blocks / p.parts;
    const uint32_t last_k_steps = atoms - (k_blocks - 1) * 4;                               // 1..4 k steps of 64 in the last k block

    if (warp == 0) {
        // ---------------- weights: TMA, and scale copies to tensor memory ----------------
        // They are constant, so nothing is waited for before the ring is filled. From then on the copies of a stage come first and
        // the load into the stage before it, whose MMAs are the ones under way, second: the copies stay a k block ahead.
        const uint64_t desc0 = sf_desc(smem_u32(smem) + kNarrowCodes);
        const uint8_t* scales = g.weight_sf + static_cast<uint64_t>(row_tile) * atoms * kSfAtomBytes;
        uint32_t load_kb = kb0, load_stage = 0, load_phase = 1, stage = 0, phase = 0;
        auto load = [&]() {
            if (!warp_look_wait(w_empty + 8 * load_stage, load_phase, abort_flag, g.status_word, kErrNarrowWeights)) return false;
            const uint32_t to = smem_u32(smem + load_stage * kNarrowStage), sf_bytes = (load_kb + 1 < k_blocks ? 4u : last_k_steps) * kSfAtomBytes;
            tma_step(w_full + 8 * load_stage, kNarrowCodes + sf_bytes, to, &map_weight, load_kb * 128, row_tile * kTileM, to + kNarrowCodes,
                     scales + static_cast<uint64_t>(load_kb) * kNarrowScales, sf_bytes);
            ++load_kb;
            if (++load_stage == p.weight_depth) { load_stage = 0; load_phase ^= 1; }
            return true;
        };
        bool alive = true;
        while (alive && load_kb < kb1 && load_kb < kb0 + p.weight_depth) alive = load();
        for (uint32_t kb = kb0; alive && kb < kb1; ++kb) {
            if (!warp_look_wait(w_full + 8 * stage, phase, abort_flag, g.status_word, kErrNarrowCopy)) break;
            tc_copy_step(tmem_base + p.sf_weight + stage * 16, desc0 + stage * (kNarrowStage >> 4), w_ready + 8 * stage);
            if (++stage == p.weight_depth) { stage = 0; phase ^= 1; }
            // the first wait for a stage to be free, which it is when the activations are there
            if (kb == kb0 + 1) asm volatile("griddepcontrol.wait;" ::: "memory");
            if (kb != kb0 && load_kb < kb1) alive = load();
        }
    } else if (warp == 2) {
        // ---------------- TMA of activations ----------------
        // They come from the launch before this one.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t slot = 0, phase = 1;
        bool alive = true;
        const uint8_t* scales = g.act_sf + static_cast<uint64_t>(token_row / 128) * atoms * kSfAtomBytes;
        for (uint32_t kb = kb0; alive && kb < kb1; ++kb) {
            const uint32_t sf_bytes = (kb + 1 < k_blocks ? 4u : last_k_steps) * kSfAtomBytes;
            const uint8_t* from = scales + static_cast<uint64_t>(kb) * kNarrowScales;
#pragma unroll
            for (uint32_t term = 0; term < kTerms; ++term) {
                if (!warp_look_wait(t_empty + 8 * slot, phase, abort_flag, g.status_word, kErrNarrowTokens)) {
                    alive = false;
                    break;
                }
                const uint32_t to = smem_u32(slots + slot * p.slot_bytes);
                tma_step(t_full + 8 * slot, p.columns * 128 + sf_bytes, to, &map_act, kb * 128, token_row + term * g.padded_tokens, to + p.columns * 128,
                         from + term * g.act_term_stride, sf_bytes);
                if (++slot == p.token_depth) { slot = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t stage = 0, w_phase = 0, slot = 0, t_phase = 0, accumulate = 0;
        bool alive = true;
        const uint32_t idesc = instr_desc(p.columns);
        const uint32_t w_desc0 = static_cast<uint32_t>(operand_desc(smem_u32(smem))), t_desc0 = static_cast<uint32_t>(operand_desc(smem_u32(slots)));
        const uint32_t slot_step = p.slot_bytes >> 4;
        for (uint32_t kb = kb0; alive && kb < kb1; ++kb) {
            if (!warp_look_wait(w_ready + 8 * stage, w_phase, abort_flag, g.status_word, kErrNarrowFull)) {
                alive = false;
                break;
            }
            const uint32_t k_steps = kb + 1 < k_blocks ? 4u : last_k_steps, w_desc = w_desc0 + stage * (kNarrowStage >> 4);
            const uint32_t sf_w = tmem_base + p.sf_weight + stage * 16, w_done = w_empty + 8 * stage;
            if (++stage == p.weight_depth) { stage = 0; w_phase ^= 1; }
#pragma unroll
            for (uint32_t term = 0; term < kTerms; ++term) {
                if (!warp_look_wait(t_ready + 8 * slot, t_phase, abort_flag, g.status_word, kErrNarrowScales)) {
                    alive = false;
                    break;
                }
                tc_step(tmem_base, w_desc, t_desc0 + slot * slot_step, idesc, sf_w, tmem_base + p.sf_token + slot * 16, accumulate, k_steps, t_empty + 8 * slot,
                        term + 1 == kTerms ? 1u : 0u, w_done);
                if (++slot == p.token_depth) { slot = 0; t_phase ^= 1; }
                accumulate = 1;
            }
        }
        if (alive && elect_one()) tc_commit(acc_full);
        __syncwarp();
    } else if (warp == 3) {
        // ---------------- scale copies of the activations, shared memory -> tensor memory ----------------
        // A slot lands after the MMAs that used it last are complete, so its scale columns are free. The codes landed on the same
        // barrier, so the MMA warp waits for the copies only.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t slot = 0, phase = 0;
        const uint64_t desc0 = sf_desc(smem_u32(slots) + p.columns * 128);
        const uint32_t slot_step = p.slot_bytes >> 4;
        for (uint32_t left = (kb1 - kb0) * kTerms; left; --left) {
            if (!warp_look_wait(t_full + 8 * slot, phase, abort_flag, g.status_word, kErrNarrowCopy)) break;
            tc_copy_step(tmem_base + p.sf_token + slot * 16, desc0 + slot * slot_step, t_ready + 8 * slot);
            if (++slot == p.token_depth) { slot = 0; phase ^= 1; }
        }
    }

    // ---------------- epilogue: tensor memory -> sums of 32 weight rows per lane and token -> global ----------------
    const bool epilogue = warp >= 4;
    const uint32_t quadrant = warp & 3, first_chunk = (warp - 4) >> 2;   // tensor-memory lanes 32 * quadrant .. + 31; every other 32 columns
    const uint32_t row0 = row_tile * kTileM + quadrant * 32;
    bool complete = true;
    if (epilogue) {
        asm volatile("griddepcontrol.wait;" ::: "memory");   // nothing is written while an earlier kernel may still read it
        // suspended: sixteen polling warps per SM took 2 to 3 % of the launch from those that issue
        complete = warp_wait_suspended(acc_full, 0, abort_flag, g.status_word, kErrNarrowAccFull);
        tc_fence_after();
    }
    __syncwarp();
    if (p.parts == 1) {
        if (epilogue && complete) {
            // all loads have landed and all MMAs have read them: the rings' space turns a chunk so that a lane holds the rows of one token
            float* turn = reinterpret_cast<float*>(smem) + (warp - 4) * 32 * kNarrowTurnPitch;
            for (uint32_t column = first_chunk * 32; token_row + column < token_end; column += 64) {
                uint32_t v[32];
                tc_load32(tmem_base + ((quadrant * 32) << 16) + column, v);
                tc_wait_ld();
#pragma unroll
                for (uint32_t i = 0; i < 32; ++i) turn[i * kNarrowTurnPitch + lane] = __uint_as_float(v[i]);
                __syncwarp();
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    const uint4 four = *reinterpret_cast<const uint4*>(turn + lane * kNarrowTurnPitch + 4 * i);
                    v[4 * i] = four.x; v[4 * i + 1] = four.y; v[4 * i + 2] = four.z; v[4 * i + 3] = four.w;
                }
                __syncwarp();   // the area is rewritten for the next chunk
                if (token_row + column + lane < token_end) narrow_store(g, token_row + column + lane, row0, v);
            }
        }
    } else {
        // Every CTA of the cluster finishes a share of the columns. It parks its sums in the space of its own rings, which are done
        // with; one meeting later all threads read the share's sums from all CTAs, four columns of a row each, every CTA's at once
        // (own is a multiple of four and a tile has 128 rows, so a warp's 32 lanes are always 32 rows of the same columns).
        // Sent to their owners instead, which takes a meeting more, and added by the few lanes that have a column, three terms: 1024 x 5120
        // at 32 tokens 11.9 us against 11.2, 6144 x 5120 at 48 tokens 15.7 against 15.5, 17408 x 5120 at 128 tokens 28.9 against 28.1.
        const uint32_t share = ((p.columns + p.parts - 1) / p.parts + 3) / 4 * 4, first = part * share;
        const uint32_t own = first < p.columns ? min(share, p.columns - first) : 0;
        float4* sums = reinterpret_cast<float4*>(smem);   // [group of four columns][row]
        float* turn = reinterpret_cast<float*>(sums + p.columns / 4 * kNarrowSumPitch);
        if (epilogue && complete) {
            for (uint32_t column = first_chunk * 32; column < p.columns; column += 64) {
                uint32_t v[32];
                tc_load32(tmem_base + ((quadrant * 32) << 16) + column, v);
                tc_wait_ld();
#pragma unroll
                for (uint32_t i = 0; i < 32; i += 4) {
                    if (column + i >= p.columns) break;
                    sums[(column + i) / 4 * kNarrowSumPitch + quadrant * 32 + lane] =
                        make_float4(__uint_as_float(v[i]), __uint_as_float(v[i + 1]), __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
                }
            }
        }
        __syncwarp();
        narrow_cluster_sync();
        const bool whole = *abort_flag == 0;
        for (uint32_t index = threadIdx.x; whole && index < own * (kTileM / 4); index += kNarrowThreads) {
            const uint32_t row = index % kTileM, column = index / kTileM * 4;
            const uint32_t here = smem_u32(sums + (first + column) / 4 * kNarrowSumPitch + row);
            float4 piece[kNarrowMaxParts], sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (uint32_t from = 0; from < kNarrowMaxParts; ++from) {
                if (from < p.parts) piece[from] = narrow_read_cluster(here, from);
            }
#pragma unroll
            for (uint32_t from = 0; from < kNarrowMaxParts; ++from) {
                if (from >= p.parts) break;
                sum.x += piece[from].x; sum.y += piece[from].y; sum.z += piece[from].z; sum.w += piece[from].w;
            }
            if (g.swiglu) {
                float* to = turn + column * kNarrowRowPitch + row;
                to[0] = sum.x; to[kNarrowRowPitch] = sum.y; to[2 * kNarrowRowPitch] = sum.z; to[3 * kNarrowRowPitch] = sum.w;
                continue;
            }
            // two rows go out as one word: the even lane of a pair takes the first two columns, the odd lane the other two
            const bool odd = row & 1;
            const float a = __shfl_xor_sync(0xffffffffu, odd ? sum.x : sum.z, 1), b = __shfl_xor_sync(0xffffffffu, odd ? sum.y : sum.w, 1);
            const __nv_bfloat162 words[2] = {__floats2bfloat162_rn((odd ? a : sum.x) * g.scale, (odd ? sum.z : a) * g.scale),
                                             __floats2bfloat162_rn((odd ? b : sum.y) * g.scale, (odd ? sum.w : b) * g.scale)};
            const uint32_t token = token_row + first + column + (odd ? 2 : 0);
            __nv_bfloat16* to = g.out + static_cast<uint64_t>(token) * g.rows + row_tile * kTileM + (row & ~1u);
            if (token < token_end) *reinterpret_cast<__nv_bfloat162*>(to) = words[0];
            if (token + 1 < token_end) *reinterpret_cast<__nv_bfloat162*>(to + g.rows) = words[1];
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // this CTA has read what it needs of the others
        if (g.swiglu) {
            __syncthreads();
            for (uint32_t index = threadIdx.x; whole && index < own * 4; index += kNarrowThreads) {
                const uint32_t column = index % own, rows32 = index / own;
                if (token_row + first + column >= token_end) continue;
                uint32_t v[32];
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    const uint4 four = *reinterpret_cast<const uint4*>(turn + column * kNarrowRowPitch + rows32 * 32 + 4 * i);
                    v[4 * i] = four.x; v[4 * i + 1] = four.y; v[4 * i + 2] = four.z; v[4 * i + 3] = four.w;
                }
                narrow_store(g, token_row + first + column, row_tile * kTileM + rows32 * 32, v);
            }
            __syncwarp();
        }
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");     // and the others of this one
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kNarrowTmemColumns) : "memory");
    }
}

// ---- host side ----------------------------------------------------------------------------------
using NarrowKernel = void (*)(CUtensorMap, CUtensorMap, NarrowParams);
constexpr NarrowKernel kNarrowKernels[3] = {gemm_narrow_kernel<1>, gemm_narrow_kernel<2>, gemm_narrow_kernel<3>};

// Clusters of `parts` CTAs that a launch may count on to run at once. The device holds 148 of 2, 93 of 3, 71 of 4, 56 of 5, 45 of
// 6, 37 of 7 and 33 of 8 on a B200 (they do not fill its SMs evenly); of those larger than 2 a sixteenth is left out, because they
// come to lie badly while the launch before still has CTAs of its own on the SMs, and a cluster that finds no place then waits for
// a whole wave (small-token linear at one token row: 56 clusters of 5 for 7168 x 4736 13.3 us, 56 of 4 9.2; 93 of 3 for
// 11904 x 5120 16.7 us, 93 of 2 11.1). Asked once per device; bind time fills the table. The question is put for a kernel of
// the same size that uses no tensor memory: for one that does the runtime always answers for one CTA per SM, although
// two fit when each allocates half of it.
__global__ void __launch_bounds__(kNarrowBound, 2) narrow_shape_kernel() {}

struct NarrowDevice {
    std::atomic<uint32_t> clusters[kNarrowMaxParts + 1];
};
NarrowDevice g_narrow_devices[64];

}  // namespace

uint32_t two_cta_clusters(int32_t ordinal, uint32_t parts) {
    std::atomic<uint32_t>& known = g_narrow_devices[ordinal & 63].clusters[parts];
    const uint32_t clusters = known.load();
    if (clusters) return clusters;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = parts;
    attribute.val.clusterDim.y = 1;
    attribute.val.clusterDim.z = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(parts);
    config.blockDim = dim3(kNarrowThreads);
    config.dynamicSmemBytes = kNarrowSmem;
    config.attrs = &attribute;
    config.numAttrs = 1;
    int found = 0;
    if (cudaOccupancyMaxActiveClusters(&found, narrow_shape_kernel, &config) != cudaSuccess || found < 1) {
        cudaGetLastError();
        found = 1;
    }
    if (parts > 2) found -= found / 16;
    known.store(static_cast<uint32_t>(found));
    return static_cast<uint32_t>(found);
}

namespace {
NarrowCut device_cut(int32_t ordinal, uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t terms) {
    uint32_t clusters[kNarrowMaxParts + 1] = {};
    for (uint32_t parts = 1; parts <= kNarrowMaxParts; ++parts) clusters[parts] = two_cta_clusters(ordinal, parts);
    return narrow_cut(clusters, rows, cols, tokens, terms);
}
}  // namespace

uint32_t gemm_narrow_ns(int32_t ordinal, uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t terms) {
    return device_cut(ordinal, rows, cols, tokens, terms).ns;
}

augur_cuda_result_v1 launch_gemm_narrow(augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_plan_v1* plan, const CUtensorMap& map_weight,
                                        uint64_t activation, const GemmParams& g) {
    NarrowParams p{};
    p.g = g;
    const NarrowCut cut = device_cut(plan->ordinal, g.rows, g.cols, g.tokens, g.terms);
    p.token_tiles = cut.token_tiles;
    p.tile_tokens = cut.tile_tokens;
    p.columns = cut.columns;
    p.parts = cut.parts;
    // Two k blocks of activations ahead, but not at the price of fewer than four weight stages; three slots at least.
    const uint32_t room = kNarrowSmem - 1024 /*alignment*/ - kNarrowState;
    p.slot_bytes = p.columns * 128 + kNarrowScales;
    p.token_depth = 2 * g.terms < 4 ? 4 : 2 * g.terms;
    while (p.token_depth > 3 && room < p.token_depth * p.slot_bytes + 4 * kNarrowStage) --p.token_depth;
    p.weight_depth = (room - p.token_depth * p.slot_bytes) / kNarrowStage;
    p.sf_weight = (p.columns + 31) / 32 * 32;
    p.sf_token = p.sf_weight + 16 * p.weight_depth;
    static_assert(128 + 16 * (kNarrowSmem / kNarrowStage) <= kNarrowTmemColumns, "scale columns of all slots fit beside the accumulator");
    // A slot index past the barrier arrays would reach the accumulator's barrier and the tensor-memory base word.
    static_assert(kNarrowSmem / kNarrowStage <= kNarrowMaxDepth && 2 * 3 /*terms*/ <= kNarrowMaxDepth, "every slot of both rings has its barriers");
    CUtensorMap map_act;
    if (!make_code_map(&map_act, activation, static_cast<uint64_t>(g.terms) * g.padded_tokens, g.cols, p.columns)) {
        return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE);
    }
    cudaLaunchAttribute attributes[2]{};
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = p.parts;
    attributes[1].val.clusterDim.y = 1;
    attributes[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t config{};
    config.stream = s->stream;
    config.attrs = attributes;
    config.numAttrs = p.parts > 1 ? 2 : 1;
    config.gridDim = dim3(g.rows / kTileM * p.token_tiles * p.parts);
    config.blockDim = dim3(kNarrowThreads);
    config.dynamicSmemBytes = kNarrowSmem;
    cudaLaunchKernelEx(&config, kNarrowKernels[g.terms - 1], map_weight, map_act, p);
    count_launch();
    return submitted();
}

cudaError_t gemm_narrow_configure_device() {
    cudaError_t e = cudaSuccess;
    for (NarrowKernel kernel : kNarrowKernels) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kNarrowSmem);
    }
    if (e == cudaSuccess) e = cudaFuncSetAttribute(narrow_shape_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kNarrowSmem);
    int ordinal = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&ordinal);
    if (e != cudaSuccess) return e;
    for (uint32_t parts = 1; parts <= kNarrowMaxParts; ++parts) two_cta_clusters(ordinal, parts);
    return cudaSuccess;
}

}  // namespace augur_sm100
