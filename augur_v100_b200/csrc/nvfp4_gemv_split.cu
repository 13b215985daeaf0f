// Small-token (1..8) NVFP4 linear on tensor memory for sm_100a: the weights stream from HBM to the tensor cores
// (tcgen05.mma kind::mxf4nvf4, 128 weight rows x 64 columns of term * 8 + token), one (128-row tile, k range) per CTA, the k ranges of a tile in a
// cluster whose CTAs meet in distributed shared memory.
//
// What bounds a linear of a decode step is the chain of things that wait for one another, not its bytes: 10 to 50 MB are 2 to 8
// us of HBM time. So the token rows become radix-8 digits (nvfp4_digits.cuh) where they are used: every CTA turns its own k range of them
// into the operand image of its ring slots, a 256-deep chunk at a time, ahead of the MMAs, anchored at the largest magnitude of that
// range. The first MMA comes about two microseconds after the input is there. A launch of its own that splits the rows once for all CTAs takes
// four, half of them its end and hand-over; it stays where a CTA has many chunks of many token rows (split_linear_own_digits), because the
// integer work, 270 instructions for eight elements in every lane, is done by every CTA again. us, launch ahead / own digits: 17408 x 5120 at 1 token row
// 13.7 / 12.3, at 8 14.9 / 14.6; 5120 x 5120 8.3 / 6.6, 9.8 / 8.8; 1024 x 5120 7.0 / 5.1, 7.0 / 7.0; two layers of linears and MLP blocks 155.7 / 149.4.
//
// Roles: warp 0 weights (TMA, scale copies), 1 MMA, 2 scale copies of the activations, 3 TMA of digits that a launch ahead left, 4..11 own digits, then
// epilogue. What a warp issues
// for a step is one block of predicated instructions (tc_step and its like). Every wait is bounded; a wait that runs out records a
// code in the plan's status word, raises a CTA-wide abort flag, and all roles fall through to the common exit.
#include "nvfp4_digits.cuh"
#include "nvfp4_gemm.cuh"
#include "nvfp4_internal.h"

namespace augur_sm100 {
namespace {
using namespace tc;

constexpr uint32_t kSplitThreads = 256;
constexpr uint32_t kSliceGroups = 16;                                  // 16-element groups of a row per split CTA: one pair per warp
constexpr uint32_t kNonFinite = 255;                                   // anchor of a row with an infinity or a NaN

constexpr uint32_t kStreamWeightStage = kStageCodeBytes + kStageSfBytes;   // 18 KB
constexpr uint32_t kStreamActStage = kChunkBytes + kStageSfBytes;          // 10 KB
constexpr uint32_t kStreamWeightDepth = 4, kStreamActDepth = 3;
constexpr uint32_t kStreamExchange = 8 * 1024;                         // the cluster's sums of the token rows and weight rows this CTA finishes
constexpr uint32_t kStreamState = 512;                                 // barriers, tensor-memory base, abort flag, a counter per warp, the rows' maxima
constexpr uint32_t kStreamRings = kStreamWeightDepth * kStreamWeightStage + kStreamActDepth * kStreamActStage;
constexpr uint32_t kStreamSmem = kStreamRings + kStreamExchange + kStreamState + 1024 /*alignment*/;
constexpr uint32_t kStreamThreads = 32 * 12;
constexpr uint32_t kStreamWorkers = 8;                                 // warps 4..11
constexpr uint32_t kStreamAhead = 10;                                  // 16-byte pieces of the token rows in flight per lane
constexpr uint32_t kStreamTmemColumns = 256;
constexpr uint32_t kStreamSfWeight = 64, kStreamSfAct = kStreamSfWeight + 16 * kStreamWeightDepth;   // behind the accumulator's 64 columns
static_assert(kStreamSfAct + 16 * kStreamActDepth <= kStreamTmemColumns, "tensor memory columns");
static_assert(2 * (kStreamSmem + 1024) <= 228 * 1024, "two CTAs per SM, a kilobyte each reserved by the system");

constexpr uint32_t kErrStreamWeights = 0x311, kErrStreamTokens = 0x312, kErrStreamFull = 0x313, kErrStreamScales = 0x314,
                   kErrStreamCopy = 0x315, kErrStreamAccFull = 0x316;

struct StreamParams {
    const uint8_t* weight_sf;     // scale region of the weight
    const uint16_t* x;            // token rows, BF16 (own digits)
    const uint8_t* split;         // the split activations and their anchors (digits of a launch ahead)
    const uint32_t* anchors;
    void* out;
    uint32_t* status_word;
    uint32_t out_rows, cols, tokens, epilogue, parts;
    float global_a, global_b;
};

// ---- digits ----------------------------------------------------------------------------------------
// Eight neighbouring elements of token row `token` in a lane, the 256 of a chunk in a warp -> the row's eight lines (term * 8 + token) of the
// slot's operand image and its block scales. The digits are those of nvfp4_digits.cuh: with A the exponent field of the row's largest
// magnitude in this CTA's k range and G that of the 16-element group's (a lane and its neighbour), not less than A - 17, an element is the
// integer x * 2^(148 - G), formed by the one rounding of a multiply-add that leaves it in the low bits of the sum. It is taken with its
// sign: plus 4 in every octal place its octal digits are the digits plus 4 either way.
template <bool kSmall>
__device__ __forceinline__ void split_octet(uint8_t* slot, const uint4 words, uint32_t row_largest, uint32_t token, uint32_t lane) {
    const uint32_t w[4] = {words.x, words.y, words.z, words.w};
    uint32_t largest = __vmaxu2(__vmaxu2(w[0] & 0x7fff7fffu, w[1] & 0x7fff7fffu), __vmaxu2(w[2] & 0x7fff7fffu, w[3] & 0x7fff7fffu));
    largest = max(largest & 0xffffu, largest >> 16);
    largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
    const int a = static_cast<int>(min(max(row_largest >> 7, 1u), 254u));   // any finite row, subnormal values with the smallest normal ones
    const int g = max(max(static_cast<int>(largest >> 7), 1), a - 17);
    // 2^(148 - G) is an F32 number from G = 21 on, which A = 38 guarantees; smaller rows (`kSmall`) are brought up by 2^64 first (exactly)
    const float scale = __uint_as_float(static_cast<uint32_t>((kSmall ? 211 : 275) - g) << 23);
    // The code of digit + 4 = 0 .. 7: from 4 on the digit, below it the sign and 4 minus that. Byte permutations look four digits up at a time.
    constexpr uint32_t kCodesLow = 0x090a0b0cu, kCodesHigh = 0x03020100u;
    uint32_t low[4], high[4];   // byte t: codes of terms t and 4 + t of two neighbouring elements
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        float x = __uint_as_float(i & 1 ? w[i >> 1] & 0xffff0000u : w[i >> 1] << 16);
        if (kSmall) x *= 0x1p64f;
        // 1.5 * 2^23 plus the integer (below 2^22): its low bits. Then 4 in every octal place, and the octal digits one to a nibble, by
        // multiply-adds as far as possible: the integer pipe for logic and shifts is what bounds the kernel at eight token rows.
        uint32_t d = __float_as_uint(__fmaf_rn(x, scale, 12582912.0f)) + (0x924924u - 0x4b400000u);
        d += 15u * (d & 0x00fff000u);
        d += 3u * (d & 0x0fc00fc0u);
        d += d & 0x38383838u;
        const uint32_t codes_low = __byte_perm(kCodesLow, kCodesHigh, d), codes_high = __byte_perm(kCodesLow, kCodesHigh, __umulhi(d, 65536u));
        low[i >> 1] = i & 1 ? low[i >> 1] + 16u * codes_low : codes_low;
        high[i >> 1] = i & 1 ? high[i >> 1] + 16u * codes_high : codes_high;
    }
    uint32_t line[8];   // line[t]: the eight codes of term t; 4 x 4 bytes transposed
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t (&b)[4] = h ? high : low;
        const uint32_t p0 = __byte_perm(b[0], b[1], 0x5140), p1 = __byte_perm(b[2], b[3], 0x5140);   // bytes 0, 0, 1, 1
        const uint32_t p2 = __byte_perm(b[0], b[1], 0x7362), p3 = __byte_perm(b[2], b[3], 0x7362);   // bytes 2, 2, 3, 3
        line[4 * h] = __byte_perm(p0, p1, 0x5410);
        line[4 * h + 1] = __byte_perm(p0, p1, 0x7632);
        line[4 * h + 2] = __byte_perm(p2, p3, 0x5410);
        line[4 * h + 3] = __byte_perm(p2, p3, 0x7632);
    }
    uint8_t* to = slot + token * 128 + (((lane >> 2) ^ token) << 4) + (lane & 3) * 4;   // rows in the 128-byte swizzle of an operand tile
#pragma unroll
    for (uint32_t t = 0; t < 8; ++t) *reinterpret_cast<uint32_t*>(to + t * 1024) = line[t];
    // block scale 2^q, q = G + 8 - A from -9 to 8, in E4M3: eight lanes hold the four groups of an atom, one word for every term
    const int q = min(g + 8 - a, 8);
    uint32_t scales = (q >= -6 ? static_cast<uint32_t>(q + 7) << 3 : 1u << (q + 9)) << (8 * ((lane >> 1) & 3));
    scales |= __shfl_xor_sync(0xffffffffu, scales, 2);
    scales |= __shfl_xor_sync(0xffffffffu, scales, 4);
    const uint32_t n = (lane & 7) * 8 + token;
    *reinterpret_cast<uint32_t*>(slot + kChunkBytes + (lane >> 3) * kSfAtomBytes + (n & 31) * 16 + (n >> 5) * 4) = scales;
}

// ---- split of a launch of its own ----------------------------------------------------------------
// grid (slices, token rows). Every CTA reads its whole row for the largest magnitude (10 KB from L2 at 5120 columns; sharing the
// maximum between CTAs would cost a meeting) and splits its slice with the exact anchor.
__global__ void __launch_bounds__(kSplitThreads)
split_rows_kernel(const uint16_t* __restrict__ x, uint8_t* __restrict__ split, uint32_t* __restrict__ anchors, uint32_t cols) {
    __shared__ uint32_t maxima[kSplitThreads / 32], row_anchor[8];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, token = blockIdx.y, groups = cols / 16;
    const uint16_t* row = x + static_cast<uint64_t>(token) * cols;
    const uint32_t group = blockIdx.x * kSliceGroups + warp * 2 + (lane >> 4);
    // A row that is not in L2 would queue behind the weight copies that the stream kernel has already issued, so every CTA asks
    // for its slice of the row now. (The launch before may still write it; L2 then holds what it writes.)
    if (threadIdx.x < kSliceGroups / 4 && blockIdx.x * kSliceGroups + threadIdx.x * 4 < groups) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(row + (blockIdx.x * kSliceGroups + threadIdx.x * 4) * 16));
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");   // x may come from the launch before, and the split may still be read by it
    const uint32_t bits = group < groups ? __ldcg(row + group * 16 + (lane & 15)) : 0;
    uint32_t packed = 0;
    const uint4* vectors = reinterpret_cast<const uint4*>(row);
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < cols / 8; i += kSplitThreads) {
        const uint4 v = __ldcg(vectors + i);
        packed = __vmaxu2(packed, __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu)));
    }
    // the codes only need the group's own maximum: they are formed and stored while the row is still arriving
    const SplitTarget to{split, static_cast<uint32_t>(split_code_bytes(cols)), 0, groups, 8};
    const uint2 where = make_uint2(group < groups ? token : ~0u, group);
    const uint32_t group_largest = split_codes(to, where, bits, 0, lane);
    const uint32_t most = __reduce_max_sync(0xffffffffu, max(packed & 0xffffu, packed >> 16));
    if (lane == 0) maxima[warp] = most;
    __syncthreads();
    uint32_t largest = 0;
#pragma unroll
    for (uint32_t i = 0; i < kSplitThreads / 32; ++i) largest = max(largest, maxima[i]);
    const uint32_t a = min(max(largest >> 7, 1u), 254u);   // any finite row, subnormal values with the smallest normal ones
    if (threadIdx.x == 0 && blockIdx.x == 0) anchors[token] = largest >= 0x7f80u ? kNonFinite : a;   // the row's outputs are NaN then
    if (lane == 0) row_anchor[token] = a;   // every warp the same value
    __syncwarp();
    split_scales(to, row_anchor, where, bits, group_largest, lane);
}

// The first look at a barrier is in line, the rest suspended where the issue slots are for digits; where a launch ahead has formed them, polling: 10112 x 8448 at
// seven token rows 15.2 us suspended, 15.0 polling, 10240 x 8192 at six 14.7 and 14.6, 5120 x 17408 at seven 18.1 and 17.9.
template <bool kOwnDigits>
__device__ __forceinline__ bool stream_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* status_word, uint32_t code) {
    if (!kOwnDigits) return warp_wait(bar, parity, abort_flag, status_word, code);
    return mbar_test(bar, parity) || warp_wait_suspended(bar, parity, abort_flag, status_word, code);
}

// ---- stream ---------------------------------------------------------------------------------------
// Four neighbouring columns of this warp's 32 accumulator rows.
__device__ __forceinline__ void load_columns(uint32_t taddr, uint32_t (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
}

// Finished sums of 32 weight rows (lane = row) for the token rows token0 .. token0 + 3.
__device__ __forceinline__ void store_rows(const StreamParams& p, uint32_t row0, uint32_t token0, uint32_t lane, const float (&y)[4]) {
    if (p.epilogue == AUGUR_NVFP4_SM100_EPILOGUE_SWIGLU_BF16) {
        // 32 physical rows = 16 gate rows (lanes 0..15) and the matching 16 up rows (lanes 16..31)
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const float up = __shfl_sync(0xffffffffu, y[j], (lane & 15) + 16) * p.global_b, gate = y[j] * p.global_a;
            if (lane < 16 && token0 + j < p.tokens) {
                static_cast<__nv_bfloat16*>(p.out)[static_cast<uint64_t>(token0 + j) * p.out_rows + row0 / 2 + lane] =
                    __float2bfloat16_rn(__fdividef(gate, 1.0f + __expf(-gate)) * up);   // a few ulp of f32, far below the rounding
            }
        }
        return;
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        if (token0 + j >= p.tokens) continue;
        const float value = y[j] * p.global_a;
        const uint64_t at = static_cast<uint64_t>(token0 + j) * p.out_rows + row0 + lane;
        if (p.epilogue == AUGUR_NVFP4_SM100_EPILOGUE_LINEAR_F32) static_cast<float*>(p.out)[at] = value;
        else static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(value);
    }
}

template <bool kOwnDigits>
__global__ void __launch_bounds__(kStreamThreads, 2)
split_stream_kernel(const __grid_constant__ CUtensorMap map_weight, const __grid_constant__ StreamParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* slots = smem + kStreamWeightDepth * kStreamWeightStage;
    float4* exchange = reinterpret_cast<float4*>(smem + kStreamRings);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStreamRings + kStreamExchange);
    const uint32_t bar0 = smem_u32(bars);
    // per slot of either ring: there, free, scales in tensor memory (and with them the codes in shared memory)
    constexpr uint32_t kBars = 3 * (kStreamWeightDepth + kStreamActDepth) + 1;
    const uint32_t w_full = bar0, w_empty = w_full + 8 * kStreamWeightDepth, w_ready = w_empty + 8 * kStreamWeightDepth;
    const uint32_t t_full = w_ready + 8 * kStreamWeightDepth, t_empty = t_full + 8 * kStreamActDepth, t_ready = t_empty + 8 * kStreamActDepth;
    const uint32_t acc_full = t_ready + 8 * kStreamActDepth;
    static_assert(kBars * 8 + 8 + kStreamThreads / 32 * 4 + 8 * 4 <= kStreamState, "the small state fits");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBars);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    uint32_t* row_largest = tmem_slot + 2 + kStreamThreads / 32;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (uint32_t b = 0; b < kBars; ++b) {
            const bool digits = bar0 + 8 * b >= t_full && bar0 + 8 * b < t_empty;   // a warp for every token row of a chunk
            mbar_init(bar0 + 8 * b, kOwnDigits && digits ? p.tokens : 1);
        }
        *abort_flag = 0;
        for (uint32_t w = 0; w < kStreamThreads / 32; ++w) abort_flag[1 + w] = 0;
        for (uint32_t token = 0; token < 8; ++token) row_largest[token] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kStreamTmemColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // first half of a meeting of the cluster: this CTA runs (its shared memory may be written from the second half on)
    if (p.parts > 1) asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");

    const uint32_t part = blockIdx.x % p.parts, tile = blockIdx.x / p.parts;
    const uint32_t k_blocks = (p.cols + kStageK - 1) / kStageK, atoms = p.cols / 64;
    const uint32_t kb0 = part * k_blocks / p.parts, kb1 = (part + 1) * k_blocks / p.parts;
    const uint32_t last_k_steps = atoms - (k_blocks - 1) * 4;   // 1..4 k steps of 64 in the last k block
    bool alive = true;

    if (warp == 0) {
        // ---------------- weights: TMA, and scale copies to tensor memory ----------------
        // They are constant, so nothing is waited for before the ring is filled. From then on the copies of a stage come first and
        // the load into the stage before it, whose MMAs are the ones under way, second: the copies stay a k block ahead.
        const uint64_t desc0 = sf_desc(smem_u32(smem) + kStageCodeBytes);
        const uint8_t* scales = p.weight_sf + static_cast<uint64_t>(tile) * atoms * kSfAtomBytes;
        uint32_t load_kb = kb0, load_stage = 0, load_phase = 1, stage = 0, phase = 0;
        auto load = [&]() {
            if (!stream_wait<kOwnDigits>(w_empty + 8 * load_stage, load_phase, abort_flag, p.status_word, kErrStreamWeights)) return false;
            const uint32_t to = smem_u32(smem + load_stage * kStreamWeightStage), sf_bytes = (load_kb + 1 < k_blocks ? 4u : last_k_steps) * kSfAtomBytes;
            tma_step(w_full + 8 * load_stage, kStageCodeBytes + sf_bytes, to, &map_weight, load_kb * 128, tile * kTileM, to + kStageCodeBytes,
                     scales + static_cast<uint64_t>(load_kb) * kStageSfBytes, sf_bytes);
            ++load_kb;
            if (++load_stage == kStreamWeightDepth) { load_stage = 0; load_phase ^= 1; }
            return true;
        };
        while (alive && load_kb < kb1 && load_kb < kb0 + kStreamWeightDepth) alive = load();
        for (uint32_t kb = kb0; alive && kb < kb1; ++kb) {
            if (!stream_wait<kOwnDigits>(w_full + 8 * stage, phase, abort_flag, p.status_word, kErrStreamCopy)) break;
            tc_copy_step(tmem_base + kStreamSfWeight + stage * 16, desc0 + stage * (kStreamWeightStage >> 4), w_ready + 8 * stage);
            if (++stage == kStreamWeightDepth) { stage = 0; phase ^= 1; }
            // the first wait for a stage to be free, which it is when the activations are there
            if (kb == kb0 + 1) asm volatile("griddepcontrol.wait;" ::: "memory");
            if (kb != kb0 && load_kb < kb1) alive = load();
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t stage = 0, w_phase = 0, slot = 0, t_phase = 0;
        const uint32_t idesc = instr_desc(kCols);
        const uint32_t w_desc0 = static_cast<uint32_t>(operand_desc(smem_u32(smem))), t_desc0 = static_cast<uint32_t>(operand_desc(smem_u32(slots)));
        for (uint32_t kb = kb0; kb < kb1; ++kb) {
            if (!stream_wait<kOwnDigits>(w_ready + 8 * stage, w_phase, abort_flag, p.status_word, kErrStreamFull) ||
                !stream_wait<kOwnDigits>(t_ready + 8 * slot, t_phase, abort_flag, p.status_word, kErrStreamScales)) {
                alive = false;
                break;
            }
            tc_step(tmem_base, w_desc0 + stage * (kStreamWeightStage >> 4), t_desc0 + slot * (kStreamActStage >> 4), idesc, tmem_base + kStreamSfWeight + stage * 16,
                    tmem_base + kStreamSfAct + slot * 16, kb != kb0 ? 1u : 0u, kb + 1 < k_blocks ? 4u : last_k_steps, t_empty + 8 * slot, 1u, w_empty + 8 * stage);
            if (++stage == kStreamWeightDepth) { stage = 0; w_phase ^= 1; }
            if (++slot == kStreamActDepth) { slot = 0; t_phase ^= 1; }
        }
        if (alive && elect_one()) tc_commit(acc_full);
        __syncwarp();
    } else if (warp == 2) {
        // ---------------- scale copies of the activations ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t slot = 0, phase = 0;
        const uint64_t desc0 = sf_desc(smem_u32(slots) + kChunkBytes);
        for (uint32_t kb = kb0; kb < kb1; ++kb) {
            if (!stream_wait<kOwnDigits>(t_full + 8 * slot, phase, abort_flag, p.status_word, kErrStreamCopy)) break;
            tc_copy_step(tmem_base + kStreamSfAct + slot * 16, desc0 + slot * (kStreamActStage >> 4), t_ready + 8 * slot);
            if (++slot == kStreamActDepth) { slot = 0; phase ^= 1; }
        }
    } else if (warp == 3 && !kOwnDigits) {
        // ---------------- TMA of the digits that the launch ahead has left (the image in memory is the one the ring holds) ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint8_t* image_sf = p.split + split_code_bytes(p.cols);
        uint32_t slot = 0, phase = 1;
        for (uint32_t kb = kb0; kb < kb1; ++kb) {
            if (!stream_wait<kOwnDigits>(t_empty + 8 * slot, phase, abort_flag, p.status_word, kErrStreamTokens)) break;
            const uint32_t to = smem_u32(slots + slot * kStreamActStage), full = t_full + 8 * slot;
            if (elect_one()) {
                mbar_expect_tx(full, kStreamActStage);
                bulk_load(to, p.split + static_cast<uint64_t>(kb) * kChunkBytes, kChunkBytes, full);
                bulk_load(to + kChunkBytes, image_sf + static_cast<uint64_t>(kb) * kStageSfBytes, kStageSfBytes, full);
            }
            __syncwarp();
            if (++slot == kStreamActDepth) { slot = 0; phase ^= 1; }
        }
    } else if (warp >= 4 && !kOwnDigits) {
        asm volatile("griddepcontrol.wait;" ::: "memory");   // the anchors; and nothing is written while an earlier kernel may still read it
    } else if (warp >= 4) {
        // ---------------- digits ----------------
        // Each token row has `share` warps of its own, which take its chunks in turn. (Not more than three: a warp that has waited for a chunk's
        // slot knows that the MMAs of all chunks up to three before it are complete, and the phase of the barrier that it waits
        // on for the next of its chunks is then the one meant.)
        const uint32_t share = p.tokens <= 2 ? 3 : p.tokens <= 4 ? 2 : 1, token = (warp - 4) / share, chunks = kb1 - kb0;
        const uint32_t own_chunks = chunks - (kb1 == k_blocks && lane >= last_k_steps * 8 ? 1u : 0u);   // those in which this lane has elements
        uint32_t chunk = (warp - 4) % share;
        if (token >= p.tokens) chunk = chunks;
        const uint4* at = reinterpret_cast<const uint4*>(p.x) + static_cast<uint64_t>(token) * (p.cols / 8) + (kb0 + chunk) * 32 + lane;
        asm volatile("griddepcontrol.wait;" ::: "memory");   // x may come from the launch before; and nothing is written while that may still read it
        // the largest magnitude, the loads of ten chunks in flight at once
        uint4 words = make_uint4(0, 0, 0, 0);
        uint32_t most = 0;
        const uint4* from = at;
        for (uint32_t c = chunk; c < chunks; c += kStreamAhead * share) {
            uint4 v[kStreamAhead];
#pragma unroll
            for (uint32_t i = 0; i < kStreamAhead; ++i) {
                v[i] = c + i * share < own_chunks ? __ldcg(from) : make_uint4(0, 0, 0, 0);
                from += share * 32;
            }
            if (c == chunk) words = v[0];
#pragma unroll
            for (uint32_t i = 0; i < kStreamAhead; ++i) {
                most = __vmaxu2(most, __vmaxu2(__vmaxu2(v[i].x & 0x7fff7fffu, v[i].y & 0x7fff7fffu), __vmaxu2(v[i].z & 0x7fff7fffu, v[i].w & 0x7fff7fffu)));
            }
        }
        most = __reduce_max_sync(0xffffffffu, max(most & 0xffffu, most >> 16));
        if (lane == 0 && token < p.tokens) atomicMax(row_largest + token, most);
        asm volatile("bar.sync 1, %0;" ::"r"(kStreamWorkers * 32) : "memory");
        const uint32_t largest = token < 8 ? row_largest[token] : 0;
        uint32_t slot = chunk % kStreamActDepth, phase = 1;   // the first of a warp's chunks lies in the first use of the ring
        for (; chunk < chunks; chunk += share) {
            at += share * 32;
            const uint4 next = chunk + share < own_chunks ? __ldcg(at) : make_uint4(0, 0, 0, 0);
            if (!warp_wait(t_empty + 8 * slot, phase, abort_flag, p.status_word, kErrStreamTokens)) {
                alive = false;
                break;
            }
            __syncwarp();
            if (largest >> 7 >= 38) split_octet<false>(slots + slot * kStreamActStage, words, largest, token, lane);
            else split_octet<true>(slots + slot * kStreamActStage, words, largest, token, lane);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(t_full + 8 * slot);
            words = next;
            slot += share;
            if (slot >= kStreamActDepth) { slot -= kStreamActDepth; phase ^= 1; }
        }
    }

    // ---------------- epilogue: two warps per quarter of the rows, four token rows each ----------------
    const bool epilogue = warp >= 4;
    const uint32_t task = warp - 4, quadrant = task & 3, token0 = (task >> 2) * 4;   // quadrant == warp % 4: the tensor-memory lanes it may read
    float y[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    bool complete = false;
    if (epilogue && alive) {
        float scale[2][4];   // term 0 of a row has the global scale 2^(A - 155), which need not be an F32 number: as the product of two that are
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t a = kOwnDigits ? row_largest[token0 + j] >> 7 : token0 + j < p.tokens ? __ldcg(p.anchors + token0 + j) : 1u;
            const int exponent = static_cast<int>(min(max(a, 1u), 254u)) - 155, half = exponent / 2;
            scale[0][j] = __uint_as_float(static_cast<uint32_t>(127 + half) << 23);
            // a row with an infinity or a NaN is NaN
            scale[1][j] = __uint_as_float(a == kNonFinite ? 0x7fc00000u : static_cast<uint32_t>(127 + exponent - half) << 23);
        }
        complete = warp_wait(acc_full, 0, abort_flag, p.status_word, kErrStreamAccFull);
        if (complete) {
            tc_fence_after();
            uint32_t v[kTerms][4];
#pragma unroll
            for (uint32_t term = 0; term < kTerms; ++term) load_columns(tmem_base + 8 * term + token0 + ((quadrant * 32) << 16), v[term]);
            tc_wait_ld();
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                // term t carries the factor 8^t relative to term 0
                float sum = 0.0f, factor = 1.0f;
#pragma unroll
                for (uint32_t term = 0; term < kTerms; ++term) {
                    sum = fmaf(__uint_as_float(v[term][j]), factor, sum);
                    factor *= 8.0f;
                }
                y[j] = sum * scale[0][j] * scale[1][j];
            }
        }
    }
    if (p.parts > 1) {
        // every (quarter of the rows, half of the token rows) is finished by one CTA of the cluster, adding in CTA order
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");   // second half: the other CTAs run
        if (epilogue) {
            const uint32_t owner = task % p.parts;
            uint32_t to;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_u32(exchange + (task / p.parts * p.parts + part) * 32 + lane)), "r"(owner));
            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(y[0]), "f"(y[1]), "f"(y[2]), "f"(y[3]) : "memory");
        }
        asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
        if (epilogue && task % p.parts == part) {
            y[0] = y[1] = y[2] = y[3] = 0.0f;
            for (uint32_t from = 0; from < p.parts; ++from) {
                const float4 sums = exchange[(task / p.parts * p.parts + from) * 32 + lane];
                y[0] += sums.x; y[1] += sums.y; y[2] += sums.z; y[3] += sums.w;
            }
        }
    }
    if (complete && (p.parts == 1 || task % p.parts == part)) store_rows(p, tile * kTileM + quadrant * 32, token0, lane, y);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kStreamTmemColumns) : "memory");
    }
}

}  // namespace

// Of the numbers up to the largest portable cluster the one with the least waves of clusters times k blocks of a part, with six k
// blocks' worth of start and end each.
uint32_t split_linear_parts(uint32_t tiles, uint32_t k_blocks, const uint32_t (&clusters)[kSplitMaxParts + 1]) {
    uint32_t best = 1, least = ~0u;
    for (uint32_t parts = 1; parts <= kSplitMaxParts && parts <= k_blocks; ++parts) {
        const uint32_t cost = (tiles + clusters[parts] - 1) / clusters[parts] * ((k_blocks + parts - 1) / parts + 6);
        if (cost < least) {
            least = cost;
            best = parts;
        }
    }
    return best;
}

// Whether the stream kernel forms the digits itself, `chunks` of them per CTA. From six token rows on two of a CTA's eight warps share every quarter of the
// SM and a chunk's digits take 0.94 us, its weights 0.82: what the launch ahead costs is lost again over some ten chunks. us at 6 and 8
// token rows, own digits / launch ahead: 17408 x 5120 (10 chunks) 14.3 / 14.1, 14.6 / 14.8; 10240 x 8192 (11) 15.6 / 14.7, 15.8 / 15.4; 17408 x 6144 (12) 16.9 / 15.9,
// 17.2 / 16.6; 10240 x 10240 (14) 18.3 / 17.0, 18.6 / 17.5; 34816 x 5120 (20) 23.0 / 20.9, 23.3 / 21.1; at five 20.7 / 21.1, 10240 x 17408 (23) 24.8 / 24.7. A long k next to
// the rows gives the launch ahead more to do, which the rule leaves out: 5120 x 17408 (12) 16.5 / 16.7, 16.8 / 17.9.
static bool split_linear_own_digits(uint32_t tokens, uint32_t chunks) { return tokens <= 5 || chunks <= 10; }

augur_cuda_result_v1 launch_split_linear(augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_plan_v1* plan,
                                         const augur_cuda_nvfp4_sm100_gemv_args_v1* a, uint32_t physical_rows, uint8_t* split) {
    CUtensorMap map_weight;
    if (!make_code_map(&map_weight, a->weight, physical_rows, a->cols)) return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE);
    StreamParams p{};
    p.weight_sf = reinterpret_cast<const uint8_t*>(a->weight) + tcgen05_codes_bytes(physical_rows, a->cols);
    p.x = reinterpret_cast<const uint16_t*>(a->input_bf16);
    p.out = reinterpret_cast<void*>(a->output);
    p.status_word = plan->status_word;
    p.out_rows = a->rows; p.cols = a->cols; p.tokens = a->tokens; p.epilogue = a->epilogue;
    p.global_a = a->global_scale; p.global_b = a->global_scale_b;
    const uint32_t tiles = physical_rows / kTileM, k_blocks = (a->cols + kStageK - 1) / kStageK;
    uint32_t clusters[kSplitMaxParts + 1] = {};
    for (uint32_t parts = 1; parts <= kSplitMaxParts; ++parts) clusters[parts] = two_cta_clusters(plan->ordinal, parts);
    p.parts = split_linear_parts(tiles, k_blocks, clusters);
    const bool own_digits = split_linear_own_digits(a->tokens, (k_blocks + p.parts - 1) / p.parts);
    cudaLaunchAttribute attributes[2]{};
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.stream = s->stream;
    config.attrs = attributes;
    config.numAttrs = 1;
    if (!own_digits) {
        uint32_t* anchors = reinterpret_cast<uint32_t*>(plan->scratch + plan->scratch_bytes + kPlanTrailerBytes - kPlanAnchorBytes);
        p.split = split;
        p.anchors = anchors;
        config.gridDim = dim3((a->cols / 16 + kSliceGroups - 1) / kSliceGroups, a->tokens);
        config.blockDim = dim3(kSplitThreads);
        cudaLaunchKernelEx(&config, split_rows_kernel, p.x, split, anchors, a->cols);
        count_launch();
        const augur_cuda_result_v1 result = submitted();
        if (result.status != AUGUR_CUDA_STATUS_OK) return result;
    }
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = p.parts;
    attributes[1].val.clusterDim.y = 1;
    attributes[1].val.clusterDim.z = 1;
    config.numAttrs = p.parts > 1 ? 2 : 1;
    config.gridDim = dim3(tiles * p.parts);
    config.blockDim = dim3(kStreamThreads);
    config.dynamicSmemBytes = kStreamSmem;
    cudaLaunchKernelEx(&config, own_digits ? split_stream_kernel<true> : split_stream_kernel<false>, map_weight, p);
    count_launch();
    return submitted();
}

cudaError_t gemv_split_configure_device() {
    const cudaError_t e = cudaFuncSetAttribute(split_stream_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(split_stream_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem);
}

}  // namespace augur_sm100
