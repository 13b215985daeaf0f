// BF16 vocabulary head for 1..8 token rows on sm_100a: logits[token][row] = sum_k w[row][k] * x[token][k] with
// BF16 weights read in place, F32 activations and F32 results.
//
// What it replaces: the register-blocked FP32 kernel of the reference
// (crates/augur-cuda-sys/native/augur_dflash_llama_bf16_head.cuh:24-72, f32_rw4: BF16 widened exactly to F32,
// exact F32 products, F32 accumulation). The head is one stream over the weights (2.5 GB at 248320 x 5120), and whatever the
// SMs do beside it costs twice: in issue slots and in power, because at this rate the GPU runs into its power limit within
// a tenth of a second. So no thread touches a weight: TMA brings tiles of up to 128 rows x 64 k into a ring in
// shared memory and tcgen05.mma kind::f16 reads them there. (With mma.sync on fragments that every lane loaded for itself, and
// the activations split by every warp for its own rows, the SM clock fell to 1.58 GHz and a pass took 510 to 540 us.)
//
//   activations  F32, split into three BF16 terms x = hi + mid + lo (8 + 8 + 8 significand bits: exact), which sit side by side on
//                the MMA n dimension (column = term * 8 + token): four warps per CTA split the 64 k of every ring stage
//                once for all its rows. Every product is exact, as in the reference; only the order of the additions differs.
//   sums         The tensor core adds into its accumulator without rounding to nearest, so the sum of a 64-k block is formed in
//                an accumulator of its own (four MMAs deep, one column per term) and added to the running sums, in registers of
//                the epilogue warps, with ordinary round-to-nearest additions: the error grows like that of the
//                reference's F32 chain.
//   rows         The tile height is what deals the rows out evenly (120 of 128 at 248320 rows on 148 SMs: 14 tiles for every CTA);
//                tiles go round the CTAs, so that all of them read one neighbourhood of the weights at a time.
//
// Every wait is bounded; a wait that runs out raises a CTA-wide abort flag, all roles fall through to the common exit, and
// the tiles that were not finished are stored as NaN.
#include "nvfp4_gemm.cuh"
#include "nvfp4_internal.h"

namespace augur_sm100 {
namespace {
using namespace tc;

static_assert(sizeof(augur_cuda_nvfp4_sm100_bf16_head_args_v1) == 64, "bf16 head ABI");

constexpr uint32_t kHeadThreads = 32 * 12;                   // warp 0 TMA, 1 MMA, 4..7 split, 8..11 epilogue (2 and 3 have no part)
constexpr uint32_t kHeadTerms = 3;
constexpr uint32_t kHeadN = 32;                              // MMA n: 24 columns, rounded up to a multiple of 16
constexpr uint32_t kHeadTile = kTileM * 128;                 // 16 KB: 128 rows x 64 k of BF16
constexpr uint32_t kHeadStage = kHeadTile + kHeadN * 128;    // and 4 KB of split activations
constexpr uint32_t kHeadStages = 11;
constexpr uint32_t kHeadAccs = 8;                            // accumulators of 32 columns
constexpr uint32_t kHeadState = 512;                         // barriers, tensor-memory base, abort flag, a counter per warp
constexpr uint32_t kHeadSmem = kHeadStages * kHeadStage + kHeadState + 1024 /*alignment*/;
constexpr uint32_t kHeadAhead = 4;                           // stages of activations that a split thread has in flight
constexpr uint32_t kHeadMaxRowBytes = 200 * 1024 / 8 - 64;   // of a token row of activations
static_assert(kHeadSmem <= 227 * 1024, "shared memory of a CTA");
static_assert((2 * kHeadStages + 2 * kHeadAccs) * 8 + 8 + kHeadThreads / 32 * 4 <= kHeadState, "the small state fits");

// A bounded wait of a whole warp (the entry has no plan to report through: tiles that were given up on are NaN).
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag) {
    return warp_look_wait(bar, parity, abort_flag, nullptr, 0);
}

// Two F32 values -> their three BF16 terms, packed (low half = first value). x = hi + mid + lo exactly: each
// subtraction is exact, and after two of them at most 8 significand bits are left.
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(x1), "f"(x0));
    const float r0 = x0 - __uint_as_float(hi << 16), r1 = x1 - __uint_as_float(hi & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(mid) : "f"(r1), "f"(r0));
    const float s0 = r0 - __uint_as_float(mid << 16), s1 = r1 - __uint_as_float(mid & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(s1), "f"(s0));
}

__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void load_columns8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}

__global__ void __launch_bounds__(kHeadThreads, 1)
bf16_head_kernel(const __grid_constant__ CUtensorMap map_weight, const float* __restrict__ x, float* __restrict__ out, uint32_t rows,
                 uint32_t cols, uint32_t tokens, uint32_t tile_rows) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kHeadStages * kHeadStage);
    const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + kHeadStages);
    const uint32_t bar_acc_full = smem_u32(bars + 2 * kHeadStages), bar_acc_empty = smem_u32(bars + 2 * kHeadStages + kHeadAccs);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kHeadStages + 2 * kHeadAccs);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kHeadStages; ++s) {
            mbar_init(bar_full + 8 * s, 1 + 4);   // the TMA's bytes and the four split warps
            mbar_init(bar_empty + 8 * s, 1);
        }
        for (uint32_t b = 0; b < kHeadAccs; ++b) {
            mbar_init(bar_acc_full + 8 * b, 1);
            mbar_init(bar_acc_empty + 8 * b, 4);
        }
        *abort_flag = 0;
        for (uint32_t w = 0; w < kHeadThreads / 32; ++w) abort_flag[1 + w] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kHeadAccs * kHeadN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Everything above runs while the launch before this one drains. From here on its results are needed (the weights are any
    // BF16 matrix, one that it writes among them), and its time does not count against the bound of the waits below.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tiles = (rows + tile_rows - 1) / tile_rows, blocks = cols / 64;
    const uint32_t mine = (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x, total = mine * blocks;   // 64-k stages of this CTA

    if (warp == 0) {
        // ---------------- weights ----------------
        uint32_t stage = 0, phase = 1, block = 0, row = blockIdx.x * tile_rows;
        for (uint32_t s = 0; s < total; ++s) {
            if (!wait(bar_empty + 8 * stage, phase, abort_flag)) break;
            if (elect_one()) {
                const uint32_t full = bar_full + 8 * stage;
                mbar_expect_tx(full, tile_rows * 128);
                tma_load_2d(smem_u32(smem + stage * kHeadStage), &map_weight, block * 128, row, full);
            }
            __syncwarp();
            if (++stage == kHeadStages) { stage = 0; phase ^= 1; }
            if (++block == blocks) { block = 0; row += gridDim.x * tile_rows; }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // F32 accumulator, both operands BF16 and K-major
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kHeadN >> 3) << 17) | ((kTileM >> 4) << 24);
        const uint64_t w_desc0 = operand_desc(smem_u32(smem)), x_desc0 = operand_desc(smem_u32(smem) + kHeadTile);
        uint32_t stage = 0, phase = 0, buffer = 0, acc_phase = 1;
        for (uint32_t s = 0; s < total; ++s) {
            if (!wait(bar_acc_empty + 8 * buffer, acc_phase, abort_flag) || !wait(bar_full + 8 * stage, phase, abort_flag)) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t w_desc = w_desc0 + stage * (kHeadStage >> 4), x_desc = x_desc0 + stage * (kHeadStage >> 4);
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) mma_bf16(tmem_base + buffer * kHeadN, w_desc + 2 * k, x_desc + 2 * k, idesc, k);   // 16 k = 32 bytes
                tc_commit(bar_empty + 8 * stage);
                tc_commit(bar_acc_full + 8 * buffer);
            }
            __syncwarp();
            if (++stage == kHeadStages) { stage = 0; phase ^= 1; }
            if (++buffer == kHeadAccs) { buffer = 0; acc_phase ^= 1; }
        }
    } else if (warp >= 4 && warp < 8) {
        // ---------------- split: thread = (token, four neighbouring k) of every stage ----------------
        // Row term * 8 + token of the operand tile, in its 128-byte swizzle. Columns of tokens that do not exist are never stored,
        // so neither are their rows here.
        const uint32_t thread = threadIdx.x - 128, token = thread >> 4, piece = thread & 15;
        const bool live = token < tokens;
        const float4* row = reinterpret_cast<const float4*>(x + static_cast<uint64_t>(live ? token : 0) * cols) + piece;
        uint8_t* place = smem + kHeadTile + token * 128 + (((piece >> 1) ^ token) << 4) + (piece & 1) * 8;
        float4 ahead[kHeadAhead];
        uint32_t fetch = 0;   // block of the next load (the row is read again for every tile)
#pragma unroll
        for (uint32_t a = 0; a < kHeadAhead; ++a) {
            ahead[a] = __ldcg(row + fetch * 16);
            if (++fetch == blocks) fetch = 0;
        }
        uint32_t stage = 0, phase = 1;
        bool alive = true;
        for (uint32_t s0 = 0; alive && s0 < total; s0 += kHeadAhead) {
#pragma unroll
            for (uint32_t a = 0; a < kHeadAhead; ++a) {
                if (s0 + a >= total) break;
                uint32_t hi[2], mid[2], lo[2];
                split3(ahead[a].x, ahead[a].y, hi[0], mid[0], lo[0]);
                split3(ahead[a].z, ahead[a].w, hi[1], mid[1], lo[1]);
                ahead[a] = __ldcg(row + fetch * 16);
                if (++fetch == blocks) fetch = 0;
                if (!wait(bar_empty + 8 * stage, phase, abort_flag)) {
                    alive = false;
                    break;
                }
                if (live) {
                    uint8_t* to = place + stage * kHeadStage;
                    *reinterpret_cast<uint2*>(to) = make_uint2(hi[0], hi[1]);
                    *reinterpret_cast<uint2*>(to + 1024) = make_uint2(mid[0], mid[1]);
                    *reinterpret_cast<uint2*>(to + 2048) = make_uint2(lo[0], lo[1]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads them through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_full + 8 * stage);
                if (++stage == kHeadStages) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp >= 8) {
        // ---------------- epilogue: lane = weight row, eight token rows x three terms ----------------
        const uint32_t quadrant = warp & 3;
        const uint32_t taddr = tmem_base + ((quadrant * 32) << 16);
        uint32_t buffer = 0, phase = 0;
        for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            float sum[kHeadTerms][8];
#pragma unroll
            for (uint32_t t = 0; t < kHeadTerms; ++t) {
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) sum[t][i] = 0.0f;
            }
            for (uint32_t block = 0; block < blocks; ++block) {
                if (!wait(bar_acc_full + 8 * buffer, phase, abort_flag)) {
                    sum[0][0] = __uint_as_float(0x7fc00000u);
                    break;
                }
                tc_fence_after();
                uint32_t v[kHeadTerms][8];
#pragma unroll
                for (uint32_t t = 0; t < kHeadTerms; ++t) load_columns8(taddr + buffer * kHeadN + 8 * t, v[t]);
                tc_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_acc_empty + 8 * buffer);
                if (++buffer == kHeadAccs) { buffer = 0; phase ^= 1; }
#pragma unroll
                for (uint32_t t = 0; t < kHeadTerms; ++t) {
#pragma unroll
                    for (uint32_t i = 0; i < 8; ++i) sum[t][i] += __uint_as_float(v[t][i]);
                }
            }
            const bool failed = *abort_flag != 0;
            const uint32_t local = quadrant * 32 + lane, row = tile * tile_rows + local;
            if (local < tile_rows && row < rows) {
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    if (i < tokens) out[static_cast<uint64_t>(i) * rows + row] = failed ? __uint_as_float(0x7fc00000u) : (sum[2][i] + sum[1][i]) + sum[0][i];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kHeadAccs * kHeadN) : "memory");
    }
}

bool check_head(int32_t d, augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_bf16_head_args_v1* a, bool full, uint32_t* tokens,
                augur_cuda_result_v1* failure) {
    *failure = invalid();
    if (!header_ok(d, s, a)) {
        if (a && s && d >= 0 && s->ordinal == d && a->abi_version != AUGUR_CUDA_ABI_VERSION_V1) {
            *failure = make_result(AUGUR_CUDA_STATUS_ABI_VERSION_MISMATCH);
        }
        return false;
    }
    if (!a->rows || !a->cols || a->rows % 16 != 0 || a->cols % 64 != 0 || a->rows > (1u << 30) || a->cols > (1u << 20)) return false;
    if (a->weight_len_bytes != static_cast<uint64_t>(a->rows) * a->cols * 2) return false;
    const uint64_t row_bytes = static_cast<uint64_t>(a->cols) * 4;
    if (a->input_len_bytes % row_bytes != 0) return false;
    const uint64_t count = a->input_len_bytes / row_bytes;
    if (count < 1 || count > AUGUR_NVFP4_SM100_MAX_SMALL_TOKENS) return false;
    *tokens = static_cast<uint32_t>(count);
    if (a->output_len_bytes != count * a->rows * 4) return false;
    if (a->cols * 4 > kHeadMaxRowBytes) return false;   // the widths that this entry has always taken
    // TMA and 16-byte vector loads (the reference's rw4 entry asks the same alignment)
    const Range r[3] = {{a->weight, a->weight_len_bytes, 16}, {a->input, a->input_len_bytes, 16}, {a->output, a->output_len_bytes, 4}};
    if (!all_disjoint(r, 3)) return false;
    return !full || inspect_device_ranges(d, r, 3, failure);
}

}  // namespace
}  // namespace augur_sm100

using namespace augur_sm100;

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_bf16_head_preflight_v1(
    int32_t d, augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_bf16_head_args_v1* a) {
    augur_cuda_result_v1 failure;
    uint32_t tokens = 0;
    if (!check_head(d, s, a, true, &tokens, &failure)) return failure;
    // a bind-time call: the kernel's shared-memory limit for this width
    const cudaError_t e = cudaFuncSetAttribute(bf16_head_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kHeadSmem);
    return e == cudaSuccess ? ok() : make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE, e);
}

extern "C" augur_cuda_result_v1 AUGUR_CUDA_CALL augur_cuda_nvfp4_sm100_bf16_head_prevalidated_submit_v1(
    int32_t d, augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_bf16_head_args_v1* a) {
    augur_cuda_result_v1 failure;
    uint32_t tokens = 0;
    if (!check_head(d, s, a, false, &tokens, &failure)) return failure;
    if (consume_injected_fault()) return make_result(AUGUR_CUDA_STATUS_DIAGNOSTIC_FAULT_INJECTED);
    cudaError_t e = cudaSetDevice(d);
    if (e != cudaSuccess) return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE, e);
    static int sm_count[64];               // per device, looked up once (a host-side attribute query, no allocation)
    if (d >= 64) return invalid();
    if (!sm_count[d]) {
        int sms = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(bf16_head_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kHeadSmem);
        if (e != cudaSuccess) return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE, e);
        sm_count[d] = sms;
    }
    // tiles of equal height, as few rounds of the SMs as 128-row tiles allow
    const uint32_t sms = static_cast<uint32_t>(sm_count[d]), rounds = (a->rows + kTileM * sms - 1) / (kTileM * sms);
    const uint32_t tile_rows = ((a->rows + rounds * sms - 1) / (rounds * sms) + 7) / 8 * 8;
    const uint32_t tiles = (a->rows + tile_rows - 1) / tile_rows;
    CUtensorMap map_weight;   // rows of cols * 2 bytes, as a map of packed codes with four times the columns
    if (!make_code_map(&map_weight, a->weight, a->rows, a->cols * 4, tile_rows)) return make_result(AUGUR_CUDA_STATUS_RUNTIME_FAILURE);
    launch_dependent(s->stream, bf16_head_kernel, tiles < sms ? tiles : sms, kHeadThreads, kHeadSmem, map_weight,
                     reinterpret_cast<const float*>(a->input), reinterpret_cast<float*>(a->output), a->rows, a->cols, tokens, tile_rows);
    count_launch();
    return submitted();
}
