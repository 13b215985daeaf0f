// Private definitions shared by the translation units of the sm_100a NVFP4 library.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <climits>
#include <cmath>
#include <cstdint>

#include "augur_cuda_nvfp4_sm100.h"

// Same private layout as the reference runtime's handle
// (crates/augur-cuda-sys/native/augur_cuda_internal.h:39-42), so handles made by
// either library are interchangeable. `owned` lives past the shared prefix.
struct augur_cuda_stream_handle {
    int32_t ordinal;
    cudaStream_t stream;
    int32_t owned;
    int32_t plans;   // live plans made on this handle; the handle is not destroyed while any exist
};

struct augur_cuda_nvfp4_sm100_plan_v1 {
    uint32_t magic;
    int32_t ordinal;
    augur_cuda_stream_t owner;
    uint8_t* scratch;          // device
    uint64_t scratch_bytes;
    uint32_t* status_word;     // device, 256 bytes reserved in front of scratch
    uint32_t sm_count;
    // Copied from the owner when the plan is made: destroy and status read-back must not dereference a
    // stream handle that its owner may already have closed. `owner` itself only serves the identity check.
    cudaStream_t owner_stream;
    uint32_t pair_clusters;    // two-CTA clusters of the pair GEMM that can be resident at once on this device
};

namespace augur_sm100 {

constexpr uint32_t kPlanMagic = 0x4e56'4634u;  // "NVF4"
constexpr uint64_t kPlanHeaderBytes = 256;     // status word + padding in front of the scratch
constexpr uint64_t kPlanAnchorBytes = 256;     // the trailer's end: the token rows' anchors of a split (nvfp4_gemv_split.cu)
constexpr uint64_t kPlanTrailerBytes = 16384 + kPlanAnchorBytes;  // behind the scratch, outside what `scratch_bytes` counts: words that only
                                               // the tensor-memory small-token kernels write (one per CTA, four sets; the anchors)

struct Range {
    uint64_t address, bytes, alignment;
};

inline bool valid(Range r) {
    return r.address && r.bytes && r.alignment && r.address % r.alignment == 0 &&
           r.bytes <= UINT64_MAX - r.address;
}
inline bool disjoint(Range a, Range b) {
    return valid(a) && valid(b) &&
           (a.address + a.bytes <= b.address || b.address + b.bytes <= a.address);
}
inline bool all_disjoint(const Range* r, size_t count) {
    for (size_t i = 0; i < count; ++i) {
        if (!valid(r[i])) return false;
        for (size_t j = i + 1; j < count; ++j) {
            if (!disjoint(r[i], r[j])) return false;
        }
    }
    return true;
}
// Conservative scalar range of the reference's checked loader
// (crates/augur-cuda-sys/native/augur_qwen35_nvfp4_qpn_sm70.cu:27-28).
inline bool scale_ok(float s) { return std::isfinite(s) && s >= 0x1p-32f && s <= 24.0f; }

template <class T>
inline bool header_ok(int32_t ordinal, augur_cuda_stream_t stream, const T* args) {
    return ordinal >= 0 && stream && stream->ordinal == ordinal && args &&
           args->abi_version == AUGUR_CUDA_ABI_VERSION_V1 && args->struct_size == sizeof(T);
}

inline augur_cuda_result_v1 make_result(augur_cuda_status_t status, cudaError_t raw = cudaSuccess) {
    return {status, static_cast<int32_t>(raw)};
}
inline augur_cuda_result_v1 ok() { return make_result(AUGUR_CUDA_STATUS_OK); }
inline augur_cuda_result_v1 invalid() { return make_result(AUGUR_CUDA_STATUS_INVALID_ARGUMENT); }

// Driver-side inspection used by every preflight: the range must be device memory of
// `ordinal` and lie inside one allocation. Also gates on compute capability 10.x.
bool inspect_device_ranges(int32_t ordinal, const Range* ranges, size_t count,
                           augur_cuda_result_v1* failure);
// Plan scratch layout: two arrival-counter regions (one per member of a two-launch program)
// at fixed offsets, then partial-sum slots. Counters must read zero when a launch starts and
// every launch leaves them at zero; keeping them apart from the slots means no launch of any
// shape can ever leave slot data where another launch expects counters.
constexpr uint32_t kMaxGroups = 16384;
constexpr uint64_t kCounterRegionBytes = static_cast<uint64_t>(kMaxGroups) * 4;
constexpr uint64_t kCounterBytes = 2 * kCounterRegionBytes;

bool plan_ok(const augur_cuda_nvfp4_sm100_plan_v1* plan, int32_t ordinal, augur_cuda_stream_t stream);
Range plan_scratch_range(const augur_cuda_nvfp4_sm100_plan_v1* plan);

// Diagnostics shared by all entry points.
bool consume_injected_fault();
void count_launch(uint64_t launches = 1);
void count_allocation();
void count_free();
augur_cuda_result_v1 submitted();  // maps cudaGetLastError to SUBMISSION_FAILURE

// Launches with programmatic stream serialisation: the grid may become resident while its predecessor drains, and
// waits for it in-kernel (griddepcontrol.wait).
template <class... Parameters, class... Arguments>
void launch_dependent(cudaStream_t stream, void (*kernel)(Parameters...), uint32_t grid, uint32_t threads, uint32_t smem_bytes,
                      const Arguments&... arguments) {
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = 1;
    config.gridDim = dim3(grid);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem_bytes;
    cudaLaunchKernelEx(&config, kernel, static_cast<Parameters>(arguments)...);
}

// The same for a kernel of small CTAs that the work behind it waits for: while they all fit the device at once, `ctas` are
// rounded up to whole clusters of eight that are to be spread over the SMs (the CTAs added find nothing to do). On its own a small
// CTA goes where the most room is, so while the launch before still fills most SMs, they pile up, ten and more, on the few that
// it does not. Larger grids even that out (quantiser, three terms: 640 CTAs are better spread, 1943 and more are not: 8.7 -> 9.1 us).
constexpr uint32_t kSpreadCtas = 8, kSpreadLimit = 1024;
template <class... Parameters, class... Arguments>
void launch_dependent_spread(cudaStream_t stream, void (*kernel)(Parameters...), uint32_t ctas, uint32_t threads, const Arguments&... arguments) {
    if (ctas > kSpreadLimit) {
        launch_dependent(stream, kernel, ctas, threads, 0, arguments...);
        return;
    }
    cudaLaunchAttribute attributes[3]{};
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = kSpreadCtas;
    attributes[1].val.clusterDim.y = 1;
    attributes[1].val.clusterDim.z = 1;
    attributes[2].id = cudaLaunchAttributeClusterSchedulingPolicyPreference;
    attributes[2].val.clusterSchedulingPolicyPreference = cudaClusterSchedulingPolicySpread;
    cudaLaunchConfig_t config{};
    config.stream = stream;
    config.attrs = attributes;
    config.numAttrs = 3;
    config.gridDim = dim3((ctas + kSpreadCtas - 1) / kSpreadCtas * kSpreadCtas);
    config.blockDim = dim3(threads);
    cudaLaunchKernelEx(&config, kernel, static_cast<Parameters>(arguments)...);
}

// One-time per-device kernel attribute setup, called from plan creation (bind time).
cudaError_t gemv_configure_device();
cudaError_t gemm_configure_device();
cudaError_t gemv_tc_configure_device();
cudaError_t gemm_narrow_configure_device();
cudaError_t gemv_split_configure_device();
// Clusters of `parts` CTAs of 384 threads and 112 KB of shared memory (two per SM) that a launch may count on to run at once.
uint32_t two_cta_clusters(int32_t ordinal, uint32_t parts);
// CTAs per 128-row tile of a small-token linear on tensor memory (a cluster) where `clusters[parts]` clusters of `parts` run at once.
constexpr uint32_t kSplitMaxParts = 8;
uint32_t split_linear_parts(uint32_t tiles, uint32_t k_blocks, const uint32_t (&clusters)[kSplitMaxParts + 1]);
// The linear of 1..8 token rows on tensor memory (nvfp4_gemv_split.cu); `split`: split_bytes(cols) of plan scratch, where digits that a launch of
// their own forms pass through.
augur_cuda_result_v1 launch_split_linear(augur_cuda_stream_t s, const augur_cuda_nvfp4_sm100_plan_v1* plan,
                                         const augur_cuda_nvfp4_sm100_gemv_args_v1* a, uint32_t physical_rows, uint8_t* split);
// Two-CTA clusters of the pair GEMM that the device can hold at once (0 if the query fails).
uint32_t gemm_pair_resident_clusters();

}  // namespace augur_sm100
