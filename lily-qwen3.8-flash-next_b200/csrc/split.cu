// The row kernel for f32 logits and up to 8 rows' parameters, and the merge kernel.
#include <atomic>

#include "merge_kernel.cuh"
#include "split_launch.cuh"

namespace lily {

LILY_SPLIT_LAUNCH_FOR(, float, INLINE_ROWS);
// (In units of their own.)
LILY_SPLIT_LAUNCH_FOR(extern, __nv_bfloat16, INLINE_ROWS);
LILY_SPLIT_LAUNCH_FOR(extern, float, INLINE_ROWS_MID);
LILY_SPLIT_LAUNCH_FOR(extern, __nv_bfloat16, INLINE_ROWS_MID);
LILY_SPLIT_LAUNCH_FOR(extern, float, INLINE_ROWS_MAX);
LILY_SPLIT_LAUNCH_FOR(extern, __nv_bfloat16, INLINE_ROWS_MAX);

template <uint32_t MAXR>
cudaError_t split_launch(const SplitArgs<MAXR> &a, uint32_t has, uint32_t rows, uint32_t dtype, size_t smem,
                         cudaStream_t stream) {
    return dtype == LILY_F32 ? split_launch_for<float>(a, has, rows, smem, stream)
                             : split_launch_for<__nv_bfloat16>(a, has, rows, smem, stream);
}

template cudaError_t split_launch<INLINE_ROWS>(const SplitArgs<INLINE_ROWS> &, uint32_t, uint32_t, uint32_t, size_t,
                                               cudaStream_t);
template cudaError_t split_launch<INLINE_ROWS_MID>(const SplitArgs<INLINE_ROWS_MID> &, uint32_t, uint32_t, uint32_t, size_t,
                                                   cudaStream_t);
template cudaError_t split_launch<INLINE_ROWS_MAX>(const SplitArgs<INLINE_ROWS_MAX> &, uint32_t, uint32_t, uint32_t, size_t,
                                                   cudaStream_t);

cudaError_t split_ready(uint32_t max_rows, uint32_t sms, int max_smem) {
    cudaError_t e = split_ready_for<float, INLINE_ROWS>(max_rows > sms, max_smem);
    auto and_then = [&](bool needed, auto ready) {
        if (e == cudaSuccess && needed) {
            e = ready(max_rows > sms, max_smem);
        }
    };
    and_then(true, split_ready_for<__nv_bfloat16, INLINE_ROWS>);
    and_then(max_rows > INLINE_ROWS, split_ready_for<float, INLINE_ROWS_MID>);
    and_then(max_rows > INLINE_ROWS, split_ready_for<__nv_bfloat16, INLINE_ROWS_MID>);
    and_then(max_rows > INLINE_ROWS_MID, split_ready_for<float, INLINE_ROWS_MAX>);
    and_then(max_rows > INLINE_ROWS_MID, split_ready_for<__nv_bfloat16, INLINE_ROWS_MAX>);
    return e;
}

uint32_t split_rows_at_once(int device, int sm_count, int max_smem, uint32_t log_blocks) {
    if (log_blocks == 0u) {
        return (uint32_t)sm_count;
    }
    // Asked for once per device; 0: not yet, else 1 + the answer.
    constexpr int DEVICES = 64;
    static std::atomic<uint32_t> known[DEVICES][4];
    std::atomic<uint32_t> *at = device >= 0 && device < DEVICES ? &known[device][log_blocks] : nullptr;
    uint32_t n = at ? at->load(std::memory_order_relaxed) : 0u;
    if (n == 0u) {
        auto kernel = split_rows_kernel<float, INLINE_ROWS, 1, HAS_ALL>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1u << log_blocks, 1, 1);
        cfg.blockDim = dim3(NT, 1, 1);
        cfg.dynamicSmemBytes = (size_t)max_smem;  // (one block per SM)
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1u << log_blocks;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 0) {
            clusters = 0;
            cudaGetLastError();
        }
        n = 1u + (uint32_t)clusters;
        if (at) {
            at->store(n, std::memory_order_relaxed);
        }
    }
    return n - 1u;
}

cudaError_t merge_ready() {
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, merge_rows_kernel);
    return e != cudaSuccess ? e
                            : cudaFuncSetAttribute(merge_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)sizeof(SmemFixed));
}

cudaError_t merge_launch(const MergeArgs &a, uint32_t rows, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(rows, 1, 1);
    cfg.blockDim = dim3(NT, 1, 1);
    cfg.dynamicSmemBytes = sizeof(SmemFixed);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, merge_rows_kernel, a);
}

}  // namespace lily
