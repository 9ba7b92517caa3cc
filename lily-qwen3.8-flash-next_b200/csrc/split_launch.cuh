// The row kernel's launches: one translation unit for each size of the argument block includes this and
// instantiates split_launch.
#pragma once

#include "split_kernel.cuh"

namespace lily {

template <typename T, uint32_t MAXR, int BPS, uint32_t HAS>
cudaError_t split_launch_one(const SplitArgs<MAXR> &a, uint32_t rows, size_t smem, int max_smem, uint64_t *attr_mask,
                             cudaStream_t stream) {
    auto kernel = split_rows_kernel<T, MAXR, BPS, HAS>;
    constexpr uint32_t variant = HAS == HAS_ALL ? (BPS == 1 ? 0u : 1u) : HAS == 0u ? 2u : HAS == HAS_SPEC ? 3u : HAS == HAS_WIDE ? 4u
                                 : HAS == HAS_SHARD ? 5u : 6u;
    constexpr uint32_t size = MAXR == INLINE_ROWS ? 0u : MAXR == INLINE_ROWS_MID ? 1u : 2u;
    constexpr uint64_t bit = 1ull << ((variant * 3u + size) * 2u + (sizeof(T) == 4 ? 0u : 1u));
    if (!(*attr_mask & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
        if (e != cudaSuccess) {
            return e;
        }
        *attr_mask |= bit;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1u << a.log_blocks, rows, 1);
    cfg.blockDim = dim3(NT, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1u << a.log_blocks;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.log_blocks ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

// One block per SM: the variants beside the general one are compiled where calls of that kind are
// common (proposals have at most 8 rows; shards' logits are a head's, f32; an argmax brings no parameters, so its
// launches all have the smallest argument block).
template <typename T, uint32_t MAXR>
cudaError_t split_launch_sole(const SplitArgs<MAXR> &a, uint32_t has, uint32_t rows, size_t smem, int max_smem,
                              uint64_t *attr_mask, cudaStream_t stream) {
    if (has == 0u) {
        return split_launch_one<T, MAXR, 1, 0u>(a, rows, smem, max_smem, attr_mask, stream);
    }
    if constexpr (MAXR == INLINE_ROWS) {
        if (has == HAS_SPEC) {
            return split_launch_one<T, MAXR, 1, HAS_SPEC>(a, rows, smem, max_smem, attr_mask, stream);
        }
        if (has == HAS_ARGMAX) {
            return split_launch_one<T, MAXR, 1, HAS_ARGMAX>(a, rows, smem, max_smem, attr_mask, stream);
        }
    }
    if constexpr (MAXR != INLINE_ROWS_MAX) {
        if (has == HAS_WIDE) {
            return split_launch_one<T, MAXR, 1, HAS_WIDE>(a, rows, smem, max_smem, attr_mask, stream);
        }
        if constexpr (sizeof(T) == 4) {
            if (has == HAS_SHARD) {
                return split_launch_one<T, MAXR, 1, HAS_SHARD>(a, rows, smem, max_smem, attr_mask, stream);
            }
        }
    }
    return split_launch_one<T, MAXR, 1, HAS_ALL>(a, rows, smem, max_smem, attr_mask, stream);
}

template <uint32_t MAXR>
cudaError_t split_launch(const SplitArgs<MAXR> &a, uint32_t has, uint32_t rows, uint32_t dtype, size_t smem, int max_smem,
                         uint64_t *attr_mask, cudaStream_t stream) {
    if constexpr (MAXR == INLINE_ROWS) {
        if (a.two_per_sm) {
            return dtype == LILY_F32
                       ? split_launch_one<float, MAXR, 2, HAS_ALL>(a, rows, smem, max_smem, attr_mask, stream)
                       : split_launch_one<__nv_bfloat16, MAXR, 2, HAS_ALL>(a, rows, smem, max_smem, attr_mask, stream);
        }
    }
    return dtype == LILY_F32 ? split_launch_sole<float>(a, has, rows, smem, max_smem, attr_mask, stream)
                             : split_launch_sole<__nv_bfloat16>(a, has, rows, smem, max_smem, attr_mask, stream);
}

}  // namespace lily
