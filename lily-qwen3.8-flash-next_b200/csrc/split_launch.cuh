// The row kernel's launches. Translation units for the sizes of the argument block and the types include this and
// instantiate split_launch_for.
#pragma once

#include <type_traits>

#include "split_kernel.cuh"

namespace lily {

template <typename T, uint32_t MAXR, int BPS, uint32_t HAS>
cudaError_t split_launch_one(const SplitArgs<MAXR> &a, uint32_t rows, size_t smem, int max_smem, uint64_t *attr_mask,
                             cudaStream_t stream) {
    auto kernel = split_rows_kernel<T, MAXR, BPS, HAS>;
    constexpr uint32_t variant = HAS == HAS_ALL ? (BPS == 1 ? 0u : 1u) : HAS == 0u ? 2u : HAS == HAS_SPEC ? 3u : HAS == HAS_WIDE ? 4u
                                 : HAS == HAS_SHARD ? 5u : HAS == HAS_ARGMAX ? 6u : HAS == HAS_UNKNOWN ? (BPS == 1 ? 7u : 8u) : 9u;
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

// One block per SM. The variants beside the general one are compiled where calls of that kind are common:
// proposals have at most 8 rows; shards' logits are a head's, f32; where no parameters travel in the arguments, the
// smallest argument block is used for any number of rows.
template <typename T, uint32_t MAXR>
cudaError_t split_launch_sole(const SplitArgs<MAXR> &a, uint32_t has, uint32_t rows, size_t smem, int max_smem,
                              uint64_t *attr_mask, cudaStream_t stream) {
    auto launch = [&](auto set) {
        return split_launch_one<T, MAXR, 1, decltype(set)::value>(a, rows, smem, max_smem, attr_mask, stream);
    };
    if constexpr (MAXR == INLINE_ROWS) {
        if (has == HAS_ARGMAX) {
            return launch(std::integral_constant<uint32_t, HAS_ARGMAX>());
        }
        if (has == HAS_UNKNOWN) {
            return launch(std::integral_constant<uint32_t, HAS_UNKNOWN>());
        }
    }
    if (a.inline_params && (a.log_blocks != 0u || !variant_many(0u, MAXR))) {
        if (has == 0u) {
            return launch(std::integral_constant<uint32_t, 0u>());
        }
        if constexpr (MAXR == INLINE_ROWS) {
            if (has == HAS_SPEC) {
                return launch(std::integral_constant<uint32_t, HAS_SPEC>());
            }
        }
        if constexpr (MAXR != INLINE_ROWS_MAX) {
            if (has == HAS_WIDE) {
                return launch(std::integral_constant<uint32_t, HAS_WIDE>());
            }
            if ((has & ~(uint32_t)(HAS_WIDE | HAS_LISTS)) == 0u) {
                return launch(std::integral_constant<uint32_t, HAS_WIDE | HAS_LISTS>());
            }
            if constexpr (sizeof(T) == 4) {
                if (has == HAS_SHARD) {
                    return launch(std::integral_constant<uint32_t, HAS_SHARD>());
                }
            }
        }
    }
    return launch(std::integral_constant<uint32_t, HAS_ALL>());
}

// Everything for logits of one type.
template <typename T, uint32_t MAXR>
cudaError_t split_launch_for(const SplitArgs<MAXR> &a, uint32_t has, uint32_t rows, size_t smem, int max_smem,
                             uint64_t *attr_mask, cudaStream_t stream) {
    if constexpr (MAXR == INLINE_ROWS) {
        if (a.two_per_sm) {
            return has == HAS_UNKNOWN ? split_launch_one<T, MAXR, 2, HAS_UNKNOWN>(a, rows, smem, max_smem, attr_mask, stream)
                                      : split_launch_one<T, MAXR, 2, HAS_ALL>(a, rows, smem, max_smem, attr_mask, stream);
        }
    }
    return split_launch_sole<T>(a, has, rows, smem, max_smem, attr_mask, stream);
}

#define LILY_SPLIT_LAUNCH_FOR(T, MAXR)                                                                            \
    template cudaError_t split_launch_for<T, MAXR>(const SplitArgs<MAXR> &, uint32_t, uint32_t, size_t, int, uint64_t *, \
                                                   cudaStream_t)

}  // namespace lily
