// The row kernel's launches. Translation units for the sizes of the argument block and the types include this and
// instantiate split_launch_for.
#pragma once

#include <type_traits>

#include "split_kernel.cuh"

namespace lily {

// Loads the kernel and raises its shared-memory limit.
template <typename T, uint32_t MAXR, int BPS, uint32_t HAS>
cudaError_t split_ready_one(int max_smem) {
    auto kernel = split_rows_kernel<T, MAXR, BPS, HAS>;
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, kernel);  // (this loads it)
    return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
}

template <typename T, uint32_t MAXR, int BPS, uint32_t HAS>
cudaError_t split_launch_one(const SplitArgs<MAXR> &a, uint32_t rows, size_t smem, cudaStream_t stream) {
    auto kernel = split_rows_kernel<T, MAXR, BPS, HAS>;
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

// The variants there are, the general one last: compiled where calls of that kind are common. Proposals have at most
// 8 rows; shards' logits are a head's, f32; where no parameters travel in the arguments, the smallest argument block is
// used for any number of rows, and it alone for two blocks per SM.
template <typename T, uint32_t MAXR, int BPS>
constexpr bool split_compiled(uint32_t has) {
    return has == HAS_ALL                          ? BPS == 1 || MAXR == INLINE_ROWS
           : has == HAS_UNKNOWN                    ? MAXR == INLINE_ROWS
           : BPS != 1                              ? false
           : has == HAS_ARGMAX || has == HAS_SPEC  ? MAXR == INLINE_ROWS
           : has == HAS_SHARD                      ? MAXR != INLINE_ROWS_MAX && sizeof(T) == 4
           : (has & HAS_WIDE) != 0u                ? MAXR != INLINE_ROWS_MAX
                                                   : true;
}

// f(variant) for each of them until one returns true.
template <typename T, uint32_t MAXR, int BPS, typename F>
void split_variants(F f) {
    auto each = [&](auto... set) {
        auto one = [&](auto v) -> bool {
            if constexpr (split_compiled<T, MAXR, BPS>(decltype(v)::value)) {
                return f(v);
            }
            return false;
        };
        (void)(one(set) || ...);
    };
    each(std::integral_constant<uint32_t, HAS_ARGMAX>(), std::integral_constant<uint32_t, 0u>(),
         std::integral_constant<uint32_t, HAS_SPEC>(), std::integral_constant<uint32_t, HAS_WIDE>(),
         std::integral_constant<uint32_t, HAS_WIDE | HAS_LISTS>(), std::integral_constant<uint32_t, HAS_SHARD>(),
         std::integral_constant<uint32_t, HAS_UNKNOWN>(), std::integral_constant<uint32_t, HAS_ALL>());
}

// Whether a launch whose rows may bring `has` may take the variant.
template <uint32_t MAXR>
bool split_takes(const SplitArgs<MAXR> &a, uint32_t variant, uint32_t has) {
    if (variant == HAS_ALL) {
        return true;
    }
    if ((variant_inline(variant) && !a.inline_params) || (variant_many(variant, MAXR) && a.log_blocks == 0u)) {
        return false;
    }
    // (HAS_UNKNOWN serves whatever it has, with parameters in the arguments or not.)
    return has == variant || ((variant == (HAS_WIDE | HAS_LISTS) || variant == HAS_UNKNOWN) && (has & ~variant) == 0u);
}

// Everything for logits of one type.
template <typename T, uint32_t MAXR, int BPS>
cudaError_t split_launch_blocks(const SplitArgs<MAXR> &a, uint32_t has, uint32_t rows, size_t smem, cudaStream_t stream) {
    cudaError_t e = cudaErrorInvalidValue;
    split_variants<T, MAXR, BPS>([&](auto v) -> bool {
        constexpr uint32_t variant = decltype(v)::value;
        if (!split_takes(a, variant, has)) {
            return false;
        }
        e = split_launch_one<T, MAXR, BPS, variant>(a, rows, smem, stream);
        return true;
    });
    return e;
}

template <typename T, uint32_t MAXR>
cudaError_t split_launch_for(const SplitArgs<MAXR> &a, uint32_t has, uint32_t rows, size_t smem, cudaStream_t stream) {
    if constexpr (MAXR == INLINE_ROWS) {
        if (a.two_per_sm) {
            return split_launch_blocks<T, MAXR, 2>(a, has, rows, smem, stream);
        }
    }
    return split_launch_blocks<T, MAXR, 1>(a, has, rows, smem, stream);
}

template <typename T, uint32_t MAXR>
cudaError_t split_ready_for(bool two_per_sm, int max_smem) {
    cudaError_t e = cudaSuccess;
    split_variants<T, MAXR, 1>([&](auto v) -> bool {
        return (e = split_ready_one<T, MAXR, 1, decltype(v)::value>(max_smem)) != cudaSuccess;
    });
    if (MAXR == INLINE_ROWS && two_per_sm && e == cudaSuccess) {
        split_variants<T, MAXR, 2>([&](auto v) -> bool {
            return (e = split_ready_one<T, MAXR, 2, decltype(v)::value>(max_smem)) != cudaSuccess;
        });
    }
    return e;
}

#define LILY_SPLIT_LAUNCH_FOR(EXTERN, T, MAXR)                                                                          \
    EXTERN template cudaError_t split_launch_for<T, MAXR>(const SplitArgs<MAXR> &, uint32_t, uint32_t, size_t, cudaStream_t); \
    EXTERN template cudaError_t split_ready_for<T, MAXR>(bool, int)

}  // namespace lily
