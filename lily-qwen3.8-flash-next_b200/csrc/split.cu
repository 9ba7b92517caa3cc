// The row kernel's translation unit: its instantiations and their launch.
#include "split_kernel.cuh"

namespace lily {

namespace {

template <typename T, uint32_t MAXR>
cudaError_t launch_one(const SplitArgs<MAXR> &a, uint32_t rows, size_t smem, int max_smem, uint32_t *attr_mask,
                       cudaStream_t stream) {
    auto kernel = split_rows_kernel<T, MAXR, 1>;
    const uint32_t bit = 1u << ((sizeof(T) == 4 ? 16 : 17) + (MAXR == INLINE_ROWS ? 0 : 2));
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

}  // namespace

template <uint32_t MAXR>
cudaError_t split_launch(const SplitArgs<MAXR> &a, uint32_t rows, uint32_t dtype, size_t smem, int max_smem,
                         uint32_t *attr_mask, cudaStream_t stream) {
    return dtype == LILY_F32 ? launch_one<float, MAXR>(a, rows, smem, max_smem, attr_mask, stream)
                             : launch_one<__nv_bfloat16, MAXR>(a, rows, smem, max_smem, attr_mask, stream);
}

template cudaError_t split_launch<INLINE_ROWS>(const SplitArgs<INLINE_ROWS> &, uint32_t, uint32_t, size_t, int, uint32_t *,
                                               cudaStream_t);
template cudaError_t split_launch<INLINE_ROWS_MAX>(const SplitArgs<INLINE_ROWS_MAX> &, uint32_t, uint32_t, size_t, int,
                                                   uint32_t *, cudaStream_t);

}  // namespace lily
