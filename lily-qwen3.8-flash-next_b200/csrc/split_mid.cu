// The row kernel for up to 64 rows' parameters.
#include "split_launch.cuh"

namespace lily {

template cudaError_t split_launch<INLINE_ROWS_MID>(const SplitArgs<INLINE_ROWS_MID> &, uint32_t, uint32_t, uint32_t, size_t,
                                                   int, uint64_t *, cudaStream_t);

}  // namespace lily
