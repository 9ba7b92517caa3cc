// The row kernel for up to 148 rows' parameters.
#include "split_launch.cuh"

namespace lily {

LILY_SPLIT_LAUNCH_FOR(, float, INLINE_ROWS_MAX);
LILY_SPLIT_LAUNCH_FOR(, __nv_bfloat16, INLINE_ROWS_MAX);

}  // namespace lily
