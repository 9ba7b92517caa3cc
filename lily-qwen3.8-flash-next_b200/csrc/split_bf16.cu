// The row kernel for bf16 logits and up to 8 rows' parameters.
#include "split_launch.cuh"

namespace lily {

LILY_SPLIT_LAUNCH_FOR(, __nv_bfloat16, INLINE_ROWS);

}  // namespace lily
