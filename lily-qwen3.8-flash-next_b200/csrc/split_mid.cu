// The row kernel for f32 logits and up to 64 rows' parameters.
#include "split_launch.cuh"

namespace lily {

LILY_SPLIT_LAUNCH_FOR(, float, INLINE_ROWS_MID);

}  // namespace lily
