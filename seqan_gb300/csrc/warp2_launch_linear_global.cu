// Packed 16-bit warp kernel instances: linear gaps, global alignments.
#include "warp2_launch.cuh"

namespace gba {
Warp2Fn warp2_fn_linear_global(int mat, bool trace) { return warp2_launch::pick<false, false>(mat, trace); }
}  // namespace gba
