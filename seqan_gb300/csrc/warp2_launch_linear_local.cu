// Packed 16-bit warp kernel instances: linear gaps, local alignments.
#include "warp2_launch.cuh"

namespace gba {
Warp2Fn warp2_fn_linear_local(int mat, bool trace) { return warp2_launch::pick<false, true>(mat, trace); }
}  // namespace gba
