// Packed 16-bit warp kernel instances: affine gaps, global alignments.
#include "warp2_launch.cuh"

namespace gba {
Warp2Fn warp2_fn_affine_global(int mat, bool trace) { return warp2_launch::pick<true, false>(mat, trace); }
}  // namespace gba
