// Packed 16-bit warp kernel instances: affine gaps, local alignments.
#include "warp2_launch.cuh"

namespace gba {
Warp2Fn warp2_fn_affine_local(int mat, bool trace) { return warp2_launch::pick<true, true>(mat, trace); }
}  // namespace gba
