// warp2_launch.cuh -- the packed 16-bit warp kernel's instances.  They are split over four
// translation units by gap model and mode (warp2_launch_*.cu) so that they compile in parallel.
#pragma once

#include "dp_warp2_kernels.cuh"

#include <cuda_runtime.h>

namespace gba {

using Warp2Fn = void (*)(Warp2Args);   // the kernel itself

Warp2Fn warp2_fn_affine_global(int mat, bool trace);
Warp2Fn warp2_fn_affine_local(int mat, bool trace);
Warp2Fn warp2_fn_linear_global(int mat, bool trace);
Warp2Fn warp2_fn_linear_local(int mat, bool trace);

namespace warp2_launch {

template <bool A, bool L>
Warp2Fn pick(int mat, bool t)
{
    static const Warp2Fn table[6] = {k_dp_warp2<A, L, W2_EQUAL, false>,   k_dp_warp2<A, L, W2_EQUAL, true>,
                                     k_dp_warp2<A, L, W2_PROFILE, false>, k_dp_warp2<A, L, W2_PROFILE, true>,
                                     k_dp_warp2<A, L, W2_TABLE, false>,   k_dp_warp2<A, L, W2_TABLE, true>};
    return table[2 * mat + (t ? 1 : 0)];
}

}  // namespace warp2_launch
}  // namespace gba
