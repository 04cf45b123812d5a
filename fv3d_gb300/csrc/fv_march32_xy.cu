// fv_march32_xy.cu -- the warp-marched FP32-mixed kernels (fv_march32.cuh) of
// the x-y plane.
#include "fv_march32.cuh"

namespace fv {

MarchKernel march_kernel_xy(bool wact, int kind, bool one) {
  if (one) return wact ? march_kernel_of<PLANE_XY, true, true>(kind) : march_kernel_of<PLANE_XY, false, true>(kind);
  return wact ? march_kernel_of<PLANE_XY, true, false>(kind) : march_kernel_of<PLANE_XY, false, false>(kind);
}

MarchMultiKernel march_multi_kernel_xy(bool wact, bool one) {
  if (one) return wact ? march_multi32<PLANE_XY, true, true> : march_multi32<PLANE_XY, false, true>;
  return wact ? march_multi32<PLANE_XY, true, false> : march_multi32<PLANE_XY, false, false>;
}

}  // namespace fv
