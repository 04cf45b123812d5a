// fv_march32_xz.cu -- the warp-marched FP32-mixed kernels (fv_march32.cuh) of
// the x-z plane.
#include "fv_march32.cuh"

namespace fv {

MarchKernel march_kernel_xz(bool wact, int kind, bool one) {
  if (one) return wact ? march_kernel_of<PLANE_XZ, true, true>(kind) : march_kernel_of<PLANE_XZ, false, true>(kind);
  return wact ? march_kernel_of<PLANE_XZ, true, false>(kind) : march_kernel_of<PLANE_XZ, false, false>(kind);
}

MarchMultiKernel march_multi_kernel_xz(bool wact, bool one) {
  if (one) return wact ? march_multi32<PLANE_XZ, true, true> : march_multi32<PLANE_XZ, false, true>;
  return wact ? march_multi32<PLANE_XZ, true, false> : march_multi32<PLANE_XZ, false, false>;
}

}  // namespace fv
