// Register-blocked transform kernels (convf.cuh) instantiated for float.
#include "convf.cuh"

namespace chgpu {

template <>
bool launch_convolutions_r<float>(const ConvLaunch& L, cudaStream_t s, int stage) {
  if (stage == 1 && L.tau) return false;
  return launch_convolutions_r_impl<float>(L, s, stage);
}
cudaError_t convr_set_smem_limits(int n) { return set_limits_type<float>(n); }

}  // namespace chgpu
