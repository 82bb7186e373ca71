// Fixed-point x rows with the closure's stresses (convx.cuh).
#include "convx.cuh"

namespace chgpu {

bool launch_fx_x_tau(const ConvLaunch& L, cudaStream_t s) {
  switch (L.d.nxd) {
#define CHGPU_LEN(N) case N: fx_launch_x<N, true>(L, s); return true;
    CHGPU_FX_XLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
    default: return false;
  }
}
cudaError_t fx_x_tau_smem_limits(int nxd) {
  switch (nxd) {
#define CHGPU_LEN(N) case N: return fx_limits_x<N, true>();
    CHGPU_FX_XLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
    default: return cudaSuccess;
  }
}

}  // namespace chgpu
