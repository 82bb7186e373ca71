// Fixed-point x rows of the budget spectra (convx.cuh).
#include "convx.cuh"

namespace chgpu {

bool launch_fx_tke_x(const TkeLaunch& L, int planes, cudaStream_t s) {
  switch (L.d.nxd) {
#define CHGPU_LEN(N) case N: fx_launch_tke_x<N>(L, planes, s); return true;
    CHGPU_FX_XLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
    default: return false;
  }
}
cudaError_t fx_tke_x_smem_limits(int nxd) {
  switch (nxd) {
#define CHGPU_LEN(N) case N: return fx_limits_tke_x<N>();
    CHGPU_FX_XLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
    default: return cudaSuccess;
  }
}

}  // namespace chgpu
