// Fixed-point z transforms (convx.cuh), VV in type double.
#include "convx.cuh"

namespace chgpu {

template <> bool launch_fx_z<double>(const ConvLaunch& L, cudaStream_t s, int stage) {
  switch (L.d.nzd) {
#define CHGPU_LEN(N) case N: fx_launch_z<double, N>(L, s, stage); return true;
    CHGPU_FX_ZLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
    default: return false;
  }
}
template <> cudaError_t fx_z_smem_limits<double>() {
  cudaError_t e = cudaSuccess;
#define CHGPU_LEN(N) if (e == cudaSuccess) e = fx_limits_z<double, N>();
  CHGPU_FX_ZLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
  return e;
}

}  // namespace chgpu
