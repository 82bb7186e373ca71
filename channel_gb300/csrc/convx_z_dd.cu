// Fixed-point z transforms (convx.cuh), VV in type dd.
#include "convx.cuh"

namespace chgpu {

template <> bool launch_fx_z<dd>(const ConvLaunch& L, cudaStream_t s, int stage) {
  switch (L.d.nzd) {
#define CHGPU_LEN(N) case N: fx_launch_z<dd, N>(L, s, stage); return true;
    CHGPU_FX_ZLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
    default: return false;
  }
}
template <> cudaError_t fx_z_smem_limits<dd>(int nzd) {
  switch (nzd) {
#define CHGPU_LEN(N) case N: return fx_limits_z<dd, N>();
    CHGPU_FX_ZLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
    default: return cudaSuccess;
  }
}

}  // namespace chgpu
