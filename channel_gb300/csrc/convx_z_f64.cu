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
template <> cudaError_t fx_z_smem_limits<double>(int nzd) {
  switch (nzd) {
#define CHGPU_LEN(N) case N: return fx_limits_z<double, N>();
    CHGPU_FX_ZLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
    default: return cudaSuccess;
  }
}

bool launch_fx_tke_z(const TkeLaunch& L, int p0, int planes, bool inverse, cudaStream_t s) {
  switch (L.d.nzd) {
#define CHGPU_LEN(N) case N: fx_launch_tke_z<N>(L, p0, planes, inverse, s); return true;
    CHGPU_FX_ZLENGTHS(CHGPU_LEN)
#undef CHGPU_LEN
    default: return false;
  }
}

}  // namespace chgpu
