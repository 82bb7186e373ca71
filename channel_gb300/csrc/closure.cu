// Velocity gradients of the coarse field for the learned closure.
//
// k_grad_xz: d/dx and d/dz, the products with i alfa0 kx and i beta0 kz,
// one thread per value.  k_grad: one thread per (mode, velocity component
// c), d/dy by the compact
// derivative COMPLEXderiv (dnsdata.f90:339-373): the d1 stencil with the
// one-sided wall values d140/d14m1/d14n/d14np1 folded in, then the two
// sweeps of the D0mat factorisation (LeftLU5divStep1 bottom-up,
// LeftLU5divStep2 top-down; rbparmat_blocking.f90:57-100).  G holds nine
// fields in the layout of V: G[3c + 0, 1, 2] = d/dx, d/dy, d/dz of V[c].
#include <cuda_runtime.h>

#include "chgpu_internal.h"
#include "kernels.cuh"

namespace chgpu {

namespace {

__device__ __forceinline__ size_t gidx(const Dims& d, int c, int iy, int m) {
  return ((size_t)c * d.nplanes + (iy + 1)) * d.nmodes + m;
}
__device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 rm(double s, double2 a) { return make_double2(s * a.x, s * a.y); }

// d/dx and d/dz: one thread per mode for kGradPlanes planes and the three
// components, which share its two wavenumbers: per value the FP64 pipe does
// the four products, where forming the wavenumbers for each took eight
// operations and the pipe's time (289 -> 165 us at 127x192x127, 0.9 GB)
constexpr int kGradPlanes = 4;
__global__ void __launch_bounds__(256) k_grad_xz(const double2* __restrict__ V, double2* __restrict__ G, Dims d) {
  const int m = blockIdx.x * 256 + threadIdx.x, p0 = blockIdx.y * kGradPlanes;
  if (m >= d.nmodes) return;
  const size_t per_c = (size_t)d.nplanes * d.nmodes;
  const int ix = m / d.nzt, kz = m - ix * d.nzt - d.nz;
  const double ka = d.alfa0 * ix, kb = d.beta0 * kz;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int p = 0; p < kGradPlanes; ++p) {
      if (p0 + p >= d.nplanes) continue;
      const size_t r = (size_t)(p0 + p) * d.nmodes + m;
      const double2 v = V[c * per_c + r];
      G[(size_t)(3 * c) * per_c + r] = make_double2(-ka * v.y, ka * v.x);
      G[(size_t)(3 * c + 2) * per_c + r] = make_double2(-kb * v.y, kb * v.x);
    }
}

// d/dy: one thread per (mode, component), the two sweeps along y.  A thread is
// one serial chain, and a small field has few of them, so nothing of a row is
// loaded at its use: the stencil's window moves through registers with the
// values that enter it fetched kAhead rows before, and the rows' coefficients
// (a cache line or two per row, read by every thread) are staged in shared
// memory kStage rows at a time.  At 47x96x47 (13 680 threads) 182 -> 101 us;
// at 127x192x127 1.30 -> 0.96 ms.
__global__ void __launch_bounds__(64) k_grad(const double2* __restrict__ V, double2* __restrict__ G,
                                             const double* __restrict__ der, const double* __restrict__ d0lu,
                                             BcRows bc, Dims d) {
  constexpr int kAhead = 4, kStage = 64;
  __shared__ double tab[kStage * 8];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = t < 3 * d.nmodes;
  const int c = active ? t / d.nmodes : 0, m = active ? t - c * d.nmodes : 0;
  const int ny = d.ny;
  auto dot5 = [&](int iy0, const double* w) {
    double2 a = rm(w[0], V[gidx(d, c, iy0, m)]);
    for (int j = 1; j < 5; ++j) a = a + rm(w[j], V[gidx(d, c, iy0 + j, m)]);
    return a;
  };
  // wall values, then Step1 bottom-up parked in the d/dy slot, then Step2
  const double2 f0 = dot5(-1, bc.d140), fm1 = dot5(-1, bc.d14m1);
  const double2 fn = dot5(ny - 3, bc.d14n), fn1 = dot5(ny - 3, bc.d14np1);
  double2* out = G + gidx(d, 3 * c + 1, 0, m) - (size_t)d.nmodes;  // out[(iy+1)*nmodes] = d/dy at iy
  auto put = [&](int iy, double2 v) {
    if (active) out[(size_t)(iy + 1) * d.nmodes] = v;
  };
  const double2 zero = make_double2(0.0, 0.0);
  {
    auto at = [&](int iy) { return iy >= -1 ? V[gidx(d, c, iy, m)] : zero; };
    // V at iy-2 ... iy+2 of the next row iy, and the kAhead values that enter the window after it
    double2 v0 = at(ny - 3), v1 = at(ny - 2), v2 = at(ny - 1), v3 = at(ny), v4 = at(ny + 1);
    double2 q[kAhead], x1 = zero, x2 = zero;
#pragma unroll
    for (int k = 0; k < kAhead; ++k) q[k] = at(ny - 4 - k);
    const double* d0 = der;  // the d0 rows, whose wall columns fold in the boundary values
    for (int base = ny - 1; base >= 1; base -= kStage) {
      __syncthreads();
      for (int i = threadIdx.x; i < kStage * 8; i += blockDim.x) {
        const int iy = base - i / 8, j = i % 8;
        if (iy >= 1) tab[i] = j < 5 ? der[(size_t)iy * 20 + 5 + j] : d0lu[(size_t)(iy - 1) * 5 + j - 3];
      }
      __syncthreads();
      for (int top = base; top > base - kStage && top >= 1; top -= kAhead) {
        double2 nq[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) nq[k] = at(top - 3 - kAhead - k);
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          const int iy = top - k;
          if (iy >= 1) {
            const double* w = tab + (base - iy) * 8;  // d1 row, then the factors 1/pivot, u1, u2
            double2 f = rm(w[0], v0) + rm(w[1], v1);
            f = f + rm(w[2], v2);
            f = f + rm(w[3], v3);
            f = f + rm(w[4], v4);
            if (iy <= 2 || iy >= ny - 2) {
              const double* dr = d0 + (size_t)iy * 20;
              if (iy == ny - 1) f = f - (rm(dr[3], fn) + rm(dr[4], fn1));
              if (iy == ny - 2) f = f - rm(dr[4], fn);
              if (iy == 1) f = f - (rm(dr[1], f0) + rm(dr[0], fm1));
              if (iy == 2) f = f - rm(dr[0], f0);
            }
            const double2 s = rm(w[6], x1) + rm(w[7], x2);
            const double2 x = rm(w[5], f - s);
            x2 = x1;
            x1 = x;
            put(iy, x);
          }
          v4 = v3;
          v3 = v2;
          v2 = v1;
          v1 = v0;
          v0 = q[k];
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) q[k] = nq[k];
      }
    }
  }
  put(-1, fm1);
  put(0, f0);
  auto parked = [&](int iy) { return active && iy <= ny - 1 ? out[(size_t)(iy + 1) * d.nmodes] : zero; };
  double2 bm2 = fm1, bm1 = f0, q[kAhead];
#pragma unroll
  for (int k = 0; k < kAhead; ++k) q[k] = parked(1 + k);
  for (int base = 1; base <= ny - 1; base += kStage) {
    __syncthreads();
    for (int i = threadIdx.x; i < kStage * 2; i += blockDim.x) {
      const int iy = base + i / 2;
      if (iy <= ny - 1) tab[i] = d0lu[(size_t)(iy - 1) * 5 + i % 2];
    }
    __syncthreads();
    for (int low = base; low < base + kStage && low <= ny - 1; low += kAhead) {
      double2 nq[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) nq[k] = parked(low + kAhead + k);
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const int iy = low + k;
        if (iy > ny - 1) break;
        const double* w = tab + (iy - base) * 2;
        const double2 vp = q[k] - (rm(w[0], bm2) + rm(w[1], bm1));
        bm2 = bm1;
        bm1 = vp;
        put(iy, vp);
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) q[k] = nq[k];
    }
  }
  put(ny, fn);
  put(ny + 1, fn1);
}

}  // namespace

void launch_gradients(const double2* V, double2* G, const double* der, const double* d0lu, const BcRows& bc,
                      const Dims& d, cudaStream_t s) {
  k_grad_xz<<<dim3((unsigned)((d.nmodes + 255) / 256), (d.nplanes + kGradPlanes - 1) / kGradPlanes), 256, 0, s>>>(V, G, d);
  const int n = 3 * d.nmodes;
  k_grad<<<(n + 63) / 64, 64, 0, s>>>(V, G, der, d0lu, bc, d);
}

}  // namespace chgpu
