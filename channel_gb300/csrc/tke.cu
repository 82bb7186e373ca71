// Spanwise spectra of the Reynolds-stress budgets on the device: the
// per-snapshot accumulation of the reference's post-processing program
// postpro/tke/uiuj_spectra.f90 (:161-240), from the handle's current field.
//
//   k_tke_prep   : the fluctuation u' = V with the mean profiles U(y), W(y)
//                  taken off the (0,0) mode (:172-174) into fields 0..2 of
//                  the work buffer W; fields 3 + 3i + k then receive
//                  du'_i/dx_k from launch_gradients (get_gradient_33,
//                  :469-486: i alfa0 kx, compact d/dy, i beta0 kz).
//   k_tke_zinv / k_tke_x / k_tke_zfwd : the convective term
//                  N_i = F(sum_k u'_k du'_i/dx_k) formed on the 3/2-padded
//                  physical grid and brought back to the kept modes with
//                  `factor`, in chunks of planes (the ttrsp block, :182-227;
//                  the sum over k is taken before the forward transform,
//                  which the linearity of the transform and of the product allows).
//   k_tke_accum  : one thread per (plane, kz), the sum over kx with weight
//                  c = 1 (kx = 0), 2 of var, prod, psdiss, ttrsp and, with a
//                  pressure field, pstrain and PHIptrsp for the six pairs
//                  uu, vv, ww, uv, vw, uw (:161-180, :230-233), added to
//                  the running sums acc[term][pair][plane][kz].
// Everything is FP64 (the reference's arithmetic), in every precision path;
// lengths with a compile-time plan take the fixed-point kernels of convx.cuh
// instead of the three here (a sample at 127x192x127: z-inverses 11.4 -> 1.09
// ms, x rows 16.1 -> 3.36, z-forward 2.83 -> 0.26, of 33.7 -> 8.05 in all).
#include <cuda_runtime.h>

#include "chgpu_internal.h"
#include "cplx.cuh"
#include "kernels.cuh"

namespace chgpu {

namespace {

__global__ void k_tke_prep(const double2* __restrict__ V, double2* __restrict__ W, const double* __restrict__ mean,
                           Dims d) {
  const size_t per_c = (size_t)d.nplanes * d.nmodes;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * per_c) return;
  const int c = (int)(t / per_c);
  const size_t r = t - (size_t)c * per_c;
  const int plane = (int)(r / d.nmodes);
  const int m = (int)(r - (size_t)plane * d.nmodes);
  double2 v = V[t];
  if (m == d.nz && c != 1) v.x -= mean[(c == 0 ? 0 : d.nplanes) + plane];  // mode (0,0): U and W
  W[t] = v;
}

// the pressure's mean profile off its (0,0) mode
__global__ void k_tke_pmean(double2* __restrict__ P, const double* __restrict__ meanp, Dims d) {
  const int plane = blockIdx.x * blockDim.x + threadIdx.x;
  if (plane < d.nplanes) P[(size_t)plane * d.nmodes + d.nz].x -= meanp[plane];
}

// z-inverse of one column of field f at one plane of the chunk
__global__ void __launch_bounds__(256) k_tke_zinv(const double2* __restrict__ W, double2* __restrict__ Zt,
                                                  const double2* __restrict__ twz, Dims d, RadixDev rz, int p0,
                                                  int C) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nzd = d.nzd, nz = d.nz, nxp = d.nx + 1;
  double2* a = reinterpret_cast<double2*>(smem_raw);
  double2* b = a + pad32_size(nzd);
  const int ix = blockIdx.x, pl = blockIdx.y, f = blockIdx.z;
  const double2* src = W + ((size_t)f * d.nplanes + p0 + pl) * d.nmodes + (size_t)ix * d.nzt;
  for (int jz = threadIdx.x; jz < nzd; jz += blockDim.x) {
    double2 v = make_double2(0.0, 0.0);
    if (jz <= nz) v = src[nz + jz];
    else if (jz >= nzd - nz) v = src[jz - nzd + nz];
    a[pad32(jz)] = v;
  }
  __syncthreads();
  double2* res = fft_block<+1>(a, b, 1, rz, twz);
  double2* out = Zt + (((size_t)f * C + pl) * nxp + ix) * nzd;
  for (int jz = threadIdx.x; jz < nzd; jz += blockDim.x) out[jz] = res[pad32(jz)];
}

// One plane row jz: for k = 0..2, the c2r of u'_k and du'_i/dx_k (i = 0..2)
// and N_i += u'_k du'_i/dx_k; then the r2c of N_0..2 with `factor`
// (g = factor/2 and twh[2M + k] = (factor/2) e^{-i pi k/M}, as in k_xrow).
__global__ void __launch_bounds__(256) k_tke_x(const double2* __restrict__ Zt, double2* __restrict__ Xt,
                                               const double2* __restrict__ twx, const double2* __restrict__ twh,
                                               Dims d, RadixDev rx, double g, int C) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = d.nxd, nx = d.nx, nxp = nx + 1, nzd = d.nzd;
  const int jz = blockIdx.x, pl = blockIdx.y;
  double2* Cb = reinterpret_cast<double2*>(smem_raw);
  double2* A = Cb + pad32_size(4 * M);
  double2* B = A + pad32_size(4 * M);
  double2* N = B + pad32_size(4 * M);
  for (int i = threadIdx.x; i < 3 * M; i += blockDim.x) N[pad32(i)] = make_double2(0.0, 0.0);
  for (int k = 0; k < 3; ++k) {
    // rows: u'_k, then du'_i/dx_k for i = 0..2 (work-buffer fields k, 3 + 3i + k)
    for (int idx = threadIdx.x; idx < 4 * M; idx += blockDim.x) {
      const int q = idx / M, kx = idx - q * M;
      const int f = q == 0 ? k : 3 + 3 * (q - 1) + k;
      double2 v = make_double2(0.0, 0.0);
      if (kx <= nx) v = Zt[(((size_t)f * C + pl) * nxp + kx) * nzd + jz];
      Cb[pad32(idx)] = v;
    }
    __syncthreads();
    // c2r packing (as k_xrow): Z = (X_k + conj X_{M-k}) + i (X_k - conj X_{M-k}) e^{+i pi k/M}
    for (int idx = threadIdx.x; idx < 4 * M; idx += blockDim.x) {
      const int q = idx / M, kx = idx - q * M;
      double2 xk = Cb[pad32(idx)];
      double2 xm = make_double2(0.0, 0.0);
      if (kx == 0) xk.y = 0.0;
      else xm = conjg(Cb[pad32(q * M + M - kx)]);
      const double2 e = xk + xm, o = cmul_s<+1>(xk - xm, twh[kx]);
      A[pad32(idx)] = e + mul_is<+1>(o);
    }
    __syncthreads();
    double2* U = fft_block<+1>(A, B, 4, rx, twx);
    for (int idx = threadIdx.x; idx < 3 * M; idx += blockDim.x) {
      const int i = idx / M, m = idx - i * M;
      const double2 u = U[pad32(m)], gi = U[pad32((1 + i) * M + m)];
      double2& n = N[pad32(idx)];
      n = make_double2(n.x + u.x * gi.x, n.y + u.y * gi.y);
    }
    __syncthreads();
  }
  double2* P = fft_block<-1>(N, A, 3, rx, twx);
  for (int idx = threadIdx.x; idx < 3 * nxp; idx += blockDim.x) {
    const int i = idx / nxp, kx = idx - i * nxp;
    const double2 zk = P[pad32(i * M + kx)];
    const double2 zm = conjg(P[pad32(i * M + (kx == 0 ? 0 : M - kx))]);
    const double2 sm = zk + zm, df = zk - zm;
    const double2 w = twh[2 * M + kx];
    Xt[(((size_t)i * C + pl) * nxp + kx) * nzd + jz] =
        make_double2(fma(g, sm.x, fma(w.x, df.y, w.y * df.x)), fma(g, sm.y, fma(w.y, df.y, -(w.x * df.x))));
  }
}

// z-forward of one column of N_i, truncated to |kz| <= nz
__global__ void __launch_bounds__(256) k_tke_zfwd(const double2* __restrict__ Xt, double2* __restrict__ N3,
                                                  const double2* __restrict__ twz, Dims d, RadixDev rz, int p0,
                                                  int C) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nzd = d.nzd, nz = d.nz, nxp = d.nx + 1;
  double2* a = reinterpret_cast<double2*>(smem_raw);
  double2* b = a + pad32_size(nzd);
  const int ix = blockIdx.x, pl = blockIdx.y, i = blockIdx.z;
  const double2* src = Xt + (((size_t)i * C + pl) * nxp + ix) * nzd;
  for (int jz = threadIdx.x; jz < nzd; jz += blockDim.x) a[pad32(jz)] = src[jz];
  __syncthreads();
  double2* res = fft_block<-1>(a, b, 1, rz, twz);
  double2* out = N3 + ((size_t)i * d.nplanes + p0 + pl) * d.nmodes + (size_t)ix * d.nzt;
  for (int izp = threadIdx.x; izp < d.nzt; izp += blockDim.x) {
    const int iz = izp - nz;
    out[izp] = res[pad32(iz >= 0 ? iz : nzd + iz)];
  }
}

// The terms accumulated per snapshot: var, prod, psdiss, ttrsp, pstrain,
// PHIptrsp (the rest follow at the end by y derivatives).
//
// Bound by the FP64 pipe: with the weights c and the factors -1, -2 ni applied
// to the sums over kx, and prod formed from the sums of var, a mode takes 66
// multiply-adds (18 more with a pressure) where applying them per mode took
// about 160; 1.63 -> 0.86 ms at 127x192x127 (1.5 GB).
template <bool PRESSURE>
__global__ void __launch_bounds__(128) k_tke_accum(const double2* __restrict__ W, const double2* __restrict__ N3,
                                                   const double2* __restrict__ P, double* __restrict__ acc,
                                                   const double* __restrict__ mgrad, Dims d) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int S = d.nplanes * d.nzt;
  if (t >= S) return;
  const int plane = t / d.nzt, izp = t - plane * d.nzt;
  const size_t FS = (size_t)d.nplanes * d.nmodes;
  constexpr int PI_[6] = {0, 1, 2, 0, 1, 0}, PJ_[6] = {0, 1, 2, 1, 2, 2};
  // sums over kx of u_i u_j, sum_k g_ik g_jk, N_i u_j, p (g_ij + g_ji), p u_i
  double uu[6], gg[6], nu[3][3], pg[PRESSURE ? 6 : 1], pu[PRESSURE ? 3 : 1];
#pragma unroll
  for (int r = 0; r < 6; ++r) uu[r] = gg[r] = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) nu[i][j] = 0.0;
#pragma unroll
  for (int r = 0; r < (PRESSURE ? 6 : 1); ++r) pg[r] = 0.0;
#pragma unroll
  for (int i = 0; i < (PRESSURE ? 3 : 1); ++i) pu[i] = 0.0;
  for (int ix = d.nx; ix >= 0; --ix) {
    if (ix == 0) {  // kx > 0 stands for -kx too
#pragma unroll
      for (int r = 0; r < 6; ++r) uu[r] *= 2.0, gg[r] *= 2.0;
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) nu[i][j] *= 2.0;
#pragma unroll
      for (int r = 0; r < (PRESSURE ? 6 : 1); ++r) pg[r] *= 2.0;
#pragma unroll
      for (int i = 0; i < (PRESSURE ? 3 : 1); ++i) pu[i] *= 2.0;
    }
    const size_t base = (size_t)plane * d.nmodes + (size_t)ix * d.nzt + izp;
    double2 u[3], n[3], gr[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      u[i] = W[i * FS + base];
      n[i] = N3[i * FS + base];
#pragma unroll
      for (int k = 0; k < 3; ++k) gr[i][k] = W[(size_t)(3 + 3 * i + k) * FS + base];
    }
    auto add = [](double& s, double2 a, double2 b) { s = fma(a.x, b.x, fma(a.y, b.y, s)); };  // s += Re(conj(a) b)
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      add(uu[r], u[PI_[r]], u[PJ_[r]]);
#pragma unroll
      for (int k = 0; k < 3; ++k) add(gg[r], gr[PI_[r]][k], gr[PJ_[r]][k]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) add(nu[i][j], n[i], u[j]);
    if constexpr (PRESSURE) {
      const double2 p = P[base];
#pragma unroll
      for (int r = 0; r < 6; ++r) add(pg[r], p, gr[PI_[r]][PJ_[r]] + gr[PJ_[r]][PI_[r]]);
#pragma unroll
      for (int i = 0; i < 3; ++i) add(pu[i], p, u[i]);
    }
  }
  auto put = [&](int q, int r, double v) { acc[(size_t)(q * 6 + r) * S + t] += v; };
  // mean velocity gradient M[j][1] (get_mean_grad): dU/dy, 0, dW/dy; the sums u_i v
  const double M[3] = {mgrad[plane], 0.0, mgrad[d.nplanes + plane]}, uv[3] = {uu[3], uu[1], uu[4]};
#pragma unroll
  for (int r = 0; r < 6; ++r) {
    const int i = PI_[r], j = PJ_[r];
    put(0, r, uu[r]);
    put(1, r, -(uv[i] * M[j] + uv[j] * M[i]));
    put(2, r, -2.0 * d.ni * gg[r]);
    put(3, r, -(nu[i][j] + nu[j][i]));
    if constexpr (PRESSURE) {
      put(4, r, pg[r]);
      if (r == 1) put(5, r, -2.0 * pu[1]);
      if (r == 3) put(5, r, -pu[0]);
      if (r == 4) put(5, r, -pu[2]);
    }
  }
}

// The spectra in the reference's order sp[plane][kz][term 0..9][pair] from the
// sums of n samples: the accumulated terms var, prod, psdiss, ttrsp, pstrain,
// PHIptrsp sit at term 0, 1, 2, 3, 5, 9 (uiuj_spectra.f90:13-14, :70), 7 stays
// zero, k_tke_fluxes writes 4, 6 and 8.
__global__ void k_tke_terms(const double* __restrict__ acc, double* __restrict__ sp, double n, int timestwo, size_t S) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 60 * S) return;
  const size_t col = t / 60;
  const int e = (int)(t - 60 * col), term = e / 6, irs = e - 6 * term;
  if (term == 4 || term == 6 || term == 8) return;
  const int q = term <= 3 ? term : term == 5 ? 4 : term == 9 ? 5 : -1;
  double v = q >= 0 ? acc[(size_t)(q * 6 + irs) * S + col] / n : 0.0;
  if (term == 0 && timestwo) v *= 2.0;  // -two (:262)
  sp[t] = v;
}

// The flux derivatives (:243-259), one thread per (term, pair, kz): PHIvdiff =
// ni d/dy var (term 8), vdiff = ni d2/dy2 var (4), ptrsp = d/dy PHIptrsp (6),
// by the compact stencils and the factored D0mat (COMPLEXderiv, dnsdata.f90:
// 339-414) with the first sweep parked in x[term * 6 + pair][plane][kz].
__global__ void __launch_bounds__(64) k_tke_fluxes(const double* __restrict__ acc, double* __restrict__ x,
                                                   double* __restrict__ sp, const double* __restrict__ der,
                                                   const double* __restrict__ d0lu, TkeRows rows, double n, Dims d) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 18 * d.nzt) return;
  const int c = t / d.nzt, izp = t - c * d.nzt, which = c / 6, irs = c - 6 * which;
  const int ny = d.ny;
  const size_t S = (size_t)d.nplanes * d.nzt, st = d.nzt;
  const double* f = acc + (size_t)((which == 2 ? 5 : 0) * 6 + irs) * S + st + izp;  // f[iy * st]
  double* xs = x + (size_t)c * S + st + izp;
  const int term = which == 0 ? 8 : which == 1 ? 4 : 6, dk = which == 1 ? 10 : 5;
  const double scale = which == 2 ? 1.0 : d.ni;
  double* out = sp + ((size_t)izp * 10 + term) * 6 + irs;  // + (iy + 1) * 60 st
  auto F = [&](int iy) { return f[(ptrdiff_t)iy * (ptrdiff_t)st] / n; };
  auto dot5 = [&](int iy0, const double* w) {
    double a = w[0] * F(iy0);
    for (int j = 1; j < 5; ++j) a += w[j] * F(iy0 + j);
    return a;
  };
  const double(&w)[4][5] = rows.w[which == 1];
  const double fm1 = dot5(-1, w[0]), f0 = dot5(-1, w[1]), fn = dot5(ny - 3, w[2]), fn1 = dot5(ny - 3, w[3]);
  double x1 = 0.0, x2 = 0.0;
  // the window F(iy - 2) ... F(iy + 2), its next value loaded ahead
  double v0 = F(ny - 3), v1 = F(ny - 2), v2 = F(ny - 1), v3 = F(ny), v4 = F(ny + 1);
  for (int iy = ny - 1; iy >= 1; --iy) {
    const double next = iy > 1 ? F(iy - 3) : 0.0;
    const double* dr = der + (size_t)iy * 20;
    double s = dr[dk] * v0 + dr[dk + 1] * v1 + dr[dk + 2] * v2 + dr[dk + 3] * v3 + dr[dk + 4] * v4;
    if (iy == ny - 1) s -= dr[3] * fn + dr[4] * fn1;
    if (iy == ny - 2) s -= dr[4] * fn;
    if (iy == 1) s -= dr[1] * f0 + dr[0] * fm1;
    if (iy == 2) s -= dr[0] * f0;
    const double* lu = d0lu + (size_t)(iy - 1) * 5;
    const double v = lu[2] * (s - (lu[3] * x1 + lu[4] * x2));
    x2 = x1;
    x1 = v;
    xs[(size_t)iy * st] = v;
    v4 = v3; v3 = v2; v2 = v1; v1 = v0; v0 = next;
  }
  auto put = [&](int iy, double v) { out[(size_t)(iy + 1) * 60 * st] = v * scale; };
  put(-1, fm1);
  put(0, f0);
  double bm2 = fm1, bm1 = f0, cur = xs[st];
  for (int iy = 1; iy <= ny - 1; ++iy) {
    const double next = iy < ny - 1 ? xs[(size_t)(iy + 1) * st] : 0.0;
    const double* lu = d0lu + (size_t)(iy - 1) * 5;
    const double v = cur - (lu[0] * bm2 + lu[1] * bm1);
    put(iy, v);
    bm2 = bm1;
    bm1 = v;
    cur = next;
  }
  put(ny, fn);
  put(ny + 1, fn1);
}

// profiles[plane][term][pair]: the sum over kz
__global__ void k_tke_profiles(const double* __restrict__ sp, double* __restrict__ prof, int nplanes, int nzt) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 60 * nplanes) return;
  const int plane = t / 60, e = t - 60 * plane;
  const double* src = sp + (size_t)plane * nzt * 60 + e;
  double s = 0.0;
#pragma unroll 8
  for (int izp = 0; izp < nzt; ++izp) s += src[(size_t)izp * 60];
  prof[t] = s;
}

}  // namespace

// 24 MB of spectra at 127x192x127: 0.7 to 1.3 ms with their copy to the host's
// memory (the derivatives' serial sweeps 0.40 of it), 14 ms when the host worked
// on the copied sums.
void launch_tke_result(const double* acc, double* sp, double* work, double* prof, const double* der,
                       const double* d0lu, const TkeRows& rows, const Dims& d, double n, int timestwo,
                       cudaStream_t s) {
  const size_t S = (size_t)d.nplanes * d.nzt;
  k_tke_terms<<<(unsigned)((60 * S + 255) / 256), 256, 0, s>>>(acc, sp, n, timestwo, S);
  k_tke_fluxes<<<(18 * d.nzt + 63) / 64, 64, 0, s>>>(acc, work, sp, der, d0lu, rows, n, d);
  k_tke_profiles<<<(60 * d.nplanes + 127) / 128, 128, 0, s>>>(sp, prof, d.nplanes, d.nzt);
}

size_t tke_z_smem(int nzd) { return 2 * (size_t)pad32_size(nzd) * sizeof(double2); }
size_t tke_x_smem(int nxd) { return (3 * (size_t)pad32_size(4 * nxd) + pad32_size(3 * nxd)) * sizeof(double2); }

cudaError_t tke_set_smem_limits(int nzd, int nxd) {
  cudaError_t e = cudaFuncSetAttribute(k_tke_zinv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tke_z_smem(nzd));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_tke_zfwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tke_z_smem(nzd));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_tke_x, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tke_x_smem(nxd));
  if (e == cudaSuccess) e = fx_z_smem_limits<double>(nzd);
  if (e == cudaSuccess) e = fx_tke_x_smem_limits(nxd);
  return e;
}

void launch_tke_snapshot(const TkeLaunch& L, cudaStream_t s) {
  const Dims& d = L.d;
  const size_t per_c = (size_t)d.nplanes * d.nmodes;
  k_tke_prep<<<(unsigned)((3 * per_c + 255) / 256), 256, 0, s>>>(L.V, L.W, L.mean, d);
  if (L.P) k_tke_pmean<<<(d.nplanes + 127) / 128, 128, 0, s>>>(L.P, L.mean + 2 * d.nplanes, d);
  launch_gradients(L.W, L.W + 3 * per_c, L.der, L.d0lu, L.bc, d, s);
  const int nxp = d.nx + 1;
  for (int p0 = 0; p0 < d.nplanes; p0 += L.chunk) {
    const int C = d.nplanes - p0 < L.chunk ? d.nplanes - p0 : L.chunk;
    // the fixed-point kernels for the lengths with a plan
    if (!launch_fx_tke_z(L, p0, C, true, s))
      k_tke_zinv<<<dim3(nxp, C, 12), 256, tke_z_smem(d.nzd), s>>>(L.W, L.Zt, L.twz, d, L.rz, p0, L.chunk);
    if (!launch_fx_tke_x(L, C, s))
      k_tke_x<<<dim3(d.nzd, C), 256, tke_x_smem(d.nxd), s>>>(L.Zt, L.Xt, L.twx, L.twh, d, L.rx, 0.5 * d.factor,
                                                            L.chunk);
    if (!launch_fx_tke_z(L, p0, C, false, s))
      k_tke_zfwd<<<dim3(nxp, C, 3), 256, tke_z_smem(d.nzd), s>>>(L.Xt, L.N3, L.twz, d, L.rz, p0, L.chunk);
  }
  const int S = d.nplanes * d.nzt;
  if (L.P)
    k_tke_accum<true><<<(S + 127) / 128, 128, 0, s>>>(L.W, L.N3, L.P, L.acc, L.mean + 3 * d.nplanes, d);
  else
    k_tke_accum<false><<<(S + 127) / 128, 128, 0, s>>>(L.W, L.N3, nullptr, L.acc, L.mean + 3 * d.nplanes, d);
}

}  // namespace chgpu
