// The three transform kernels of `convolutions` (dnsdata.f90:487-602) for the
// FP64 and double-float paths on 64-bit block fixed point (fx.cuh), with the
// register-blocked passes of rfft.cuh:
//
//   k_zinv_x : one group of TPR threads per (plane, component, column kx).
//              The modes go straight to registers in the transform's input
//              distribution, the 3/2 zero band stays zero
//              (dnsdata.f90:504-510); Zb gets the physical-z column.  Two
//              scales: pass 1 combines one thread's inputs, so the largest
//              sum over a thread bounds it, the later passes' values are
//              bounded by the sum over the column.
//   k_xrow_x : one group per plane row jz, NR rows per block, staged through
//              shared memory as the zTOx / xTOz transposes
//              (mpi_transpose.f90:50-117).  Per row: u, v, w packed for the
//              half-length c2r (dnsdata.f90:533-535) and transformed, each
//              normalised by the row's largest value so that the six
//              products (:581-584) are 64x64-bit products of full-width
//              numbers; the CFL maximum in FP64 (:552-556); the products
//              transformed forward and unpacked for kx = 0..nx (:586-588).
//   k_zfwd_x : one group per (plane, product, column): the column's scale
//              from its largest value, the forward transform, |kz| <= nz
//              stored (:590).
//
// V, Zb and Pb are FP64; VV is FP64 or, in the double-float path (whose
// stencils read it), double-float.
//
// What bounds them (GB300, counters at 255x64x255): latency at 12 (k_xrow_x,
// by its rows' shared memory) to 15 warps per SM, with 46-56% of the issue
// slots and 58-59% of the integer multiply-add pipe taken; in the z kernels the
// conversions of their inputs and outputs also take half of the FP64 pipe.  Not
// memory: 2 TB/s in the z kernels.  Against the FP64-pipe transforms they
// replace, ms per step: k_zinv, k_xrow, k_zfwd 3.77, 23.2, 7.47 -> 0.85, 4.75,
// 1.55 at 127x192x127, 108, 853, 214 -> 24, 185, 49 at 383x384x383; the
// double-float ones 41, 291, 70 -> 24, 185, 56.  In-place packing by pairs of
// entries, one code path for the three inverse rows: k_xrow_x 38.7 -> 28.7 ms at
// 255x256x255.
#pragma once

#include <cuda_runtime.h>

#include "chgpu_internal.h"
#include "cplx.cuh"
#include "fx.cuh"
#include "kernels.cuh"
#include "rfft.cuh"

namespace chgpu {

namespace {

// reductions over a transform group; TPR > 32: through scratch (the group's
// exchange buffer, not in use)
enum { kRedMax, kRedSum, kRedOr };
template <int OP> __device__ __forceinline__ int red_op(int a, int b) {
  return OP == kRedMax ? max(a, b) : OP == kRedSum ? a + b : (a | b);
}
template <int OP, int TPR> __device__ __forceinline__ int group_reduce(int v, void* scratch, int t) {
#pragma unroll
  for (int o = (TPR < 32 ? TPR : 32) / 2; o > 0; o >>= 1) v = red_op<OP>(v, __shfl_xor_sync(0xffffffffu, v, o));
  if constexpr (TPR > 32) {
    int* s = static_cast<int*>(scratch);
    if ((t & 31) == 0) s[t >> 5] = v;
    group_sync<TPR>();
    v = s[0];
#pragma unroll
    for (int k = 1; k < TPR / 32; ++k) v = red_op<OP>(v, s[k]);
    group_sync<TPR>();
  }
  return v;
}

__device__ __forceinline__ void xblock_max_atomic(double v, double* target) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __shared__ double wmax[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) wmax[wid] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) m = wmax[i] > m ? wmax[i] : m;
    // non-negative doubles order like their bit patterns
    atomicMax(reinterpret_cast<unsigned long long*>(target), (unsigned long long)__double_as_longlong(m));
  }
}

// The planes a physical-z buffer holds: `planes` of them from `first` on.
struct FxWindow {
  int first, planes;
};

// columns per z block: 128 threads, at most 32 columns
template <int TPR> constexpr int fx_zcols() { return (128 / TPR) < 32 ? (128 / TPR) : 32; }
// shared memory per x row in elements: SLOTS rows, the last the padded
// exchange buffer (u and v in physical space before it in k_xrow_x, u, v and
// w in k_tke_x_x), then pad so that a block's transposing accesses (NR rows
// of consecutive elements) spread over the banks: a wavefront of 16-byte
// elements is 8 lanes, NR rows of 8 / NR elements
template <int M, int TPR, int SLOTS = 3> constexpr int fx_row_stride(int nr) {
  int s = SLOTS * M + TPR;
  while (s % 8 != (nr < 8 ? 8 / nr % 8 : 1)) ++s;
  return s;
}
// rows per x block: at most 32 and 128 threads, within a third of an SM's 228
// KB (1 KB reserved per block)
template <int M, int TPR, int SLOTS = 3> constexpr int fx_xrows() {
  int nr = 32;
  const int budget = 233472 / 3 - 1024;
  while (nr > 1 && (nr * fx_row_stride<M, TPR, SLOTS>(nr) * 16 > budget || nr * TPR > 128)) nr /= 2;
  while (nr * TPR < 32) nr *= 2;
  return nr;
}
// resident blocks the registers are capped for: what shared memory allows, at
// most 12 warps per SM (168 registers) with 12 points per thread, 16 with 8
template <int M, int TPR, int SLOTS = 3> constexpr int fx_xminb() {
  const int nr = fx_xrows<M, TPR, SLOTS>();
  const int by_smem = 233472 / (nr * fx_row_stride<M, TPR, SLOTS>(nr) * 16 + 1024);
  const int by_regs = (M / TPR == 8 ? 512 : 384) / (nr * TPR);
  const int b = by_smem < by_regs ? by_smem : by_regs;
  return b < 1 ? 1 : b;
}
// resident z blocks: as many as the registers allow, 12, 20 or 24 warps per SM
// with 24, 12 or 8 points per thread (k_zfwd_x at nzd = 256 and 79x101x75:
// 0.382 ms per step with 12 warps, 0.322 with 20, 0.300 with 24)
template <int E, int TPR, int NC> constexpr int fx_zminb() {
  return (E == 24 ? 384 : E == 12 ? 640 : 768) / (NC * TPR);
}

// Between two passes: the values of the group's transform shifted so that the
// largest |re|, |im| is just below 2^BITS, or by `most` >= -62 to the left if
// that is less.  Returns the shift to the left.
template <int E, int TPR, int BITS>
__device__ __forceinline__ int fx_renormalise(fx2 (&a)[E], int most, void* scratch, int t) {
  int m = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int hx = fx_up(a[e].x), hy = fx_up(a[e].y);
    m |= (hx ^ (hx >> 31)) | (hy ^ (hy >> 31));
  }
  m = group_reduce<kRedOr, TPR>(m, scratch, t);
  const int s = min(BITS - (64 - __clz(m)), most);
  if (s >= 0) {
#pragma unroll
    for (int e = 0; e < E; ++e) a[e] = fx2{a[e].x << s, a[e].y << s};
  } else {
#pragma unroll
    for (int e = 0; e < E; ++e) a[e] = fx_shr(a[e], -s);
  }
  return s;
}

// Inverse x transform of one row, whose spectrum (FP64, kx = 0..nx) sits in
// the slot F, by its TPR threads: the physical values a[e] at pair t + TPR e,
// normalised so that the row's largest |re|, |im| is just below 2^kRowBits.
// X: the row's exchange buffer (F may be it).  Returns their scale (a zero
// row: kZeroRow or more, beyond every scale); bad |= bit if a mode is not finite.
// Every thread of the block calls it.
constexpr int kRowBits = 60, kZeroRow = 4000;
template <int E, int TPR>
__device__ __forceinline__ int fx_inverse_row(fx2 (&a)[E], fx2* F, fx2* X, int t, int nx, const fx2* __restrict__ tw,
                                              const fx2* __restrict__ twh, int* scratch, int& bad, int bit) {
  using Io = FxIo<double>;
  constexpr int M = E * TPR;
  double2* Fr = reinterpret_cast<double2*>(F);
  int emax = 0;
#pragma unroll 4
  for (int n = t; n <= nx; n += TPR) emax = max(emax, max(Io::expo(Fr[n].x), Io::expo(Fr[n].y)));
  emax = group_reduce<kRedMax, TPR>(emax, scratch, t);
  // |re|, |im| < 2^57, so that the packed |re|, |im| stay below 2^60
  const int s0 = emax == 0 ? kZeroRow : 57 - (emax - Io::kBias + 1);
  if (emax == Io::kExpMax) bad |= bit;
  // c2r by the half-length packing, in place and two entries at a time
  // (only Re of the kx = 0 entry; the x zero band kx > nx, dnsdata.f90:535):
  // with s = X_k + conj X_{M-k} and r = i (X_k - conj X_{M-k}) e^{+i pi k/M}
  //   Z_k = s + r,  Z_{M-k} = conj(s - r)
#pragma unroll 2
  for (int k = t; k <= M / 2; k += TPR) {
    const int kc = M - k;
    fx2 xk{0, 0}, xm{0, 0};
    if (k <= nx) xk = fx_load<double>(Fr[k], s0);
    if (k == 0) xk.y = 0;
    else if (kc <= nx) {
      xm = fx_load<double>(Fr[kc], s0);
      xm.y = -xm.y;
    }
    const fx2 s = xk + xm, r = mul_is<+1>(fx_cmul4<+1>(xk - xm, fx_ldw(twh + k)));
    F[k] = s + r;
    if (k > 0 && kc != k) F[kc] = fx2{s.x - r.x, r.y - s.y};
  }
  group_sync<TPR>();
#pragma unroll
  for (int e = 0; e < E; ++e) a[e] = F[t + TPR * e];
  // the scales of pass 1 (its values are bounded by the largest sum of
  // |re| + |im| over a thread) and of the later passes (the sum over the
  // row), both sums below 2^61: shifts d1, then d2
  unsigned b1 = 0;  // in units of 2^39, at most 2 E 2^21 + 2 E
#pragma unroll
  for (int e = 0; e < E; ++e)
    b1 += (unsigned)(abs(fx_up(a[e].x)) >> 7) + (unsigned)(abs(fx_up(a[e].y)) >> 7) + 2u;
  const unsigned bs = (unsigned)group_reduce<kRedSum, TPR>((int)b1, scratch, t);
  b1 = (unsigned)group_reduce<kRedMax, TPR>((int)b1, scratch, t);
  const int d1 = max(0, 32 - __clz((int)b1) + 39 - 61), d2 = max(d1, 32 - __clz((int)bs) + 39 - 61) - d1;
#pragma unroll
  for (int e = 0; e < E; ++e) a[e] = fx_shr(a[e], d1);
  group_sync<TPR>();  // every read of the packed row before its slot or X is written
  rfft_regs<E, TPR, +1>(a, X, t, tw, [&] {
#pragma unroll
    for (int e = 0; e < E; ++e) a[e] = fx_shr(a[e], d2);
  });
  // normalise: the row's largest |re|, |im| just below 2^kRowBits
  int m = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int hx = fx_up(a[e].x), hy = fx_up(a[e].y);
    m |= (hx ^ (hx >> 31)) | (hy ^ (hy >> 31));
  }
  m = group_reduce<kRedOr, TPR>(m, scratch, t);
  const int sh = __clz(m) - (64 - kRowBits);
#pragma unroll
  for (int e = 0; e < E; ++e) a[e] = fx2{a[e].x << sh, a[e].y << sh};
  return s0 - d1 - d2 - 2 + sh;  // one pass at quarter scale
}

// Forward x transform of one row times `factor`, kx = 0..nx as FP64 values in
// X: a[] holds the row's values below 2^58 at the given scale; nf: they are
// not finite.  `factor` enters in the unpacking: g = (factor/2) 2^-fac.exp in
// [1/2, 1) as fac and in twh[M + k] = g e^{-i pi k/M}.
template <int E, int TPR>
__device__ __forceinline__ void fx_forward_row(fx2 (&a)[E], fx2* X, int t, int nx, const fx2* __restrict__ tw,
                                               const fx2* __restrict__ twh, FxFactor fac, int scale, bool nf,
                                               int* scratch) {
  constexpr int M = E * TPR;
  // below 2^62 after the first pass; before the others they are scaled by
  // their actual largest value to kMid bits, from which no later value exceeds
  // 2^62 and the outputs 2^61 (for the unpacking)
  static_assert(E <= 12, "12 sqrt(2) 2^57.6 < 2^62");
  constexpr int kMid = fx_bits(fx_growth(E, TPR, false), 61);
  // the passes after the first and the unpacking are at quarter scale
  int So = scale - 2 * rplan_passes(E, TPR) - fac.exp;
  rfft<E, TPR, -1, true>(a, X, t, tw, [&](int o, fx2 v) { X[o] = v; }, [&] {
    So += fx_renormalise<E, TPR, kMid>(a, 64, scratch, t);
  });
  const int mode = nf ? kNan : So < FxIo<double>::kSMin || So > FxIo<double>::kSMax ? 1 : 0;
  group_sync<TPR>();
  // r2c unpacking, kx = 0..nx (HFT, dnsdata.f90:586), at quarter scale, in
  // place and two entries at a time: with s = g (Z_k + conj Z_{M-k}) and
  // r = (g w_k) (-i) (Z_k - conj Z_{M-k})
  //   X_k = s + r,  X_{M-k} = conj(s - r)
  double2* Xr = reinterpret_cast<double2*>(X);
#pragma unroll 2
  for (int k = t; k <= min(M / 2, nx); k += TPR) {
    const int kc = M - k;
    const fx2 zk = X[k], zc = X[k == 0 ? 0 : kc];
    const fx2 sm{zk.x + zc.x, zk.y - zc.y}, df{zk.x - zc.x, zk.y + zc.y};
    const fx2 r = fx_cmul<-1>(fx2{df.y, -df.x}, fx_ldw(twh + M + k));
    const fx2 s{fx_mad(0, sm.x, fac.gh, fac.gl), fx_mad(0, sm.y, fac.gh, fac.gl)};
    Xr[k] = fx_store_any(s + r, So, mode);
    if (kc <= nx && kc != k) Xr[kc] = fx_store_any(fx2{s.x - r.x, r.y - s.y}, So, mode);
  }
}

// a[e] += src[TPR e] (FP32 pairs, zeros when not active): values below 2^56
// at scale S become the sums, below 2^56 too, at the scale that both allow.
// Returns whether a source value is not finite.
template <int E, int TPR>
__device__ __forceinline__ bool fx_add_f32(fx2 (&a)[E], int& S, const float2* __restrict__ src, bool active, int t,
                                           int* scratch) {
  float2 f[E];
  int emax = 0;  // 1 for subnormal numbers, 0 for zeros only
#pragma unroll
  for (int e = 0; e < E; ++e) {
    f[e] = active ? __ldg(src + TPR * e) : make_float2(0.f, 0.f);
    auto ex = [](float v) {
      const int b = __float_as_int(v) & 0x7fffffff;
      return b ? max(b >> 23, 1) : 0;
    };
    emax = max(emax, max(ex(f[e].x), ex(f[e].y)));
  }
  emax = group_reduce<kRedMax, TPR>(emax, scratch, t);
  // |f| < 2^(emax - 126): at scale S1 below 2^55, as a at S - 1
  const int S1 = emax == 0 ? kZeroRow : 55 - (emax - 126);
  const int So = min(S - 1, S1);
  const int da = min(S - So, 62);
  // f = +-m 2^(b - 150), b the exponent field (1 for subnormal numbers)
  auto add = [&](long long x, float v) -> long long {
    const int bits = __float_as_int(v), b = max((bits >> 23) & 0xff, 1);
    const int m = (bits & 0x7fffff) | ((bits & 0x7f800000) ? 0x800000 : 0);
    const int sh = b - 150 + So;  // at most 31
    const long long r = sh >= 0 ? (long long)m << min(sh, 31) : ((long long)m + ((1ll << min(-sh, 31)) >> 1)) >> min(-sh, 31);
    return x + (bits < 0 ? -r : r);
  };
#pragma unroll
  for (int e = 0; e < E; ++e) {
    a[e] = fx_shr(a[e], da);
    a[e] = fx2{add(a[e].x, f[e].x), add(a[e].y, f[e].y)};
  }
  S = So;
  return emax == 255;
}

}  // namespace

template <int E, int TPR, int NC>
__global__ void __launch_bounds__(NC * TPR, fx_zminb<E, TPR, NC>()) k_zinv_x(const double2* __restrict__ V,
                                                                       double2* __restrict__ Zb,
                                                                       const fx2* __restrict__ tw, Dims d, int plane0,
                                                                       FxWindow win, int ix_lo, int ix_hi) {
  using In = FxIo<double>;
  constexpr int N = E * TPR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  fx2* buf = reinterpret_cast<fx2*>(smem_raw) + (threadIdx.x / TPR) * rbuf_size<E, TPR>();
  const int t = threadIdx.x % TPR;
  const int c = blockIdx.z, plane = plane0 + blockIdx.y;
  const int ix = ix_lo + blockIdx.x * NC + (int)(threadIdx.x / TPR);
  const bool active = ix < ix_hi;
  const int nz = d.nz, nzt = d.nzt;
  const int cx = active ? ix : ix_lo;
  const double2* src = V + (((size_t)c * d.nplanes + plane) * (d.nx + 1) + cx) * nzt;
  double2 raw[E];
  int emax = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int jz = t + TPR * e;
    const int izp = jz <= nz ? nz + jz : (jz >= N - nz ? jz - N + nz : -1);
    raw[e] = make_double2(0.0, 0.0);
    if (active && izp >= 0) raw[e] = __ldg(src + izp);
    emax = max(emax, max(In::expo(raw[e].x), In::expo(raw[e].y)));
  }
  emax = group_reduce<kRedMax, TPR>(emax, buf, t);
  unsigned B = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) B += fx_lead_at(raw[e].x, emax) + fx_lead_at(raw[e].y, emax);
  const unsigned B1 = (unsigned)group_reduce<kRedMax, TPR>((int)B, buf, t);
  B = (unsigned)group_reduce<kRedSum, TPR>((int)B, buf, t);
  const int S1 = emax == 0 ? 0 : fx_cap<double>(fx_scale_sum<double>(emax, B1, 62), 1);
  const int S = emax == 0 ? 0 : fx_cap<double>(fx_scale_sum<double>(emax, B, 62), 1);
  fx2 a[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {  // conversions only where there is a mode: they fill half the FP64 pipe
    const int jz = t + TPR * e;
    a[e] = fx2{0, 0};
    if (jz <= nz || jz >= N - nz) a[e] = fx_load<double>(raw[e], S1);
  }
  const int So = S - 2;  // one pass at quarter scale
  const bool nan = fx_nan<double>(So, emax == In::kExpMax);
  double2* dst = Zb + (((size_t)c * win.planes + plane - win.first) * (d.nx + 1) + cx) * N;
  rfft<E, TPR, +1>(
      a, buf, t, tw,
      [&](int o, fx2 v) {
        if (active) dst[o] = fx_store<double>(v, So, nan);
      },
      [&] {
#pragma unroll
        for (int e = 0; e < E; ++e) a[e] = fx_shr(a[e], S1 - S);
      });
}

// The scale from the column's largest value leaves room for the growth of a
// white column; one whose spectrum is no larger than its peak (all modes in
// phase) loses the passes' quarters instead, 2 bits each.  Its later passes get
// them back by a shift between passes 1 and 2, where an FP64 transform would be
// the more accurate one without: from 256 points on, 384 excepted (relative
// error of the products of a coherent spectrum at 256, 512, 1024, 1536 points:
// FP64 transforms 2.6, 4.1, 2.8, 3.5e-16, without 2.8, 4.9, 8.4, 20e-16).
template <typename T> constexpr bool fx_zfwd_mid(int E, int TPR) {
  return std::is_same<T, double>::value && (E == 12 ? TPR > 32 : TPR >= 32);
}
template <typename T, int E, int TPR, int NC>
__global__ void __launch_bounds__(NC * TPR, fx_zminb<E, TPR, NC>()) k_zfwd_x(const double2* __restrict__ Pb,
                                                                       typename C2<T>::t* __restrict__ VV,
                                                                       const fx2* __restrict__ tw, Dims d, int plane0,
                                                                       FxWindow win) {
  using V2 = typename C2<T>::t;
  using Io = FxIo<double>;
  constexpr int N = E * TPR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  fx2* buf = reinterpret_cast<fx2*>(smem_raw) + (threadIdx.x / TPR) * rbuf_size<E, TPR>();
  const int t = threadIdx.x % TPR;
  const int p = blockIdx.z, plane = plane0 + blockIdx.y;
  const int nxp = d.nx + 1;
  const int ix = blockIdx.x * NC + (int)(threadIdx.x / TPR);
  const bool active = ix < nxp;
  const int nz = d.nz, nzt = d.nzt;
  const int cx = active ? ix : 0;
  const double2* src = Pb + (((size_t)p * win.planes + plane - win.first) * nxp + cx) * N;
  double2 raw[E];
  int emax = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    raw[e] = active ? ldg_v(src + t + TPR * e) : make_double2(0.0, 0.0);
    emax = max(emax, max(Io::expo(raw[e].x), Io::expo(raw[e].y)));
  }
  emax = group_reduce<kRedMax, TPR>(emax, buf, t);
  // |re|, |im| < 2^(emax - bias + 1)
  constexpr bool MID = fx_zfwd_mid<T>(E, TPR);
  constexpr int kIn = MID ? fx_bits(fx_growth_first(E), 62) : fx_forward_bits(E, TPR, 62);
  constexpr int kQuarters = fx_quarters(E, TPR);
  const int S = emax == 0 ? 0 : fx_cap<T>(kIn - (emax - Io::kBias + 1), kQuarters);
  fx2 a[E];
#pragma unroll
  for (int e = 0; e < E; ++e) a[e] = fx_load<double>(raw[e], S);
  int So = S - 2 * kQuarters;
  V2* dst = VV + (((size_t)p * d.nplanes + plane) * nxp + cx) * nzt + nz;
  rfft<E, TPR, -1>(
      a, buf, t, tw,
      [&](int o, fx2 v) {
        if (!active) return;
        const bool nan = fx_nan<T>(So, emax == Io::kExpMax);
        if (o <= nz) dst[o] = fx_store<T>(v, So, nan);
        else if (o >= N - nz) dst[o - N] = fx_store<T>(v, So, nan);
      },
      [&] {
        if constexpr (MID)
          So += fx_renormalise<E, TPR, fx_bits(fx_growth(E, TPR, false), 62)>(a, FxIo<T>::kSMax - So, buf, t);
      });
}

// Row layout in shared memory: u and v in physical space (M each), then the
// padded exchange buffer X (M + TPR), which first holds the row's w spectrum.
// w stays in registers: the last pass leaves each thread exactly the elements
// the products' forward transforms start from.  TAU: the closure's stresses
// tau[p][plane][jz][x] (FP32, x pairs packed like the transform) are added to
// the products at the smaller of the two scales (the step's x rows at 47x96x47
// 0.76 ms with them, 0.33 without, 3.3 through the FP64-pipe rows).
template <int E, int TPR, int NR, int MINB, bool TAU>
__global__ void __launch_bounds__(NR * TPR, MINB) k_xrow_x(const double2* __restrict__ Zb,
                                                           double2* __restrict__ Pb,
                                                           const fx2* __restrict__ tw, const fx2* __restrict__ twh,
                                                           Dims d, FxFactor fac, int plane0, int compute_cfl,
                                                           const double* __restrict__ rdy, DevScalars* sc,
                                                           const float2* __restrict__ tau) {
  using V2 = double2;
  static_assert(sizeof(V2) == sizeof(fx2), "rows are converted in place");
  constexpr int M = E * TPR;
  constexpr int RS = fx_row_stride<M, TPR>(NR);
  constexpr int NT = NR * TPR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V2* S = reinterpret_cast<V2*>(smem_raw);
  fx2* Sf = reinterpret_cast<fx2*>(smem_raw);
  const int row = threadIdx.x / TPR, t = threadIdx.x % TPR;
  fx2* U = Sf + row * RS;
  fx2* X = U + 2 * M;  // the exchange buffer
  __shared__ int red[TPR > 32 ? NR * (TPR / 32) : 1];
  int* scratch = red + (TPR > 32 ? row * (TPR / 32) : 0);
  const int nx = d.nx, nxp = nx + 1, nzd = d.nzd;
  const int plane = plane0 + blockIdx.y;
  const int jz0 = blockIdx.x * NR;
  const int nrow = min(NR, nzd - jz0);
  // the block's rows of the three spectra (zTOx): NR consecutive jz per kx, w
  // into X
  for (int c = 0; c < 3; ++c) {
    const V2* src = Zb + ((size_t)c * d.nplanes + plane) * nxp * nzd + jz0;
    for (int i = threadIdx.x; i < nxp * NR; i += NT) {
      const int r = i % NR, k = i / NR;
      V2 v = make_double2(0.0, 0.0);
      if (r < nrow) v = ldg_v(src + (size_t)k * nzd + r);
      S[r * RS + c * M + k] = v;
    }
  }
  __syncthreads();
  int su = 0, sv = 0, sw = 0;  // scales of u, v, w in physical space
  int bad = 0;                 // bit c: component c of this row is not finite
  fx2 w[E];                    // w in physical space, w[e] at x pair t + TPR e
  // w first: its spectrum sits in the exchange buffer
#pragma unroll 1
  for (int cc = 0; cc < 3; ++cc) {
    const int c = cc == 0 ? 2 : cc - 1;
    fx2* F = U + c * M;
    fx2 a[E];
    const int sc = fx_inverse_row<E, TPR>(a, F, X, t, nx, tw, twh, scratch, bad, 1 << c);
    if (c == 0) su = sc;
    else if (c == 1) sv = sc;
    else sw = sc;
    if (cc == 0) {
#pragma unroll
      for (int e = 0; e < E; ++e) w[e] = a[e];
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) F[t + TPR * e] = a[e];
    }
  }
  // each thread reads back only its own physical values
  auto val = [&](int c, int e) -> fx2 {
    return c == 2 ? w[e] : U[c * M + t + TPR * e];
  };
  // CFL (dnsdata.f90:552-556) over the physical values of this row, in FP64
  if (compute_cfl) {
    double cfl = 0.0;
    bool inf = false;
    if (plane >= 2 && plane <= d.ny && row < nrow) {
      double r[3] = {d.rdx, rdy[plane], d.rdz};
      const int s3[3] = {su, sv, sw};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        inf = inf || ((bad >> c) & 1);
        const int s = max(-2000, min(-s3[c], 2000)), s1 = s >> 1;  // a velocity below 2^-960 may count as zero
        r[c] = r[c] * FxIo<double>::pow2(s1) * FxIo<double>::pow2(s - s1);
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const fx2 u = val(0, e), v = val(1, e), ww = val(2, e);
        auto mag = [](long long x) { return __ll2double_rn(x < 0 ? -x : x); };
        cfl = fmax(cfl, fma(mag(ww.x), r[2], fma(mag(v.x), r[1], mag(u.x) * r[0])));
        cfl = fmax(cfl, fma(mag(ww.y), r[2], fma(mag(v.y), r[1], mag(u.y) * r[0])));
      }
    }
    if (inf) cfl = (double)INFINITY;  // a non-finite velocity shows up as an infinite CFL
    xblock_max_atomic(cfl, &sc->cfl);
  }
  // products (dnsdata.f90:581-584), those with w first (w then dies): ww,
  // vw, uw, uu, vv, uv -> Pb slots 2, 4, 5, 0, 1, 3.  Factors below 2^60: the
  // products are below 2^56
#pragma unroll 1
  for (int q = 0; q < 6; ++q) {
    const int p = q == 0 ? 2 : q == 1 ? 4 : q == 2 ? 5 : q == 3 ? 0 : q == 4 ? 1 : 3;
    // factors of product p (uu, vv, ww, uv, vw, uw)
    const int fa = p < 3 ? p : (p == 5 ? 0 : p - 3);
    const int fb = p < 3 ? p : (p == 3 ? 1 : 2);
    fx2 a[E];
    if (q < 3) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const fx2 y = w[e], x = q == 0 ? y : U[fa * M + t + TPR * e];
        a[e] = fx2{fx_mul(x.x, y.x), fx_mul(x.y, y.y)};
      }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const fx2 x = U[fa * M + t + TPR * e], y = U[fb * M + t + TPR * e];
        a[e] = fx2{fx_mul(x.x, y.x), fx_mul(x.y, y.y)};
      }
    }
    const int sa = fa == 0 ? su : (fa == 1 ? sv : sw), sb = fb == 0 ? su : (fb == 1 ? sv : sw);
    bool nf = ((bad >> fa) | (bad >> fb)) & 1;
    int sp = sa + sb - 64;
    if constexpr (TAU) {
      const float2* tp = tau + (((size_t)p * d.nplanes + plane) * nzd + jz0 + row) * M + t;
      const bool inf = fx_add_f32<E, TPR>(a, sp, tp, row < nrow, t, scratch);
      nf = nf || inf;
    }
    fx_forward_row<E, TPR>(a, X, t, nx, tw, twh, fac, sp, nf, scratch);
    __syncthreads();
    // xTOz: the block's rows of product p, NR consecutive jz per kx
    V2* dst = Pb + ((size_t)p * d.nplanes + plane) * nxp * nzd + jz0;
    for (int i = threadIdx.x; i < nxp * NR; i += NT) {
      const int r = i % NR, k = i / NR;
      if (r < nrow) dst[(size_t)k * nzd + r] = S[r * RS + 2 * M + k];
    }
    __syncthreads();
  }
}

// The convective term of the budget spectra on one plane row jz (tke.cu):
// N_i = sum_k u_k g_ik of the fields Zt[f][plane of the chunk][kx][jz] (u_k:
// f = k, g_ik = du_i/dx_k: f = 3 + 3i + k), transformed forward with `factor`
// to Xt[i].  Row layout: u_k in physical space (M each), then the exchange
// buffer, where each g_ik is staged and transformed; N_i stays in registers,
// at the smallest scale of its terms.  Eight warps per SM (four slots a row)
// for 15 transforms a row, bound like k_xrow_x by issue and latency: 16.1 ->
// 3.4 ms per sample at 127x192x127 against the FP64-pipe row kernel.  N_i in a
// fifth slot instead would leave five warps.
template <int E, int TPR, int NR, int MINB>
__global__ void __launch_bounds__(NR * TPR, MINB) k_tke_x_x(const double2* __restrict__ Zt, double2* __restrict__ Xt,
                                                            const fx2* __restrict__ tw, const fx2* __restrict__ twh,
                                                            Dims d, FxFactor fac, int chunk) {
  constexpr int M = E * TPR;
  constexpr int RS = fx_row_stride<M, TPR, 4>(NR);
  constexpr int NT = NR * TPR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* S = reinterpret_cast<double2*>(smem_raw);
  const int row = threadIdx.x / TPR, t = threadIdx.x % TPR;
  fx2* U = reinterpret_cast<fx2*>(smem_raw) + row * RS;
  fx2* X = U + 3 * M;
  __shared__ int red[TPR > 32 ? NR * (TPR / 32) : 1];
  int* scratch = red + (TPR > 32 ? row * (TPR / 32) : 0);
  const int nx = d.nx, nxp = nx + 1, nzd = d.nzd;
  const int jz0 = blockIdx.x * NR;
  const int nrow = min(NR, nzd - jz0);
  // the block's rows of field f into slot c: NR consecutive jz per kx
  auto stage = [&](int f, int c) {
    const double2* src = Zt + ((size_t)f * chunk + blockIdx.y) * nxp * nzd + jz0;
    for (int i = threadIdx.x; i < nxp * NR; i += NT) {
      const int r = i % NR, k = i / NR;
      S[r * RS + c * M + k] = r < nrow ? ldg_v(src + (size_t)k * nzd + r) : make_double2(0.0, 0.0);
    }
  };
  for (int c = 0; c < 3; ++c) stage(c, c);
  __syncthreads();
  fx2 N[E];
  int su[3];
  int bad = 0;  // not finite: bit 0 a component of u, bit 1 + i a gradient of N_i
  int sn = kZeroRow;
  // step 0..2: u_k; then for each i the three g_ik
#pragma unroll 1
  for (int q = 0; q < 12; ++q) {
    const int i = q / 3 - 1, k = q % 3;
    fx2* F = i < 0 ? U + k * M : X;
    if (i >= 0) {
      __syncthreads();
      stage(3 + 3 * i + k, 3);
      __syncthreads();
    }
    fx2 a[E];
    const int sc = fx_inverse_row<E, TPR>(a, F, X, t, nx, tw, twh, scratch, bad, 1 << (i + 1));
    if (i < 0) {
      if (k == 0) su[0] = sc;
      else if (k == 1) su[1] = sc;
      else su[2] = sc;
#pragma unroll
      for (int e = 0; e < E; ++e) F[t + TPR * e] = a[e];
      continue;
    }
    // each thread reads back only its own physical values; products below
    // 2^56, their sum below 3 2^56
    if (k == 0) {
      sn = 2 * kZeroRow;
#pragma unroll
      for (int e = 0; e < E; ++e) N[e] = fx2{0, 0};
    }
    const int sp = sc + (k == 0 ? su[0] : k == 1 ? su[1] : su[2]) - 64, so = min(sn, sp);
    const int dn = min(sn - so, 62), dp = min(sp - so, 62);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const fx2 u = U[k * M + t + TPR * e];
      N[e] = fx_shr(N[e], dn) + fx_shr(fx2{fx_mul(a[e].x, u.x), fx_mul(a[e].y, u.y)}, dp);
    }
    sn = so;
    if (k == 2) {
      group_sync<TPR>();  // every read of the exchange buffer before it is written again
      fx_forward_row<E, TPR>(N, X, t, nx, tw, twh, fac, sn, (bad & (1 | 2 << i)) != 0, scratch);
      __syncthreads();
      double2* dst = Xt + ((size_t)i * chunk + blockIdx.y) * nxp * nzd + jz0;
      for (int j = threadIdx.x; j < nxp * NR; j += NT) {
        const int r = j % NR, kx = j / NR;
        if (r < nrow) dst[(size_t)kx * nzd + r] = S[r * RS + 3 * M + kx];
      }
    }
  }
}

namespace {

template <typename T, int N>
void fx_launch_z(const ConvLaunch& L, cudaStream_t s, int stage) {
  using V2 = typename C2<T>::t;
  constexpr int E = FxLen<N>::E, TPR = FxLen<N>::TPR, NC = fx_zcols<TPR>();
  const size_t sm = (size_t)NC * rbuf_size<E, TPR>() * sizeof(fx2);
  const Dims& d = L.d;
  if constexpr (std::is_same<T, double>::value) {
    if (stage == 0) {
      dim3 grid((L.ix_hi - L.ix_lo + NC - 1) / NC, L.nplanes, 3);
      k_zinv_x<E, TPR, NC><<<grid, NC * TPR, sm, s>>>(L.V, (double2*)L.Zb, (const fx2*)L.fx.z, d, L.plane0,
                                                      FxWindow{0, d.nplanes}, L.ix_lo, L.ix_hi);
    }
  }
  if (stage == 2) {
    dim3 grid((d.nx + 1 + NC - 1) / NC, L.nplanes, 6);
    k_zfwd_x<T, E, TPR, NC><<<grid, NC * TPR, sm, s>>>((const double2*)L.Pb, (V2*)L.VV, (const fx2*)L.fx.z, d,
                                                       L.plane0, FxWindow{0, d.nplanes});
  }
}

// TAU: with the closure's stresses L.tau
template <int M, bool TAU>
void fx_launch_x(const ConvLaunch& L, cudaStream_t s) {
  constexpr int E = FxLen<M>::E, TPR = FxLen<M>::TPR;
  constexpr int NR = fx_xrows<M, TPR>(), MINB = fx_xminb<M, TPR>();
  const size_t sm = (size_t)NR * fx_row_stride<M, TPR>(NR) * sizeof(fx2);
  const Dims& d = L.d;
  dim3 grid((d.nzd + NR - 1) / NR, L.nplanes);
  k_xrow_x<E, TPR, NR, MINB, TAU><<<grid, NR * TPR, sm, s>>>((const double2*)L.Zb, (double2*)L.Pb,
                                                             (const fx2*)L.fx.x, (const fx2*)L.fx.pack, d, L.fx.fac,
                                                             L.plane0, L.compute_cfl, L.rdy, L.sc, L.tau);
}

// z transforms of the budget spectra: 12 fields to a chunk, 3 back from it
template <int N>
void fx_launch_tke_z(const TkeLaunch& L, int p0, int planes, bool inverse, cudaStream_t s) {
  constexpr int E = FxLen<N>::E, TPR = FxLen<N>::TPR, NC = fx_zcols<TPR>();
  const size_t sm = (size_t)NC * rbuf_size<E, TPR>() * sizeof(fx2);
  const int nxp = L.d.nx + 1;
  const dim3 grid((nxp + NC - 1) / NC, planes, inverse ? 12 : 3);
  const FxWindow win{p0, L.chunk};
  if (inverse)
    k_zinv_x<E, TPR, NC><<<grid, NC * TPR, sm, s>>>(L.W, L.Zt, (const fx2*)L.fx.z, L.d, p0, win, 0, nxp);
  else
    k_zfwd_x<double, E, TPR, NC><<<grid, NC * TPR, sm, s>>>(L.Xt, L.N3, (const fx2*)L.fx.z, L.d, p0, win);
}
template <int M>
void fx_launch_tke_x(const TkeLaunch& L, int planes, cudaStream_t s) {
  constexpr int E = FxLen<M>::E, TPR = FxLen<M>::TPR;
  constexpr int NR = fx_xrows<M, TPR, 4>(), MINB = fx_xminb<M, TPR, 4>();
  const size_t sm = (size_t)NR * fx_row_stride<M, TPR, 4>(NR) * sizeof(fx2);
  const dim3 grid((L.d.nzd + NR - 1) / NR, planes);
  k_tke_x_x<E, TPR, NR, MINB><<<grid, NR * TPR, sm, s>>>(L.Zt, L.Xt, (const fx2*)L.fx.x, (const fx2*)L.fx.pack, L.d,
                                                         L.fx.fac, L.chunk);
}

template <typename K> cudaError_t fx_allow_smem(K* kernel, size_t bytes, bool max_carveout = false) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && max_carveout)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  return e;
}
// shared-memory limits of one length's kernels
template <typename T, int N> cudaError_t fx_limits_z() {
  constexpr int E = FxLen<N>::E, TPR = FxLen<N>::TPR, NC = fx_zcols<TPR>();
  const size_t sm = (size_t)NC * rbuf_size<E, TPR>() * sizeof(fx2);
  cudaError_t e = std::is_same<T, double>::value ? fx_allow_smem(k_zinv_x<E, TPR, NC>, sm) : cudaSuccess;
  return e == cudaSuccess ? fx_allow_smem(k_zfwd_x<T, E, TPR, NC>, sm) : e;
}
template <int M, bool TAU> cudaError_t fx_limits_x() {
  constexpr int E = FxLen<M>::E, TPR = FxLen<M>::TPR;
  constexpr int NR = fx_xrows<M, TPR>(), MINB = fx_xminb<M, TPR>();
  return fx_allow_smem(k_xrow_x<E, TPR, NR, MINB, TAU>, (size_t)NR * fx_row_stride<M, TPR>(NR) * sizeof(fx2), true);
}
template <int M> cudaError_t fx_limits_tke_x() {
  constexpr int E = FxLen<M>::E, TPR = FxLen<M>::TPR;
  constexpr int NR = fx_xrows<M, TPR, 4>(), MINB = fx_xminb<M, TPR, 4>();
  return fx_allow_smem(k_tke_x_x<E, TPR, NR, MINB>, (size_t)NR * fx_row_stride<M, TPR, 4>(NR) * sizeof(fx2), true);
}

}  // namespace

}  // namespace chgpu
