// 64-bit fixed-point arithmetic of the FP64 and double-float transforms.
//
// GB300 does 2 FP64 fused multiply-adds per SM and clock, but 72 integer
// multiply-adds 32x32+64 -> 64 bits (one instruction of the heavy FMA pipe)
// and 63 64-bit additions (measured).  A radix-2 butterfly costs 6 FP64
// instructions (3 clocks of an SM) or, on integers with 62 significant bits,
// 12 of those multiply-adds and about as many additions (0.2 clocks each).  So the
// transforms hold their data as block fixed point: every column or row of a
// transform has one power-of-two scale S, an element x is the 64-bit integer
// F = x 2^S, and S is chosen from the data so that no intermediate value of
// the transform can overflow (fx_scale_sum, fx_forward_bits).  In and out are FP64
// (or double-float) values.  Bits held between them: the z-inverse 62 of the sum
// of a column's moduli; the x rows 57 of a row's largest mode, 60 of its largest
// physical value, 56 of the largest product two rows allow; the z-forward 56 to
// 58 of a column's largest value; the forward passes scale by a quarter each
// (2 bits), shifted back up between passes 1 and 2 in the x rows and in the long
// z-forward ones.  In all that leaves an error below an FP64 transform's (white
// and falling spectra 0.8 to 3.4e-16, FP64 transforms 2.5 to 6.1e-16, up to 1536
// points; spectra in phase, at the bounds of the headroom, 1.3 to 3.9e-16, 2.2
// to 4.4e-16: tests/test_gpu_fixed_point.py and test_gpu_fixed_point_range.py).
//
// A product a W / 2^64 of 64-bit integers is formed from balanced 32-bit
// halves (a = ah 2^32 + al, |al| <= 2^31): ah wh + (ah wl + al wh + 2^31) >> 32;
// the dropped al wl is at most a quarter unit and has no bias.
#pragma once

#include <cuda_runtime.h>

#include "cplx.cuh"

namespace chgpu {

struct __align__(16) fx2 {
  long long x, y;
};
__device__ __forceinline__ fx2 operator+(fx2 a, fx2 b) { return fx2{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ fx2 operator-(fx2 a, fx2 b) { return fx2{a.x - b.x, a.y - b.y}; }

// The 32-bit halves of a register pair.  Through mov.b64, because a 64-bit
// shift and truncation make the compiler see a 64x64-bit product in
// (long long)fx_hi(a) * w and form that (72 instructions per complex product
// where this takes 20).
__device__ __forceinline__ int fx_up(long long a) {
  int h;
  asm("{.reg .b32 t;\n\tmov.b64 {t,%0},%1;}" : "=r"(h) : "l"(a));
  return h;
}
__device__ __forceinline__ int fx_lo(long long a) {
  int l;
  asm("{.reg .b32 t;\n\tmov.b64 {%0,t},%1;}" : "=r"(l) : "l"(a));
  return l;
}
// balanced upper half: a = fx_hi(a) 2^32 + fx_lo(a) with fx_lo signed
__device__ __forceinline__ int fx_hi(long long a) { return fx_up(a) + (int)((unsigned)fx_lo(a) >> 31); }
// the same of a compile-time weight
__host__ __device__ constexpr int fx_chi(long long w) { return (int)((w >> 32) + ((w >> 31) & 1)); }
__host__ __device__ constexpr int fx_clo(long long w) { return (int)(unsigned)(unsigned long long)w; }
__device__ __forceinline__ long long fx_wide(int a, int b) { return (long long)a * b; }
// cross terms' upper half added to the product of the upper halves
__device__ __forceinline__ long long fx_fold(long long cross, long long acc) { return acc + (long long)fx_up(cross); }
constexpr long long kFxRound = 0x80000000ll;

// add + a W / 2^64, W = wh 2^32 + wl
__device__ __forceinline__ long long fx_mad(long long add, long long a, int wh, int wl) {
  const int ah = fx_hi(a), al = fx_lo(a);
  long long c = fx_wide(ah, wl) + kFxRound;
  c = fx_wide(al, wh) + c;
  return fx_fold(c, fx_wide(ah, wh) + add);
}
// a b / 2^64
__device__ __forceinline__ long long fx_mul(long long a, long long b) { return fx_mad(0, a, fx_hi(b), fx_lo(b)); }
// rounded a / 4
__device__ __forceinline__ long long fx_quarter(long long a) { return (a + 2) >> 2; }
__device__ __forceinline__ fx2 fx_quarter(fx2 a) { return fx2{fx_quarter(a.x), fx_quarter(a.y)}; }

// A twiddle of a table: (re hi, re lo, im hi, im lo) of w 2^62, the halves
// balanced.  A product with it is a quarter of the true one.  Forward
// transforms use it so: the two bits of headroom it frees per pass hold the
// pass's growth.  Backward ones, whose values are bounded by the l1 norm of
// their input (2^62), do so in their second pass and shift the factor left by
// two first in later ones (fx_cmul4, moduli up to 2^60).
struct __align__(16) fxw {
  int rh, rl, ih, il;
};
// a w / 4 (SIGN < 0) or a conj(w) / 4 (SIGN > 0)
template <int SIGN> __device__ __forceinline__ fx2 fx_cmul(fx2 a, fxw w) {
  const int xh = fx_hi(a.x), xl = fx_lo(a.x), yh = fx_hi(a.y), yl = fx_lo(a.y);
  const int nh = -w.ih, nl = -w.il;
  const int rh = SIGN < 0 ? nh : w.ih, rl = SIGN < 0 ? nl : w.il;  // multiplies y in the real part
  const int ih = SIGN < 0 ? w.ih : nh, il = SIGN < 0 ? w.il : nl;  // multiplies x in the imaginary part
  long long c = fx_wide(xh, w.rl) + kFxRound;
  c = fx_wide(xl, w.rh) + c;
  c = fx_wide(yh, rl) + c;
  c = fx_wide(yl, rh) + c;
  long long d = fx_wide(yh, w.rl) + kFxRound;
  d = fx_wide(yl, w.rh) + d;
  d = fx_wide(xh, il) + d;
  d = fx_wide(xl, ih) + d;
  return fx2{fx_fold(c, fx_wide(yh, rh) + fx_wide(xh, w.rh)), fx_fold(d, fx_wide(xh, ih) + fx_wide(yh, w.rh))};
}
__device__ __forceinline__ fx2 fx_shl2(fx2 a) { return fx2{a.x << 2, a.y << 2}; }
template <int SIGN> __device__ __forceinline__ fx2 fx_cmul4(fx2 a, fxw w) { return fx_cmul<SIGN>(fx_shl2(a), w); }
// rounded a / 2^n, 0 <= n < 63
__device__ __forceinline__ fx2 fx_shr(fx2 a, int n) {
  const long long h = (1ll << n) >> 1;
  return fx2{(a.x + h) >> n, (a.y + h) >> n};
}
__device__ __forceinline__ fxw fx_ldw(const fx2* p) {
  const int4 v = __ldg(reinterpret_cast<const int4*>(p));
  return fxw{v.x, v.y, v.z, v.w};
}
template <> __device__ __forceinline__ fx2 ldg_v<fx2>(const fx2* p) {
  const longlong2 v = __ldg(reinterpret_cast<const longlong2*>(p));
  return fx2{v.x, v.y};
}

// Constants of the register DFTs as c = c0 + w 2^-64 with c0 in {-1, 0, 1}
// and |w 2^-64| <= 1/2, so that c a = c0 a + (a w) / 2^64 at full scale;
// q = c 2^62 for the quarter-scale product.
struct FxC {
  int c0;
  long long w, q;
};
#define CHGPU_FX_CONST __host__ __device__ __forceinline__ constexpr
CHGPU_FX_CONST FxC fx_neg(FxC c) {
  // 1/2 = 1 - 2^63/2^64 and -1/2 = 0 - 2^63/2^64: 2^63 itself does not fit
  if (c.w == (-0x7fffffffffffffffll - 1)) return FxC{c.c0 == 1 ? 0 : 1, c.w, -c.q};
  return FxC{-c.c0, -c.w, -c.q};
}
// by value, so that device code holds immediates
CHGPU_FX_CONST FxC fx_sqrt3_2() { return FxC{1, -2471395088767036514ll, 3993837246235628775ll}; }
CHGPU_FX_CONST FxC fx_sqrt1_2() { return FxC{1, -5402926248376769404ll, 3260954456333195553ll}; }
// cos(15 e degrees) for 0 <= e <= 6
CHGPU_FX_CONST FxC fx_cos24_first(int e) {
  return e == 0   ? FxC{1, 0, 1ll << 62}
         : e == 1 ? FxC{1, -628557561968679382ll, 4454546627935218059ll}
         : e == 2 ? fx_sqrt3_2()
         : e == 3 ? fx_sqrt1_2()
         : e == 4 ? FxC{1, -0x7fffffffffffffffll - 1, 1ll << 61}
         : e == 5 ? FxC{0, 4774368686408090022ll, 1193592171602022505ll}
                  : FxC{0, 0, 0};
}
// cos(15 e degrees)
CHGPU_FX_CONST FxC fx_cos24(int e) {
  const int f = ((e % 24) + 24) % 24, g = f > 12 ? 24 - f : f;
  return g > 6 ? fx_neg(fx_cos24_first(12 - g)) : fx_cos24_first(g);
}
// N dividing 24
CHGPU_FX_CONST FxC fx_cosN(int N, int m) { return fx_cos24(m * (24 / N)); }
CHGPU_FX_CONST FxC fx_sinN(int N, int m) { return fx_cos24(m * (24 / N) - 6); }

// a (c + i s) at full scale, c and s compile-time constants
__device__ __forceinline__ fx2 fx_cmulc(fx2 a, FxC c, FxC s) {
  const FxC n = fx_neg(s);
  const int xh = fx_hi(a.x), xl = fx_lo(a.x), yh = fx_hi(a.y), yl = fx_lo(a.y);
  const int ch = fx_chi(c.w), cl = fx_clo(c.w), sh = fx_chi(s.w), sl = fx_clo(s.w), nh = fx_chi(n.w), nl = fx_clo(n.w);
  long long p = fx_wide(xh, cl) + kFxRound;
  p = fx_wide(xl, ch) + p;
  p = fx_wide(yh, nl) + p;
  p = fx_wide(yl, nh) + p;
  long long q = fx_wide(yh, cl) + kFxRound;
  q = fx_wide(yl, ch) + q;
  q = fx_wide(xh, sl) + q;
  q = fx_wide(xl, sh) + q;
  long long re = fx_wide(xh, ch) + fx_wide(yh, nh), im = fx_wide(yh, ch) + fx_wide(xh, sh);
  if (c.c0 == 1) { re += a.x; im += a.y; }
  if (c.c0 == -1) { re -= a.x; im -= a.y; }
  if (n.c0 == 1) re += a.y;
  if (n.c0 == -1) re -= a.y;
  if (s.c0 == 1) im += a.x;
  if (s.c0 == -1) im -= a.x;
  return fx2{fx_fold(p, re), fx_fold(q, im)};
}
// the same at quarter scale
__device__ __forceinline__ fx2 fx_cmulc_q(fx2 a, FxC c, FxC s) {
  return fx_cmul<-1>(a, fxw{fx_chi(c.q), fx_clo(c.q), fx_chi(s.q), fx_clo(s.q)});
}
// sqrt(1/2) (SR + i SI) a for signs SR, SI
template <int SR, int SI> __device__ __forceinline__ fx2 fx_mul_diag(fx2 a) {
  // (SR x - SI y, SI x + SR y)
  const long long p = (SR > 0 ? a.x : -a.x) - (SI > 0 ? a.y : -a.y), q = (SI > 0 ? a.x : -a.x) + (SR > 0 ? a.y : -a.y);
  constexpr int h = fx_chi(fx_sqrt1_2().w), l = fx_clo(fx_sqrt1_2().w);
  return fx2{fx_mad(p, p, h, l), fx_mad(q, q, h, l)};
}

// register DFTs (the splits of Dft<8> and DftComposite, cplx.cuh)
template <> struct Dft<3, fx2> {
  template <int SIGN> __device__ __forceinline__ static void run(fx2* a) {
    const fx2 t = a[1] + a[2], d = a[1] - a[2];
    const fx2 m = fx2{a[0].x - (t.x >> 1), a[0].y - (t.y >> 1)};
    constexpr int ch = fx_chi(fx_sqrt3_2().w), cl = fx_clo(fx_sqrt3_2().w);
    const fx2 h = fx2{fx_mad(d.x, d.x, ch, cl), fx_mad(d.y, d.y, ch, cl)};  // sqrt(3)/2 d
    a[0] = a[0] + t;
    const fx2 r = mul_is<SIGN>(h);
    a[1] = m + r;
    a[2] = m - r;
  }
};
template <> struct Dft<8, fx2> {
  template <int SIGN> __device__ __forceinline__ static void run(fx2* a) {
    dft4<SIGN>(a[0], a[2], a[4], a[6]);
    dft4<SIGN>(a[1], a[3], a[5], a[7]);
    a[3] = fx_mul_diag<1, SIGN>(a[3]);   // w8^1
    a[5] = mul_is<SIGN>(a[5]);           // w8^2
    a[7] = fx_mul_diag<-1, SIGN>(a[7]);  // w8^3
    fx2 y[8];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      y[k1] = a[2 * k1] + a[2 * k1 + 1];
      y[k1 + 4] = a[2 * k1] - a[2 * k1 + 1];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = y[k];
  }
};
// 3 P points as DFT3 over r1, twiddles w_{3P}^(r2 k1), DFT_P over r2
template <int P, int SIGN, bool QUARTER> __device__ __forceinline__ void fx_dft3p(fx2* a) {
  constexpr int N = 3 * P;
#pragma unroll
  for (int r2 = 0; r2 < P; ++r2) {
    fx2 b[3] = {a[r2], a[P + r2], a[2 * P + r2]};
    Dft<3, fx2>::template run<SIGN>(b);
    a[r2] = b[0];
    a[P + r2] = b[1];
    a[2 * P + r2] = b[2];
  }
  fx2 y[N];
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1) {
    fx2 c[P];
#pragma unroll
    for (int r2 = 0; r2 < P; ++r2) {
      fx2 v = a[k1 * P + r2];
      const int m = r2 * k1;
      if (m == 0) {
        if (QUARTER) v = fx_quarter(v);
      } else if (QUARTER) {
        v = fx_cmulc_q(v, fx_cosN(N, m), SIGN > 0 ? fx_sinN(N, m) : fx_neg(fx_sinN(N, m)));
      } else if (4 * m == N) {
        v = mul_is<SIGN>(v);
      } else {
        v = fx_cmulc(v, fx_cosN(N, m), SIGN > 0 ? fx_sinN(N, m) : fx_neg(fx_sinN(N, m)));
      }
      c[r2] = v;
    }
    Dft<P, fx2>::template run<SIGN>(c);
#pragma unroll
    for (int k2 = 0; k2 < P; ++k2) y[k1 + 3 * k2] = c[k2];
  }
#pragma unroll
  for (int k = 0; k < N; ++k) a[k] = y[k];
}
// First pass of a transform: forward transforms of 24 points per thread are
// scaled by a quarter inside, whose two bits let the input use the word's full
// width; backward ones run at full scale.
__host__ __device__ constexpr bool fx_first_quarter(int E, int SIGN) { return SIGN < 0 && E == 24; }
template <int E, int SIGN, bool QUARTER> __device__ __forceinline__ void fx_first(fx2* a) {
  if constexpr (E == 24) fx_dft3p<8, SIGN, QUARTER>(a);
  else if constexpr (E == 12) fx_dft3p<4, SIGN, false>(a);
  else Dft<E, fx2>::template run<SIGN>(a);
}

// ---------------------------------------------------------------------------
// scales
// ---------------------------------------------------------------------------
// What the kernels read and write: FP64 pairs; double-float pairs are written
// only.
template <typename T> struct FxIo;
template <> struct FxIo<double> {
  using V2 = double2;
  static constexpr int kBias = 1023, kExpMax = 2047;
  __device__ static int expo(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }
  // leading 19 significand bits, in units of 2^(expo - kBias - 18)
  __device__ static int lead(double v) { return ((__double2hiint(v) & 0xfffff) | 0x100000) >> 2; }
  // round(v 2^S); zero below one unit, and where v is below the normal range
  __device__ static long long in(double v, int S) {
    const int hi = __double2hiint(v), e = hi & 0x7ff00000, t = e + (S << 20);
    const double s = __hiloint2double((hi & (int)0x800fffff) | t, __double2loint(v));
    return (e != 0 && t >= 0x100000) ? __double2ll_rn(s) : 0ll;
  }
  __device__ static double out(long long f, int S) {
    const double d = __ll2double_rn(f);
    return f == 0 ? 0.0 : __hiloint2double(__double2hiint(d) - (S << 20), __double2loint(d));
  }
  static constexpr int kSMin = -961, kSMax = 1022;  // scales at which out() holds for |f| <= 2^62
  __device__ static double pow2(int s) { return __hiloint2double((1023 + s) << 20, 0); }  // -1022 <= s <= 1023
  // the same at any scale, rounded once: subnormal, zero and infinite too
  __device__ static double out_any(long long f, int S) {
    const int s = max(-2000, min(-S, 2000)), s1 = s >> 1;
    return __ll2double_rn(f) * pow2(s1) * pow2(s - s1);
  }
  __device__ static double nan() { return __longlong_as_double(0x7ff8000000000000ll); }
};
template <> struct FxIo<dd> {
  using V2 = cdd;
  __device__ static float pow2(int s) { return __int_as_float((127 + s) << 23); }  // -126 <= s <= 127
  __device__ static dd out(long long f, int S) {
    const float h = __ll2float_rn(f), l = __ll2float_rn(f - __float2ll_rn(h));
    const int s1 = (-S) >> 1;
    const float f1 = pow2(s1), f2 = pow2(-S - s1);
    return dd(h * f1 * f2, l * f1 * f2);
  }
  static constexpr int kSMin = -252, kSMax = 252;
  __device__ static dd nan() { return dd(__int_as_float(0x7fc00000), 0.f); }
};
// The z kernels hold data that would take a larger scale than kSMax (below
// 2^(bits - kSMax) throughout, zeros among them) at a smaller one, so that one unit
// of the result is at least the smallest normal number 2^-1022 (double-float:
// 2^-252, where every value rounds to zero).  NaN is written where the data are
// not finite, and at scales below kSMin, whose column's or row's bound exceeds
// the type's range: values within a factor 2^11 of overflow.
template <typename T> __device__ __forceinline__ int fx_cap(int S, int quarters) {
  return min(S, FxIo<T>::kSMax + 2 * quarters);
}
template <typename T> __device__ __forceinline__ bool fx_nan(int S, bool bad) { return bad || S < FxIo<T>::kSMin; }
template <typename T> __device__ __forceinline__ typename FxIo<T>::V2 fx_store(fx2 v, int S, bool nan) {
  using Io = FxIo<T>;
  typename Io::V2 r;
  if (nan) {
    r.x = Io::nan();
    r.y = r.x;
  } else {
    r.x = Io::out(v.x, S);
    r.y = Io::out(v.y, S);
  }
  return r;
}
// The x rows' (FP64), whose scale a product's two factors have set: any scale,
// NaN only for data that are not finite (-1).
constexpr int kNan = -1;
__device__ __forceinline__ double2 fx_store_any(fx2 v, int S, int mode) {  // mode 0: kSMin <= S <= kSMax; 1: another
  using Io = FxIo<double>;
  if (mode == 0) return make_double2(Io::out(v.x, S), Io::out(v.y, S));
  return mode == kNan ? make_double2(Io::nan(), Io::nan()) : make_double2(Io::out_any(v.x, S), Io::out_any(v.y, S));
}
template <typename T> __device__ __forceinline__ fx2 fx_load(typename FxIo<T>::V2 v, int S) {
  return fx2{FxIo<T>::in(v.x, S), FxIo<T>::in(v.y, S)};
}
// Largest scale with sum 2^S <= 2^bits.  emax: the largest exponent, B: the
// sum of the inputs' leading bits shifted to emax, plus one each (so
// B 2^(emax - bias - 18) is at least the sum of |re| + |im|).
template <typename T> __device__ __forceinline__ int fx_scale_sum(int emax, unsigned B, int bits) {
  return bits - (32 - __clz((int)B)) - (emax - FxIo<T>::kBias - 18);
}
template <typename T> __device__ __forceinline__ unsigned fx_lead_at(T v, int emax) {
  return (unsigned)(FxIo<T>::lead(v) >> min(emax - FxIo<T>::expo(v), 31)) + 1u;
}

}  // namespace chgpu
