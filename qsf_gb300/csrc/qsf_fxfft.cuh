// qsf_fxfft.cuh -- block-fixed-point (int64) arithmetic of the transforms for sm_103a.
//
// GB300 issues about 2 FP64 instructions per clock per SM but ~128 integer
// instructions, so the split step's FFTs run on the integer pipes: a line (or a group of
// lines) is held as 64-bit integers sharing one power-of-two block exponent,
// value = int * 2^-scale.  Additions are exact; products by twiddles and butterfly
// constants (62 fractional bits) keep the top 64 bits of the 124-bit product to within
// 1-2 units, from 32 x 32 -> 64-bit partial products.  After every radix pass the
// block is renormalised so that its largest component again uses all bits the next
// pass can afford (62 minus the pass's growth), i.e. block floating point with a 55-60
// bit mantissa at every pass.  Against an exact DFT this is ~3.5x more accurate than an
// FP64 FFT (normwise relative error ~6e-17 vs ~2.3e-16 at N = 48 .. 2048); FP64
// storage of psi is unchanged.  The transforms themselves are in qsf_lines.cuh.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "qsf_fft.cuh"

namespace qsf {

typedef long long i64;
typedef unsigned long long u64;

// a * w / 2^62 for w in 2^62 fixed point, from three signed 32 x 32 -> 64-bit partial
// products (IMAD.WIDE): both operands are split into a high word and a signed low
// word, x = xh 2^32 + xl with xl in [-2^31, 2^31); the low x low product (at most one
// unit of the result) is dropped and the middle terms are rounded, so the result lies
// within 1.5 units of the exact quotient.  Needs |a|, |w| < 2^62.5.
__device__ __forceinline__ i64 mulq62(i64 a, i64 w) {
  const int al = (int)a, wl = (int)w;
  const int ah = (int)((a - (i64)al) >> 32), wh = (int)((w - (i64)wl) >> 32);
  const i64 mid = (i64)ah * wl + (i64)al * wh + (1LL << 29);
  return (i64)(((u64)((i64)ah * wh) << 2) + (u64)(mid >> 30));
}

__device__ __forceinline__ longlong2 fadd(longlong2 a, longlong2 b) { return make_longlong2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ longlong2 fsub(longlong2 a, longlong2 b) { return make_longlong2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ longlong2 fconj(longlong2 a) { return make_longlong2(a.x, -a.y); }
// a * w with w in 2^62 fixed point (|w| <= 1, components of a below 2^62): three
// rounded products (Gauss / Karatsuba): re = c(a+b) - b(c+d), im = c(a+b) + a(d-c)
__device__ __forceinline__ longlong2 fmul62(longlong2 a, longlong2 w) {
  const i64 k1 = mulq62(a.x + a.y, w.x);
  const i64 k2 = mulq62(a.x, w.y - w.x);
  const i64 k3 = mulq62(a.y, w.x + w.y);
  return make_longlong2(k1 - k3, k1 + k2);
}
// Twiddle products from pre-split tables.  A twiddle w in 2^62
// fixed point is stored as the signed 32-bit halves of each component, w = wh 2^32 + wl
// with wl = (int)w (int4 {re lo, re hi, im lo, im hi}; the host keeps every low half
// away from -2^31 so that it can be negated).  The complex product a * w / 2^64 takes
// the four high x high products exactly, sums the eight middle products of each output
// component in one 64-bit word (rounded at bit 32) and drops the four low x low ones:
// within 1 unit of the exact quotient, from twelve 32 x 32 -> 64-bit multiply-adds and
// no 64-bit shifts.  Callers pre-scale a by 4 (components below 2^61), so the product
// comes out at the scale of an untwiddled element.
// the high half of the signed split x = hi 2^32 + (int)x
__device__ __forceinline__ int split_hi(i64 x) { return (int)(x >> 32) + (int)((unsigned)x >> 31); }
__device__ __forceinline__ longlong2 fmul_tw(longlong2 a, int4 w) {
  const int axl = (int)a.x, axh = split_hi(a.x), ayl = (int)a.y, ayh = split_hi(a.y);
  const int nyl = -w.z, nyh = -w.w;
  i64 rm = (1LL << 31), im = (1LL << 31);
  rm += (i64)axh * w.x;
  rm += (i64)axl * w.y;
  rm += (i64)ayh * nyl;
  rm += (i64)ayl * nyh;
  im += (i64)axh * w.z;
  im += (i64)axl * w.w;
  im += (i64)ayh * w.x;
  im += (i64)ayl * w.y;
  i64 re = rm >> 32, ii = im >> 32;
  re += (i64)axh * w.y;
  re += (i64)ayh * nyh;
  ii += (i64)axh * w.w;
  ii += (i64)ayh * w.y;
  return make_longlong2(re, ii);
}
// the signed 32-bit halves of a compile-time 64-bit constant
__host__ __device__ constexpr int k_lo(i64 c) {
  return (int)((c & 0xffffffffLL) >= 0x80000000LL ? (c & 0xffffffffLL) - 0x100000000LL : (c & 0xffffffffLL));
}
__host__ __device__ constexpr int k_hi(i64 c) { return (int)((c - (i64)k_lo(c)) >> 32); }
// a * C / 2^64 for a compile-time C (|C| < 2^63, |a| < 2^62): three multiply-adds,
// within 0.75 units
template <i64 C>
__device__ __forceinline__ i64 mulk64(i64 a) {
  constexpr int cl = k_lo(C), ch = k_hi(C);
  const int al = (int)a, ah = split_hi(a);
  const i64 m = (i64)ah * cl + (i64)al * ch + (1LL << 31);
  return (m >> 32) + (i64)ah * ch;
}
// a * c for a constant c = C / 2^63 (|c| < 1): within 1.5 units
template <i64 C>
__device__ __forceinline__ i64 mulk63(i64 a) { return (i64)((u64)mulk64<C>(a) << 1); }
// a * (CR + i CI) / 2^63 for compile-time constants: the complex form of mulk64 (merged
// middle words), doubled; within 2 units per component
template <i64 CR, i64 CI>
__device__ __forceinline__ longlong2 fmulk63(longlong2 a) {
  constexpr int rl = k_lo(CR), rh = k_hi(CR), il = k_lo(CI), ih = k_hi(CI), nl = k_lo(-CI), nh = k_hi(-CI);
  const int axl = (int)a.x, axh = split_hi(a.x), ayl = (int)a.y, ayh = split_hi(a.y);
  i64 rm = (1LL << 31), im = (1LL << 31);
  rm += (i64)axh * rl;
  rm += (i64)axl * rh;
  rm += (i64)ayh * nl;
  rm += (i64)ayl * nh;
  im += (i64)axh * il;
  im += (i64)axl * ih;
  im += (i64)ayh * rl;
  im += (i64)ayl * rh;
  i64 re = rm >> 32, ii = im >> 32;
  re += (i64)axh * rh;
  re += (i64)ayh * nh;
  ii += (i64)axh * ih;
  ii += (i64)ayh * rh;
  return make_longlong2((i64)((u64)re << 1), (i64)((u64)ii << 1));
}
// butterfly constants in 2^63 fixed point (|c| < 1)
#define QSF_K63_SQRT1_2 6521908912666391106LL   /* round(2^63 / sqrt(2)) */
#define QSF_K63_C16_1 8521284645587064995LL     /* round(2^63 cos(pi/8)) */
#define QSF_K63_S16_1 3529631669043774883LL     /* round(2^63 sin(pi/8)) */
#define QSF_K63_SQRT3_2 7987674492471257551LL   /* round(2^63 sqrt(3)/2) */
#define QSF_K63_C5_1 2850178704830799621LL      /* round(2^63 cos(2pi/5)) */
#define QSF_K63_C5_2 (-7461864723258187525LL)   /* round(2^63 cos(4pi/5)) */
#define QSF_K63_S5_1 8771948077865237882LL      /* round(2^63 sin(2pi/5)) */
#define QSF_K63_S5_2 5421362059670026167LL      /* round(2^63 sin(4pi/5)) */

// OR of the component magnitudes (x ^ (x >> 63) is |x| or |x| - 1): its bit length is
// the block maximum's bit length, or one less when that maximum is a negative power of two
__device__ __forceinline__ u64 fmag(longlong2 x) { return (u64)(x.x ^ (x.x >> 63)) | (u64)(x.y ^ (x.y >> 63)); }
__device__ __forceinline__ int bitlen(u64 v) { return 64 - __clzll((long long)v); }
template <bool FWD> __device__ __forceinline__ longlong2 fmul_si(longlong2 a) {
  return FWD ? make_longlong2(a.y, -a.x) : make_longlong2(-a.y, a.x);
}

template <bool FWD> __device__ __forceinline__ void fbfly2(longlong2& a, longlong2& b) {
  const longlong2 t = a;
  a = fadd(t, b);
  b = fsub(t, b);
}
template <bool FWD>
__device__ __forceinline__ void fbfly4(longlong2& x0, longlong2& x1, longlong2& x2, longlong2& x3) {
  const longlong2 t0 = fadd(x0, x2), t1 = fsub(x0, x2), t2 = fadd(x1, x3), t3 = fmul_si<FWD>(fsub(x1, x3));
  x0 = fadd(t0, t2);
  x2 = fsub(t0, t2);
  x1 = fadd(t1, t3);
  x3 = fsub(t1, t3);
}
// w8^1 * a and w8^3 * a, w8 = exp(sign 2 pi i / 8)
__device__ __forceinline__ i64 mul_sqrt1_2(i64 a) { return mulk63<QSF_K63_SQRT1_2>(a); }
template <bool FWD> __device__ __forceinline__ longlong2 fw8_1(longlong2 a) {
  return FWD ? make_longlong2(mul_sqrt1_2(a.x + a.y), mul_sqrt1_2(a.y - a.x))
             : make_longlong2(mul_sqrt1_2(a.x - a.y), mul_sqrt1_2(a.x + a.y));
}
template <bool FWD> __device__ __forceinline__ longlong2 fw8_3(longlong2 a) {
  return FWD ? make_longlong2(mul_sqrt1_2(a.y - a.x), -mul_sqrt1_2(a.x + a.y))
             : make_longlong2(-mul_sqrt1_2(a.x + a.y), mul_sqrt1_2(a.x - a.y));
}
template <bool FWD> __device__ __forceinline__ void fbfly8(longlong2* v) {
  longlong2 a0 = fadd(v[0], v[4]), a4 = fsub(v[0], v[4]);
  longlong2 a1 = fadd(v[1], v[5]), a5 = fsub(v[1], v[5]);
  longlong2 a2 = fadd(v[2], v[6]), a6 = fsub(v[2], v[6]);
  longlong2 a3 = fadd(v[3], v[7]), a7 = fsub(v[3], v[7]);
  a5 = fw8_1<FWD>(a5);
  a6 = fmul_si<FWD>(a6);
  a7 = fw8_3<FWD>(a7);
  fbfly4<FWD>(a0, a1, a2, a3);
  fbfly4<FWD>(a4, a5, a6, a7);
  v[0] = a0; v[4] = a2; v[2] = a1; v[6] = a3;
  v[1] = a4; v[5] = a6; v[3] = a5; v[7] = a7;
}
template <bool FWD> __device__ __forceinline__ void fbfly3(longlong2* v) {
  const longlong2 t1 = fadd(v[1], v[2]), t2 = fsub(v[1], v[2]);
  // m1 = v0 - t1/2 ; X1 = m1 + i k t2, X2 = m1 - i k t2, k = sign * sqrt(3)/2
  const longlong2 m1 = make_longlong2(v[0].x - ((t1.x + 1) >> 1), v[0].y - ((t1.y + 1) >> 1));
  const i64 kx = mulk63<QSF_K63_SQRT3_2>(t2.x), ky = mulk63<QSF_K63_SQRT3_2>(t2.y);
  v[0] = fadd(v[0], t1);
  if (FWD) {  // k = -sqrt3/2
    v[1] = make_longlong2(m1.x + ky, m1.y - kx);
    v[2] = make_longlong2(m1.x - ky, m1.y + kx);
  } else {
    v[1] = make_longlong2(m1.x - ky, m1.y + kx);
    v[2] = make_longlong2(m1.x + ky, m1.y - kx);
  }
}
template <bool FWD> __device__ __forceinline__ void fbfly5(longlong2* v) {
  const longlong2 t1 = fadd(v[1], v[4]), t2 = fadd(v[2], v[3]), t3 = fsub(v[1], v[4]), t4 = fsub(v[2], v[3]);
  const longlong2 x0 = v[0];
#define QSF_M5(x, K) mulk63<QSF_K63_##K>(x)
  const longlong2 a1 = make_longlong2(x0.x + QSF_M5(t1.x, C5_1) + QSF_M5(t2.x, C5_2),
                                      x0.y + QSF_M5(t1.y, C5_1) + QSF_M5(t2.y, C5_2));
  const longlong2 a2 = make_longlong2(x0.x + QSF_M5(t1.x, C5_2) + QSF_M5(t2.x, C5_1),
                                      x0.y + QSF_M5(t1.y, C5_2) + QSF_M5(t2.y, C5_1));
  // b1 = s1 t3 + s2 t4, b2 = s2 t3 - s1 t4 with s = sign * sin
  longlong2 b1 = make_longlong2(QSF_M5(t3.x, S5_1) + QSF_M5(t4.x, S5_2), QSF_M5(t3.y, S5_1) + QSF_M5(t4.y, S5_2));
  longlong2 b2 = make_longlong2(QSF_M5(t3.x, S5_2) - QSF_M5(t4.x, S5_1), QSF_M5(t3.y, S5_2) - QSF_M5(t4.y, S5_1));
#undef QSF_M5
  if (FWD) {
    b1 = make_longlong2(-b1.x, -b1.y);
    b2 = make_longlong2(-b2.x, -b2.y);
  }
  v[0] = make_longlong2(x0.x + t1.x + t2.x, x0.y + t1.y + t2.y);
  v[1] = make_longlong2(a1.x - b1.y, a1.y + b1.x);
  v[4] = make_longlong2(a1.x + b1.y, a1.y - b1.x);
  v[2] = make_longlong2(a2.x - b2.y, a2.y + b2.x);
  v[3] = make_longlong2(a2.x + b2.y, a2.y - b2.x);
}
template <bool FWD> __device__ __forceinline__ void fbfly16(longlong2* v) {
  longlong2 a[16];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    longlong2 x0 = v[r], x1 = v[r + 4], x2 = v[r + 8], x3 = v[r + 12];
    fbfly4<FWD>(x0, x1, x2, x3);
    a[r * 4 + 0] = x0;
    a[r * 4 + 1] = x1;
    a[r * 4 + 2] = x2;
    a[r * 4 + 3] = x3;
  }
  constexpr i64 sg = FWD ? -1 : 1;
  a[1 * 4 + 1] = fmulk63<QSF_K63_C16_1, sg * QSF_K63_S16_1>(a[1 * 4 + 1]);     // w^1
  a[1 * 4 + 3] = fmulk63<QSF_K63_S16_1, sg * QSF_K63_C16_1>(a[1 * 4 + 3]);     // w^3
  a[3 * 4 + 1] = fmulk63<QSF_K63_S16_1, sg * QSF_K63_C16_1>(a[3 * 4 + 1]);     // w^3
  a[3 * 4 + 3] = fmulk63<-QSF_K63_C16_1, -sg * QSF_K63_S16_1>(a[3 * 4 + 3]);   // w^9
  a[1 * 4 + 2] = fw8_1<FWD>(a[1 * 4 + 2]);                              // w^2
  a[2 * 4 + 1] = fw8_1<FWD>(a[2 * 4 + 1]);                              // w^2
  a[2 * 4 + 2] = fmul_si<FWD>(a[2 * 4 + 2]);                            // w^4
  a[2 * 4 + 3] = fw8_3<FWD>(a[2 * 4 + 3]);                              // w^6
  a[3 * 4 + 2] = fw8_3<FWD>(a[3 * 4 + 2]);                              // w^6
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    longlong2 x0 = a[0 * 4 + k1], x1 = a[1 * 4 + k1], x2 = a[2 * 4 + k1], x3 = a[3 * 4 + k1];
    fbfly4<FWD>(x0, x1, x2, x3);
    v[k1 + 0] = x0;
    v[k1 + 4] = x1;
    v[k1 + 8] = x2;
    v[k1 + 12] = x3;
  }
}
template <int R, bool FWD> __device__ __forceinline__ void fbfly(longlong2* v) {
  if constexpr (R == 2) fbfly2<FWD>(v[0], v[1]);
  else if constexpr (R == 3) fbfly3<FWD>(v);
  else if constexpr (R == 4) fbfly4<FWD>(v[0], v[1], v[2], v[3]);
  else if constexpr (R == 5) fbfly5<FWD>(v);
  else if constexpr (R == 8) fbfly8<FWD>(v);
  else if constexpr (R == 16) fbfly16<FWD>(v);
}

// a pre-split twiddle back in one 64-bit word per component
__device__ __forceinline__ longlong2 tw_join(int4 w) {
  return make_longlong2((i64)((u64)(i64)w.y << 32) + (i64)w.x, (i64)((u64)(i64)w.w << 32) + (i64)w.z);
}

// Exponent bits of a double's magnitude (0 for 0 / denormals)
__device__ __forceinline__ int dexp(double x) { return (int)((__double_as_longlong(x) >> 52) & 0x7ff); }

// round(x * 2^s) as int64 using integer operations only (x finite, result < 2^63)
__device__ __forceinline__ i64 d2fx(double x, int s) {
  const u64 b = (u64)__double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ff);
  if (e == 0) return 0;  // zero or denormal: below any representable fixed-point step here
  const u64 m = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const int sh = e - 1075 + s;  // x * 2^s = m * 2^sh
  i64 r;
  if (sh >= 0) r = (i64)(m << sh);
  else if (sh <= -64) r = 0;
  else r = (i64)((m + (1ull << (-sh - 1))) >> (-sh));
  return (b >> 63) ? -r : r;
}
// x * 2^-s as a double (round to nearest even), integer operations only
__device__ __forceinline__ double fx2d(i64 x, int s) {
  if (x == 0) return 0.0;
  const u64 sign = x < 0 ? 0x8000000000000000ull : 0ull;
  u64 a = (u64)(x < 0 ? -x : x);
  const int lz = __clzll((long long)a);
  a <<= lz;  // top bit set: value = a * 2^(63 - lz - 63)
  u64 mant = a >> 11;
  const u64 rem = a & 0x7ffull;
  int e = (63 - lz) - s + 1023;  // exponent of the leading bit
  if (rem > 0x400ull || (rem == 0x400ull && (mant & 1ull))) {
    ++mant;
    if (mant >> 53) {
      mant >>= 1;
      ++e;
    }
  }
  if (e <= 0) return 0.0;  // underflow below the normal range: negligible here
  return __longlong_as_double((long long)(sign | ((u64)e << 52) | (mant & 0xFFFFFFFFFFFFFull)));
}

}  // namespace qsf
