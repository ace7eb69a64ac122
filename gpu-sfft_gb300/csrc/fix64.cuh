// 64-bit fixed-point complex arithmetic for the FP64 FFT passes.
//
// GB300's FP64 pipe retires 1.73 operations per clock and SM (measured; DFMA
// and DADD alike, conversions 2.06), its integer pipes 64.5 32 x 32 + 64 ->
// 64-bit multiply-adds and 50.7 64-bit additions.  A transform does
// additions for the most part, so the same butterflies on integers of 62 bits
// cost a tenth of the clocks -- and carry more bits than a double does.
//
// A number is a signed 64-bit integer; a product splits both factors into a
// signed high limb and a signed ("balanced") low limb, v = h 2^32 + l with
// -2^31 <= l < 2^31, and drops l * l' (at most 1/4 of the result's last bit):
//   v w 2^-64 = h h' + (h l' + l h') 2^-32,
// three 32 x 32 multiply-adds, all signed.  |v| stays below 2^62.5 and twiddle
// factors are scaled by 2^60 or 2^62, so that no sum of limbs overflows.
//
// Host and device code alike (the CPU checks of the arithmetic run it too).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gsfft {
namespace fx {

#define FX_FN __host__ __device__ __forceinline__

struct C64 {  // complex fixed-point number
  long long x, y;
};
// twiddle factor as limbs: re = rh 2^32 + rl, im = ih 2^32 + il
typedef int4 Tw;  // x = rh, y = rl, z = ih, w = il

FX_FN int limb_lo(long long v) { return (int)(unsigned)v; }
FX_FN int limb_hi(long long v) { return (int)(v >> 32) + (int)((unsigned)v >> 31); }
FX_FN long long mulw(int a, int b) {
#ifdef __CUDA_ARCH__
  long long d;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
  return d;
#else
  return (long long)a * b;
#endif
}
// One multiply-add instruction (written as C, the compiler splits it into a
// product and an addition).  Its result takes the place of c, so a constant c
// would cost moves: the sums below start with a product.
FX_FN long long madw(int a, int b, long long c) {
#ifdef __CUDA_ARCH__
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (long long)a * b + c;
#endif
}
FX_FN int top(long long v) { return (int)(v >> 32); }

FX_FN unsigned long long umulhi(unsigned long long a, unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
#endif
}

FX_FN C64 add(C64 a, C64 b) { return C64{a.x + b.x, a.y + b.y}; }
FX_FN C64 sub(C64 a, C64 b) { return C64{a.x - b.x, a.y - b.y}; }
FX_FN C64 mul_mi(C64 a) { return C64{a.y, -a.x}; }  // a * -i

// v 2^-32, rounded, times one.  one = 1 (or 2) comes in a register whose value the
// compiler cannot see: the sign extension of a high word is then one multiplication instead of a
// shift and a move.
FX_FN long long top64(long long v, int one) { return mulw(limb_hi(v), one); }

// x w 2^-64, rounded; |x| <= 2^62.5, |w| <= 2^62; one = 1
FX_FN C64 cmul(C64 x, Tw w, int one) {
  const int xh = limb_hi(x.x), xl = limb_lo(x.x), yh = limb_hi(x.y), yl = limb_lo(x.y);
  const int nyh = -yh, nih = -w.z;  // high limbs only: they never hold -2^31
  const long long tr = madw(yl, nih, madw(nyh, w.w, madw(xl, w.x, mulw(xh, w.y))));
  const long long ti = madw(yl, w.x, madw(yh, w.y, madw(xl, w.z, mulw(xh, w.w))));
  return C64{madw(nyh, w.z, madw(xh, w.x, top64(tr, one))), madw(yh, w.x, madw(xh, w.z, top64(ti, one)))};
}

FX_FN Tw limbs(C64 w) { return Tw{limb_hi(w.x), limb_lo(w.x), limb_hi(w.y), limb_lo(w.y)}; }

// product of two twiddle factors scaled by 2^62, again scaled by 2^62
FX_FN C64 tw_mul(C64 a, Tw b, int one) {
  const C64 p = cmul(a, b, one);  // scaled by 2^60
  return C64{(long long)((unsigned long long)p.x << 2), (long long)((unsigned long long)p.y << 2)};
}

// a / 16, rounded
FX_FN C64 div16(C64 a) { return C64{(a.x + 8) >> 4, (a.y + 8) >> 4}; }

// Constants c = ch 2^-31 + cl 2^-63 of the in-register butterflies:
// cos(pi/4); cos(pi/8), sin(pi/8)
#define FX_C8H 1518500250
#define FX_C8L (-51432894)
#define FX_C16H 1984016189
#define FX_C16L (-902489949)
#define FX_S16H 821806413
#define FX_S16L 1565705635

// x * c for |x| <= 2^62.5, rounded to a multiple of two; one = 1
FX_FN long long mul_c8(long long v, int one) {
  const int h = limb_hi(v), l = limb_lo(v);
  const long long t = madw(l, FX_C8H, mulw(h, FX_C8L));
  const long long p = madw(h, FX_C8H, top64(t, one));
  return p + p;
}
// x exp(-i pi/4), x exp(-3 i pi/4)
FX_FN C64 rot1_8(C64 v, int one) { return C64{mul_c8(v.x + v.y, one), mul_c8(v.y - v.x, one)}; }
FX_FN C64 rot3_8(C64 v, int one) { return C64{mul_c8(v.y - v.x, one), -mul_c8(v.x + v.y, one)}; }

// x (c - i s), the constants given as limbs; |x| <= 2^60.5
template <int CH, int CL, int SH, int SL>
FX_FN C64 rot_c(C64 v, int one) {
  const int xh = limb_hi(v.x), xl = limb_lo(v.x), yh = limb_hi(v.y), yl = limb_lo(v.y);
  const long long tr = madw(yl, SH, madw(yh, SL, madw(xl, CH, mulw(xh, CL))));
  const long long ti = madw(xl, -SH, madw(xh, -SL, madw(yl, CH, mulw(yh, CL))));
  const int x2 = 2 * xh, y2 = 2 * yh, two = 2 * one;
  return C64{madw(y2, SH, madw(x2, CH, top64(tr, two))), madw(x2, -SH, madw(y2, CH, top64(ti, two)))};
}
FX_FN C64 rot1_16(C64 v, int one) { return rot_c<FX_C16H, FX_C16L, FX_S16H, FX_S16L>(v, one); }
FX_FN C64 rot3_16(C64 v, int one) { return rot_c<FX_S16H, FX_S16L, FX_C16H, FX_C16L>(v, one); }
FX_FN C64 rot9_16(C64 v, int one) { return rot_c<-FX_C16H, -FX_C16L, -FX_S16H, -FX_S16L>(v, one); }

// 4-point DFT of v[0], v[S], v[2S], v[3S], in place
template <int S> FX_FN void dft4(C64 *v) {
  const C64 a = add(v[0], v[2 * S]), b = sub(v[0], v[2 * S]);
  const C64 c = add(v[S], v[3 * S]), d = mul_mi(sub(v[S], v[3 * S]));
  v[0] = add(a, c);
  v[S] = add(b, d);
  v[2 * S] = sub(a, c);
  v[3 * S] = sub(b, d);
}

// E-point DFT in registers, E = 2, 4, 8, 16; X[k] is left in v[dft_at<E>(k)].
// 8 and 16 points as 4 x 2 and 4 x 4: v[(E/4) a + b], first over a.  one = 1
template <int E> FX_FN constexpr int dft_at(int k) { return E <= 4 ? k : (E / 4) * (k & 3) + (k >> 2); }

template <int E> FX_FN void dft(C64 *v, int one) {
  if constexpr (E == 2) {
    const C64 a = v[0], b = v[1];
    v[0] = add(a, b);
    v[1] = sub(a, b);
  } else if constexpr (E == 4) {
    dft4<1>(v);
  } else if constexpr (E == 8) {
    dft4<2>(v);
    dft4<2>(v + 1);
    v[3] = rot1_8(v[3], one);
    v[5] = mul_mi(v[5]);
    v[7] = rot3_8(v[7], one);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int k = 0; k < 4; k++) {
      const C64 a = v[2 * k], b = v[2 * k + 1];
      v[2 * k] = add(a, b);
      v[2 * k + 1] = sub(a, b);
    }
  } else {
    dft4<4>(v);
    dft4<4>(v + 1);
    dft4<4>(v + 2);
    dft4<4>(v + 3);
    v[5] = rot1_16(v[5], one);
    v[6] = rot1_8(v[6], one);
    v[7] = rot3_16(v[7], one);
    v[9] = rot1_8(v[9], one);
    v[10] = mul_mi(v[10]);
    v[11] = rot3_8(v[11], one);
    v[13] = rot3_16(v[13], one);
    v[14] = rot3_8(v[14], one);
    v[15] = rot9_16(v[15], one);
    dft4<1>(v);
    dft4<1>(v + 4);
    dft4<1>(v + 8);
    dft4<1>(v + 12);
  }
}

// double -> fixed: d 2^(P - (emax - 1022)) truncated, where emax is the largest
// exponent field of the block (so the result is below 2^P), c = emax + 62 - P; e is
// d's own exponent field.
// The 53-bit mantissa at bits 9..61 is shifted right by c - exponent; a zero, a
// subnormal or a value far below the block's largest shifts out.  On the integer
// pipes: conversion instructions run at 2.06 a clock and SM, and the pass waited
// for them (126 -> 142 us).
FX_FN unsigned double_hi(double d) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2hiint(d);
#else
  unsigned long long b;
  __builtin_memcpy(&b, &d, 8);
  return (unsigned)(b >> 32);
#endif
}
FX_FN unsigned double_lo(double d) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(d);
#else
  unsigned long long b;
  __builtin_memcpy(&b, &d, 8);
  return (unsigned)b;
#endif
}
FX_FN int exponent(double d) { return (int)((double_hi(d) >> 20) & 0x7ffu); }  // its field
FX_FN long long from_double(double d, int e, int c) {
  const unsigned lo = double_lo(d), hi = double_hi(d);
  const int s = c - e;
  const unsigned long long m = (((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << 9;
#ifdef __CUDA_ARCH__
  unsigned long long v;
  asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(s));  // shifts of 64 and more give 0
#else
  const unsigned long long v = s > 63 ? 0 : m >> s;
#endif
  return (int)hi < 0 ? -(long long)v : (long long)v;
}

// cos and sin of 2 pi f 2^-64, scaled by 2^62, to within two units: Taylor
// series in 64-bit fixed point on the first octant (pi/4 at most; nine terms
// leave less than 2^-66), the other octants by symmetry.
FX_FN void sincos62(unsigned long long f, long long *cs, long long *sn) {
  const unsigned oct = (unsigned)(f >> 61);
  unsigned long long a = f & 0x1fffffffffffffffull;
  if (oct & 1u) a = 0x2000000000000000ull - a;
  const unsigned long long PI_HALF_63 = 0xC90FDAA22168C235ull;  // pi/2 2^63
  const unsigned long long hi = umulhi(a, PI_HALF_63), lo = a * PI_HALF_63;
  const unsigned long long x = (hi << 3) | (lo >> 61);  // the angle in radians, 2^64
  const unsigned long long z = umulhi(x, x);
  unsigned long long tc = 0, ts = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int k = 9; k >= 1; k--) {
    const unsigned long long one = 0xffffffffffffffffull;
    const unsigned long long zc = umulhi(z, one / (unsigned)((2 * k - 1) * (2 * k)));
    const unsigned long long zs = umulhi(z, one / (unsigned)((2 * k) * (2 * k + 1)));
    tc = zc - umulhi(zc, tc);
    ts = zs - umulhi(zs, ts);
  }
  const long long c = (1LL << 62) - (long long)((tc + 2) >> 2);
  const long long s = (long long)((x - umulhi(x, ts) + 2) >> 2);
  const bool swap = ((oct + 1u) & 2u) != 0;  // octants 1, 2, 5, 6
  long long C = swap ? s : c, S = swap ? c : s;
  if (oct >= 2u && oct < 6u) C = -C;
  if (oct >= 4u) S = -S;
  *cs = C;
  *sn = S;
}

// exp(-2 pi i num / 2^logden) scaled by 2^62
FX_FN C64 unit_root(unsigned long long num, int logden) {
  long long c, s;
  sincos62(logden ? num << (64 - logden) : 0ull, &c, &s);
  return C64{c, -s};
}

}  // namespace fx
}  // namespace gsfft
