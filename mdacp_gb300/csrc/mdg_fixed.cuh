// Fixed-point pair arithmetic: the FP64 form's pair distance and force on the
// integer and float units.
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM sub-partition
// (fma.f64 measured 64-76), one 32 x 32 + 64 bit multiply-add per 4-5, a 64-bit
// add or a logical operation per 2, a float operation per 1.  A pair of about 17
// FP64 instructions costs 1,100 cycles on the FP64 pipe and 160 as the
// operations below (a loop of them on registers alone: 159 with the words split
// as here, 282 with every product in integers).
//
// Formats (the unit of the last bit):
//   position  high word 2^-29 modulo 8 sigma, 32 bits, and the rest, within
//             half a unit of it, as a float (in units of 2^-28): exact for a
//             double coordinate of 1/4 or more in magnitude, below that to
//             2^-55.  The difference of two high words, read as a signed number,
//             is the separation of any pair closer than 4 sigma per axis
//   R = r^2   2^-58 (r < 4)
//   y = 1/r^2 2^-62, y^2 2^-63, z = y^3 2^-61, y^4 2^-62, y^7 2^-59
//   df        2^-55, the force factor 24 y^4 - 48 y^7 + 8 C2 of a pair no
//             closer than kFixNear (|df| < 121)
//   sums      2^-52, integers (the same in any order); what lies below the
//             products of high words by 2^-30 is summed in float, whose
//             rounding is 2^-54 of the force
// These units are fixed, so a pair's error does not shrink with its force as a
// double's does: RMS against exact arithmetic (the double expression's) 7.5e-15
// (1.0e-14) at 1.0-1.12 sigma, 5.3e-16 (7.5e-16) at 1.12-1.5, 1.3e-16 (1.7e-16) at 1.5-2,
// but 1.1e-16 (3.7e-17) at 2.0-2.3, 1.2e-16 (1.5e-17) at 2.3-2.5 and, with a cut-off of
// 3.5, 1.2e-16 (6.7e-18) at 2.5-3 and 1.4e-16 (2.2e-18) at 3-3.5.  A sum with a near
// pair, as a liquid's rows have, is as exact as the double sum; one of far pairs
// alone (a gas between collisions) is good to 2^-52 absolute, not to its last bits.
// The observers' sums cut z and z^2 at 2^-54 likewise.
//
// The functions are plain C++ on fixed-width types; a host compiler builds
// them too.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define MDG_HD __host__ __device__ __forceinline__
#else
#define MDG_HD inline
#endif

namespace mdg {

constexpr int kFixPosBits = 61, kFixR2Bits = 58, kFixDfBits = 55, kFixSumBits = 52;
// Pairs closer than this r^2 (r = 0.918) take the FP64 expression: y^4 stays
// below 2 and |df| below 121.  In a liquid at T = 1.5 about one pair in 10^4 does.
constexpr double kFixNear = 0.8425;

MDG_HD int64_t fix_mads(int32_t a, int32_t b, int64_t c) { return (int64_t)((uint64_t)((int64_t)a * b) + (uint64_t)c); }
MDG_HD uint64_t fix_madu(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }
MDG_HD uint32_t fix_hi(uint64_t v) { return (uint32_t)(v >> 32); }
MDG_HD uint32_t fix_lo(uint64_t v) { return (uint32_t)v; }
// v as hi 2^32 + lo with both words signed.
MDG_HD int32_t fix_shi(int64_t v) { return (int32_t)(fix_hi((uint64_t)v) + (fix_lo((uint64_t)v) >> 31)); }
MDG_HD int32_t fix_slo(int64_t v) { return (int32_t)fix_lo((uint64_t)v); }

// A double as a multiple of 2^-61 modulo 8 (bits below are cut; non-finite
// values give some number).
MDG_HD int64_t fix_from_double(double v) {
#ifdef __CUDA_ARCH__
  const uint64_t b = (uint64_t)__double_as_longlong(v);
#else
  uint64_t b;
  memcpy(&b, &v, 8);
#endif
  const int e = (int)((b >> 52) & 0x7FF);
  const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const int s = e - 1075 + kFixPosBits;  // value = m 2^(e - 1075)
  uint64_t u;
  if (s >= 0) u = s < 64 ? m << s : 0;
  else u = s > -64 ? m >> -s : 0;
  if (e == 0) u = 0;
  return (int64_t)((int64_t)b < 0 ? 0 - u : u);
}

// A fixed-point position: high words, the rest, and a word for the caller
// (the home cell).
struct alignas(32) FixPos {
  int32_t x, y, z;
  float lx, ly, lz;
  int32_t w, pad;
};

MDG_HD float fix_rest(int64_t v) { return (float)fix_slo(v) * (1.0f / 8589934592.0f); }

MDG_HD FixPos fix_position(double x, double y, double z, int32_t w) {
  const int64_t a = fix_from_double(x), b = fix_from_double(y), c = fix_from_double(z);
  return FixPos{fix_shi(a), fix_shi(b), fix_shi(c), fix_rest(a), fix_rest(b), fix_rest(c), w, 0};
}

// Separation of a pair: high words (also as floats) and the rest.
struct FixSep {
  int32_t x, y, z;
  float fx, fy, fz, lx, ly, lz;
};

MDG_HD FixSep fix_sep(int32_t x, int32_t y, int32_t z, float lx, float ly, float lz) {
  return FixSep{x, y, z, (float)x, (float)y, (float)z, lx, ly, lz};
}

// The cross products of high words and rests, twice of which r^2 takes, are
// rounded to 2^-55 (of the size 2^-51 that their float sum is good to where the
// rests matter): across three faces the rests add up to 0.75 an axis, and a
// sum in units of 2^-56 would leave 32 bits from 3.1 sigma on.  In this unit
// it holds to 6.2 sigma; converted to 64 bits instead, 32,000 atoms took 2.5 %
// longer a step.
MDG_HD uint64_t fix_r2(const FixSep &d) {
  const int64_t h = fix_mads(d.z, d.z, fix_mads(d.y, d.y, fix_mads(d.x, d.x, 0)));
  const float c = 0.5f * fmaf(d.fz, d.lz, fmaf(d.fy, d.ly, d.fx * d.lx));  // 2^-56
#ifdef __CUDA_ARCH__
  const int32_t i = __float2int_rn(c);
#else
  const int32_t i = (int32_t)lrintf(c);
#endif
  return (uint64_t)h + ((uint64_t)(int64_t)i << 3);  // twice the cross products
}

// High 64 bits of a * b, low by one or two: the product of the low words and
// the cut of the middle ones are left out.  a.hi b.lo + a.lo b.hi must stay
// below 2^64.
MDG_HD uint64_t fix_mulhi(uint64_t a, uint64_t b) {
  const uint64_t c = fix_madu(fix_hi(a), fix_lo(b), fix_madu(fix_lo(a), fix_hi(b), 0));
  return fix_madu(fix_hi(a), fix_hi(b), 0) + fix_hi(c);
}
MDG_HD uint64_t fix_sqrhi(uint64_t a) {
  return fix_madu(fix_hi(a), fix_hi(a), 0) + (fix_madu(fix_hi(a), fix_lo(a), 0) >> 31);
}

// 1/R: the float estimate Y (26 fractional bits) of the reciprocal, its
// residual t = R Y - 1 exactly in the low 64 bits of the product (|t| < 2^-21),
// and Y (1 - t + t^2).
MDG_HD uint64_t fix_recip(uint64_t R) {
  uint32_t Y;
#ifdef __CUDA_ARCH__
  float y0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(__uint2float_rn(fix_hi(R))));
  Y = __float2uint_rn(y0 * 4503599627370496.0f);
#else
  Y = (uint32_t)(4503599627370496.0f / (float)fix_hi(R) + 0.5f);
#endif
  const uint64_t T = fix_madu(fix_lo(R), Y, 0);
  const int32_t th = (int32_t)(fix_hi(T) + fix_hi(R) * Y);  // t, 2^-52; the low word of T below it
  const uint64_t t = ((uint64_t)(uint32_t)th << 32) | fix_lo(T);
  const uint64_t t2 = (uint64_t)fix_mads(th, th, 0);  // t^2, 2^-104
  // 1 - t + t^2, 2^-63
  const uint64_t U = 0x8000000000000000ull - (uint64_t)((int64_t)t >> 21) + (fix_hi(t2) >> 9);
  const uint32_t Y5 = Y << 5;
  return fix_madu(Y5, fix_hi(U), 0) + fix_hi(fix_madu(Y5, fix_lo(U), 0));
}

// Powers of y: y^2 (2^-63) and z = y^3 (2^-61).
MDG_HD void fix_powers(uint64_t y, uint64_t &y2, uint64_t &z) {
  y2 = fix_sqrhi(y) << 3;
  z = fix_mulhi(y2, y);
}

// The force factor of a pair at R (kFixNear <= r^2), 2^-55; c8 = fix_c8.
MDG_HD int64_t fix_force(uint64_t R, int64_t c8) {
  uint64_t y2, z;
  fix_powers(fix_recip(R), y2, z);
  const uint64_t y4 = fix_sqrhi(y2);
  const int64_t v = (int64_t)((y4 >> 4) - fix_mulhi(y4, z));  // (24 y^4 - 48 y^7) / 3
  return v + (v << 1) + c8;
}

// 8 C2 in the unit of df, less the mean of what fix_force cuts off (3/4 unit
// of 2^-59 from y^7, half a unit of 2^-58 and 5/8 of 2^-62 from y^4).
MDG_HD int64_t fix_c8(double c2x8) {
  const double cut = 48.0 * 0.75 / 576460752303423488.0 - 24.0 * (0.5 / 288230376151711744.0 + 0.625 / 4611686018427387904.0);
  return (int64_t)((c2x8 - cut) * 36028797018963968.0);
}

// Sum of df * d over a row.  df is a high word (2^-23), 22 middle bits (2^-45)
// and 10 low ones; the products with a separation's high word are exact integer
// sums for the first two (x and mx: up to 2^11 pairs), float for the last, as
// is the high word's with the separation's rest.  s: the sum of df's high word
// for fix_sum_fits.
struct FixForce {
  int64_t x, y, z;     // 2^-52
  int64_t mx, my, mz;  // 2^-74
  float cx, cy, cz, s;  // 2^-51; s 2^-23
};

MDG_HD void fix_add(FixForce &f, int64_t df, const FixSep &d) {
  const int32_t h = fix_shi(df), l = fix_slo(df), m = l >> 10;
  const float fh = (float)h, fl = (float)(l & 1023) * (1.0f / 8589934592.0f);
  f.x = fix_mads(h, d.x, f.x);
  f.y = fix_mads(h, d.y, f.y);
  f.z = fix_mads(h, d.z, f.z);
  f.mx = fix_mads(m, d.x, f.mx);
  f.my = fix_mads(m, d.y, f.my);
  f.mz = fix_mads(m, d.z, f.mz);
  f.cx = fmaf(fh, d.lx, fmaf(fl, d.fx, f.cx));
  f.cy = fmaf(fh, d.ly, fmaf(fl, d.fy, f.cy));
  f.cz = fmaf(fh, d.lz, fmaf(fl, d.fz, f.cz));
  f.s += fh;
}

// Whether the components' sums stayed inside 2^11.  df is at most 2 where it
// attracts (r > 1.12), and a repelling pair's force is at most 1.13 |df|, so
// the sum of the n forces' magnitudes is at most 7 n - 1.13 sum(df); sums of
// magnitudes below 2^11 cannot overflow, in any order.
MDG_HD bool fix_sum_fits(const FixForce &f, int n) { return f.s >= (float)(7 * n - 1700) * 8388608.0f; }

// A component of the force in units of 2^-52.
MDG_HD double fix_sum(int64_t v, int64_t m, float c) {
  const float rest = fmaf((float)(int32_t)(m & 0x3FFFFF), 1.0f / 8388608.0f, c);
  return (double)(v + (m >> 22)) + 2.0 * (double)rest;
}

#ifdef __CUDACC__
// 32-byte load of a position: read-only data, or (COH) data that the kernel
// itself writes between grid barriers.
template <bool COH>
__device__ __forceinline__ FixPos ld_fix(const FixPos *p) {
  long long a, b, c, d;
  if (COH) asm volatile("ld.global.v4.s64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p) : "memory");
  else asm("ld.global.nc.v4.s64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
  FixPos v;
  v.x = (int)a;
  v.y = (int)(a >> 32);
  v.z = (int)b;
  v.lx = __int_as_float((int)(b >> 32));
  v.ly = __int_as_float((int)c);
  v.lz = __int_as_float((int)(c >> 32));
  v.w = (int)d;
  v.pad = 0;
  return v;
}
#endif

}  // namespace mdg
