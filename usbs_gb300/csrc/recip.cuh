// Correctly rounded FP64 reciprocal in integer arithmetic.
//
// On GB300 a dependent FP64 instruction takes 60 cycles (150 while all eight warps
// of a CTA use the SM's FP64 unit), and 1 / x is a chain of them: 350 cycles alone,
// 660 with eight warps.  The integer pipes are otherwise idle in the kernels
// that wait for one pivot's reciprocal: 310 and 370 cycles here.  Newton's
// iteration for 1/d in fixed point from the FP32 hardware approximation (about
// 2^-22), then the exact remainder decides the rounding, so the result is that of
// an IEEE division.
#pragma once
#include <stdint.h>

namespace usbs {

__device__ __forceinline__ double recip_exact(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7ff);
  const unsigned long long f = b & 0xfffffffffffffull;
  // zero, subnormal, infinite, NaN, powers of two and results that are not
  // normal: the division itself
  if (ex == 0 || ex >= 2045 || f == 0ull) return 1.0 / x;
  const unsigned long long M = f | 0x10000000000000ull;        // 2^52 < M < 2^53
  const unsigned long long D = M << 11;                         // d = D 2^-64 in (1/2, 1)
  // y0 ~ 1/d in (1, 2), scale 2^-31, from the leading 24 bits of d
  const float d0 = __uint_as_float(0x3f000000u | (unsigned)((f >> 29) & 0x7fffffu));
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d0));
  const unsigned Y0 = (__float_as_uint(fminf(r0, 0x1.fffffep0f)) << 8) | 0x80000000u;
  // e0 = 1 - d y0 (|e0| < 2^-20), scale 2^-63
  const unsigned Dh = (unsigned)(D >> 32), Dl = (unsigned)D;
  const unsigned long long T = (unsigned long long)Dh * Y0 + __umulhi(Dl, Y0);
  const long long e0 = (long long)(0x8000000000000000ull - T);
  // y1 = y0 + y0 e0 (error 2^-41), scale 2^-62
  const unsigned long long Y1 =
      ((unsigned long long)Y0 << 31) + (unsigned long long)(((long long)(int)(e0 >> 12) * (long long)Y0) >> 20);
  // y2 = y1 + y1 e1, e1 = 1 - d y1 scale 2^-62 (|e1| < 2^22)
  const long long e1 = (long long)(0x4000000000000000ull - __umul64hi(D, Y1));
  const unsigned long long Y2 =
      Y1 + (unsigned long long)(((long long)(unsigned)(Y1 >> 32) * (long long)(int)e1) >> 30);
  // quotient floor(2^105 / M) or a neighbour, corrected by the exact remainder
  unsigned long long Q = Y2 >> 10;
  long long R = (long long)(0ull - Q * M);                      // 2^105 - Q M (mod 2^64)
  if (R < 0) { --Q; R += (long long)M; }
  if (R >= (long long)M) { ++Q; R -= (long long)M; }
  if (2 * R > (long long)M) ++Q;                                // nearest (no ties)
  const unsigned long long out = ((unsigned long long)(2045 - ex) << 52) + (Q - 0x10000000000000ull);
  return __longlong_as_double((long long)((b & 0x8000000000000000ull) | out));
}

}  // namespace usbs
