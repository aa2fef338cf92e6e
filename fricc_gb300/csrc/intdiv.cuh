// Correctly rounded FP64 quotients on the integer pipe.  An FP64 division is ~10
// dependent FP64 instructions, of which GB300 issues two per SM and clock; the
// passes that divide every element were bound by them.
//
// With the 53-bit significands ma, mr of a and R and a word V at most 7 below
// 2^116 / mr, Q = floor(2^11 ma V / 2^64) lies at most 8 below 2^63 ma / mr, a
// number of 63 or 64 bits.  Where the 10 or 11 bits to be rounded off are
// farther than QUOT_SLACK below the halfway case, or above it, the nearest double
// follows from Q; else (about 1%) from comparing ma 2^63 with that case times
// mr.  Operands or quotients that are not normal take the division.
#pragma once
#include <cuda_runtime.h>

constexpr unsigned QUOT_SLACK = 12;

// V for one R used many times: floor(2^116 / mr), or 0 where R is not normal
// and positive
__device__ __forceinline__ unsigned long long recip_word(double R) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(R);
  const unsigned e = (unsigned)(u >> 52);
  if (e < 1 || e > 2046) return 0;  // zero, subnormal, negative, infinite or NaN
  const unsigned long long mr = (u & 0xfffffffffffffull) | (1ull << 52);
  return mr == 1ull << 52 ? ~0ull : (unsigned long long)(((unsigned __int128)1 << 116) / mr);
}

// V for an R of its own: the FP32 reciprocal of the leading 32 bits and two
// Newton steps y (2 - y d), which stay below 1/d for a y below it
__device__ __forceinline__ unsigned long long recip_word_once(unsigned long long mr) {
  const unsigned long long d = mr << 11;
  const unsigned dh = (unsigned)(d >> 32);
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)dh));
  const unsigned y0 = __float2uint_rz(f * 9223367638808264704.0f);  // (1 - 2^-21) 2^63: below by 2^-20 at most
  const unsigned long long e = (1ull << 63) - ((unsigned long long)y0 * dh + y0);  // against dh + 1 > d 2^-32
  const unsigned long long y = ((unsigned long long)y0 << 32) + (((unsigned long long)y0 * (unsigned)(e >> 11)) >> 20);
  const unsigned long long e2 = (1ull << 63) - 1 - __umul64hi(y, d);
  return y + __umul64hi(y, e2 << 1);
}

// a / R from the bits of both and V; V != 0, exponents of both in 1..2046 and the
// quotient's too (the caller's check: quot_normal)
__device__ __forceinline__ bool quot_normal(unsigned long long u, unsigned long long ur) {
  const int ea = (int)(u >> 52) & 0x7ff, er = (int)(ur >> 52) & 0x7ff, e = ea - er + 1023;
  return ea >= 1 && ea <= 2046 && er >= 1 && er <= 2046 && e >= 3 && e <= 2044;
}
__device__ __forceinline__ double quot_round(unsigned long long u, unsigned long long ur, unsigned long long V) {
  const int e = ((int)(u >> 52) & 0x7ff) - ((int)(ur >> 52) & 0x7ff) + 1023;
  const unsigned long long ma = (u & 0xfffffffffffffull) | (1ull << 52), q = __umul64hi(ma << 11, V);
  const int drop = 10 + (int)(q >> 63);  // bits to round off
  const unsigned low = (unsigned)q & ((1u << drop) - 1), half = 1u << (drop - 1);
  bool up = low > half;
  if (low - (half - QUOT_SLACK) <= QUOT_SLACK) {
    const unsigned long long mr = (ur & 0xfffffffffffffull) | (1ull << 52);
    const unsigned long long h = (q & ~((1ull << drop) - 1)) + half, hi = __umul64hi(h, mr), lo = h * mr;
    const unsigned long long t_hi = ma >> 1, t_lo = ma << 63;
    up = t_hi > hi || (t_hi == hi && (t_lo > lo || (t_lo == lo && ((q >> drop) & 1))));
  }
  // (the significand's leading bit adds one to the exponent)
  return __longlong_as_double((long long)((((unsigned long long)(e - 12 + drop) << 52) + (q >> drop) + up) |
                                          ((u ^ ur) & (1ull << 63))));
}

// fl(a / R), R shared by many a: rv = recip_word(R); a >= 0 or NaN
__device__ __forceinline__ double div_by(double a, double R, unsigned long long rv) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(a), ur = (unsigned long long)__double_as_longlong(R);
  if (rv != 0 && quot_normal(u, ur)) return quot_round(u, ur, rv);
  return u == 0 && rv != 0 ? 0.0 : __ddiv_rn(a, R);
}

// fl(a / R)
static __device__ __noinline__ double div_slow(double a, double R) { return __ddiv_rn(a, R); }
__device__ __forceinline__ double div_exact(double a, double R) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(a), ur = (unsigned long long)__double_as_longlong(R);
  if (!quot_normal(u, ur)) return div_slow(a, R);
  return quot_round(u, ur, recip_word_once((ur & 0xfffffffffffffull) | (1ull << 52)));
}
