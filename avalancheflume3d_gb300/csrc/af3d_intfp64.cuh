// af3d_intfp64.cuh -- correctly rounded FP64 division and square root on the integer pipe.
//
// An FP64 instruction holds the FP64 unit of an SM sub-partition for 64 to 76 cycles on this GPU
// (measured: a warp's DFMAs issue 64 cycles apart, dependent or not, whatever the number of active
// lanes), so a division (563 cycles of that unit) or a square root (623) costs what nine or ten
// multiply-adds do.  The functions here return the same bits from integer arithmetic: the
// hardware's FP32 reciprocal (square root) estimate, one Newton step in 32-bit fixed point, then
// long division (long-hand square root) in two digits of about 28 bits, each digit's remainder
// formed exactly modulo 2^64.  The exact last remainder decides the rounding, so the result is
// the correctly rounded one by construction (a quotient or square root of 53-bit numbers is
// never half-way between two of them unless it is representable).  Operands or results outside
// the normal range (and NaN) take the hardware instruction.  Measured, exact mode, the same bits:
// the 262,144-clump flume's 20 steps with their copies 13.4 -> 9.7 ms, 20,011 clumps in the filling
// hopper 107 -> 82 us a step, 512 clumps (one warp's serial chain) 65 -> 56 us.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace af3d {

#ifdef __CUDACC__
__device__ __forceinline__ unsigned long long bits_of(double x) { return (unsigned long long)__double_as_longlong(x); }
__device__ __forceinline__ double of_bits(unsigned long long u) { return __longlong_as_double((long long)u); }
__device__ __forceinline__ unsigned mulhi_u(unsigned a, unsigned b) { return __umulhi(a, b); }
__device__ __forceinline__ int mulhi_s(int a, int b) { return __mulhi(a, b); }
__device__ __forceinline__ float float_of_bits(unsigned u) { return __uint_as_float(u); }
__device__ __forceinline__ unsigned bits_of_float(float x) { return __float_as_uint(x); }
__device__ __forceinline__ float rcp_estimate(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_estimate(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The instructions for operands out of range; not inlined, so that their registers do not weigh
// on the usual path.
static __device__ __noinline__ double div_instr(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_instr(double x) { return sqrt(x); }
#define AF3D_HD __device__ __forceinline__
#else
inline unsigned long long bits_of(double x) { unsigned long long u; std::memcpy(&u, &x, 8); return u; }
inline double of_bits(unsigned long long u) { double x; std::memcpy(&x, &u, 8); return x; }
inline unsigned mulhi_u(unsigned a, unsigned b) { return (unsigned)((unsigned long long)a * b >> 32); }
inline int mulhi_s(int a, int b) { return (int)((long long)a * b >> 32); }
inline float float_of_bits(unsigned u) { float x; std::memcpy(&x, &u, 4); return x; }
inline unsigned bits_of_float(float x) { unsigned u; std::memcpy(&u, &x, 4); return u; }
// The host build exists for the tests: the estimates may be off by a few units in the last place.
extern int g_estimate_ulps;
inline float rcp_estimate(float x) { return float_of_bits(bits_of_float(1.0f / x) + g_estimate_ulps); }
inline float rsqrt_estimate(float x) { return float_of_bits(bits_of_float(1.0f / std::sqrt(x)) + g_estimate_ulps); }
inline double div_instr(double a, double b) { return a / b; }
inline double sqrt_instr(double x) { return std::sqrt(x); }
#define AF3D_HD inline
#endif

// The FP32 estimate y of a number in (1/2, 1], in Q23: y + 1 in (1.5, 2] holds it in its last 23 bits.
// An estimate past 1 (of the reciprocal or root of a mantissa at or just above 1) is one unit below
// it, as 1 is, so that it fits 31 bits in Q31 and the Newton step takes it from there.
AF3D_HD unsigned estimate_q23(float y) {
  const unsigned e = bits_of_float(y + 1.0f) - 0x3F800001u;
  return e < 0x7FFFFFu ? e : 0x7FFFFFu;
}

// A divisor's 53-bit mantissa and the reciprocal of (mantissa / 2^52) in Q31, within two units.
struct Divisor {
  double b;
  unsigned long long m;
  unsigned r;
};

AF3D_HD Divisor divisor_of(double b) {
  const unsigned long long ub = bits_of(b);
  const unsigned hi = (unsigned)(ub >> 32), lo = (unsigned)ub;
  Divisor d;
  d.b = b;
  d.m = ((unsigned long long)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo;
  const unsigned top = ((hi & 0xFFFFFu) << 3) | (lo >> 29);
  const unsigned r0 = estimate_q23(rcp_estimate(float_of_bits(0x3F800000u | top))) << 8;   // Q31, below 2^31
  // one Newton step: r0 + r0 (1 - b r0), the residual in Q50
  const unsigned bh = (unsigned)(d.m >> 21);   // Q31
  const long long e = (1LL << 62) - (long long)((unsigned long long)bh * r0);
  d.r = r0 + (unsigned)(mulhi_s((int)r0, (int)(e >> 12)) >> 18);
  return d;
}

// a / d.b, correctly rounded.
AF3D_HD double div_by(double a, const Divisor &d) {
  const unsigned long long ua = bits_of(a), ub = bits_of(d.b);
  const unsigned ah = (unsigned)(ua >> 32), bhi = (unsigned)(ub >> 32);
  const int ea = (int)((ah >> 20) & 0x7FFu), eb = (int)((bhi >> 20) & 0x7FFu);
  const unsigned sign = (ah ^ bhi) & 0x80000000u;
  const int er = ea - eb + 1022;   // the quotient's biased exponent, or one less than it
  const bool zero = (ua << 1) == 0ull;
  const bool fast = (unsigned)(eb - 1) < 2046u && (zero || ((unsigned)(ea - 1) < 2046u && (unsigned)(er - 1) < 2044u));
  if (!fast) return div_instr(a, d.b);
  const unsigned long long ma = ((unsigned long long)((ah & 0xFFFFFu) | 0x100000u) << 32) | (unsigned)ua;
  // first digit: a/b in Q30, within three units
  const unsigned q1 = mulhi_u((unsigned)(ma >> 21), d.r);
  const long long rem = (long long)((ma << 30) - q1 * d.m);   // |rem| < 2^55, exact
  // second digit: rem 2^25 / m, rounded down: the truncations and d.r's error put the product's
  // quarter between 0.15 and 1.5 below it
  const int q2 = (mulhi_s((int)(rem >> 24), (int)d.r) - 1) >> 2;
  const unsigned long long rem2 = ((unsigned long long)rem << 25) - (unsigned long long)(long long)q2 * d.m;
  unsigned long long Q = ((unsigned long long)q1 << 25) + (long long)q2;
  Q += rem2 >= d.m;   // floor(ma 2^55 / m), 55 or 56 bits
  const int s = 2 + (int)(Q >> 55);
  const unsigned long long mant = (Q + (1ull << (s - 1))) >> s;   // 53 bits, or 2^53
  const unsigned long long r = (((unsigned long long)(unsigned)(er + s - 3)) << 52) + mant;
  return of_bits((zero ? 0ull : r) | (unsigned long long)sign << 32);
}

// 1/sqrt(v) for v = M / 2^52 in [1, 4), in Q31 within two units.
AF3D_HD unsigned rsqrt_q31(unsigned long long M, unsigned hi_float) {
  const unsigned r23 = estimate_q23(rsqrt_estimate(float_of_bits(hi_float)));
  const unsigned vh = (unsigned)(M >> 22);                       // Q30
  const unsigned t = (unsigned)(((unsigned long long)r23 * r23) >> 15);   // y^2 in Q31
  const long long e = (1LL << 61) - (long long)((unsigned long long)vh * t);   // 1 - v y^2 in Q61
  const unsigned r0 = r23 << 8;
  return r0 + (unsigned)(mulhi_s((int)r0, (int)(e >> 11)) >> 19);
}

// sqrt(x), correctly rounded.
AF3D_HD double sqrt_rn(double x) {
  const unsigned long long u = bits_of(x);
  const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
  const int e = (int)(hi >> 20);
  if (!((unsigned)(e - 1) < 2046u)) return sqrt_instr(x);   // zero, subnormal, negative, inf, NaN
  const int odd = ~e & 1;   // x = v 4^k with v in [1, 4): the unbiased exponent e - 1023 is odd when e is even
  const unsigned long long M = (((unsigned long long)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo) << odd;
  const unsigned r = rsqrt_q31(M, (0x3F800000u + ((unsigned)odd << 23)) | (((hi & 0xFFFFFu) << 3) | (lo >> 29)));
  // first digit: sqrt(v) in Q29
  const unsigned s1 = mulhi_u((unsigned)(M >> 22), r);
  const long long rem = (long long)((M << 6) - (unsigned long long)s1 * s1);   // Q58, exact
  // second digit, to Q54, rounded down: the truncations, r's error and the square of the digit
  // put the product's half between 0.05 and 1.9 below it
  const int q2 = (mulhi_s((int)(rem >> 3), (int)r) - 1) >> 1;
  unsigned long long S = ((unsigned long long)s1 << 25) + (long long)q2;
  const unsigned long long rem2 = (M << 56) - S * S;   // Q108 modulo 2^64, exact and below 2^58
  S += (long long)(rem2 - 2 * S - 1) >= 0;   // floor(sqrt) in Q54, 55 bits
  const unsigned long long mant = (S + 2) >> 2;
  return of_bits(((unsigned long long)(unsigned)(((e - 1023 - odd) >> 1) + 1022) << 52) + mant);
}

AF3D_HD double div_rn(double a, double b) { return div_by(a, divisor_of(b)); }

#ifdef __CUDACC__
// A Divisor of a constant, formed by the compiler.
__host__ __device__ constexpr Divisor constant_divisor(double b, unsigned long long bits) {
  const unsigned long long m = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  return Divisor{b, m, (unsigned)((1ull << 63) / (m >> 20)) - 1u};
}

// The Q31 number r in [2^30, 2^31) times 2^(e - 1022): a double with that mantissa.
__device__ __forceinline__ double double_of_q31(unsigned r, int e) {
  const unsigned f = max(r, 0x40000000u) & 0x3FFFFFFFu;
  return of_bits((unsigned long long)(((unsigned)e << 20) + (f >> 10)) << 32 | (unsigned long long)(f << 22));
}

// 1/b within an ulp (not correctly rounded): the 31-bit reciprocal and one FP64 Newton step.
__device__ __forceinline__ double reciprocal(double b) {
  const unsigned hi = (unsigned)(bits_of(b) >> 32);
  const int e = (int)((hi >> 20) & 0x7FFu);
  if (!((unsigned)(e - 2) < 2043u)) return div_instr(1.0, b);
  double y = double_of_q31(divisor_of(b).r, 2045 - e);
  y = of_bits(bits_of(y) | (unsigned long long)(hi & 0x80000000u) << 32);
  return __fma_rn(y, __fma_rn(-b, y, 1.0), y);
}

// s = sqrt(x), correctly rounded, and inv = 1/s within an ulp (inf for x = 0).
__device__ __forceinline__ double sqrt_and_inverse(double x, double &inv) {
  const double s = sqrt_rn(x);
  inv = reciprocal(s);
  return s;
}
#endif

#undef AF3D_HD
}  // namespace af3d
