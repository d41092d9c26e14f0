// Correctly rounded FP64 division and square root, and FP64 comparisons, in
// integer instructions.
//
// GB300 has one FP64 lane for 64 FP32 lanes: an FP64 instruction, a
// comparison included, holds its SM quarter's FP64 unit for about 64 cycles
// per warp, so the compiler's division or square root (a dozen chained FP64
// instructions) takes 550 to 670 cycles.  The functions here compute the same
// value, the IEEE 754 quotient or root rounded to nearest even, from the bit
// patterns on the integer pipes.
//
// Method (high-radix digit recurrence, Ercegovac and Lang, "Digital
// Arithmetic", ch. 5 and 6, with the digits from a short reciprocal): an FP32
// seed of 1/b (1/sqrt(x)) is refined by one Newton step in 32-bit fixed point
// to about 2^-28, always from below; two digits of the quotient (root), 31
// and 23 bits, come from products with it, each after an exact remainder.
// The 54-bit candidate is then less than 2 off the exact value scaled by
// 2^53.  A quotient (root) of two normal 53-bit numbers is never half way
// between two others, so rounding needs only the sign of the exact remainder
// at the odd number H next to the candidate: above it the result is
// (H + 1) / 2, below it (H - 1) / 2.  Operands outside the plain range
// (zeros except a zero dividend, subnormals, infinities, NaN, results near
// the ends of the exponent range) take the compiler's operation.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fc3dgpu {

#if defined(__CUDA_ARCH__)
__device__ __forceinline__ uint32_t ie_rcp_seed(uint32_t f) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
  return __float_as_uint(y);
}
__device__ __forceinline__ uint32_t ie_rsqrt_seed(uint32_t f) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
  return __float_as_uint(y);
}
__device__ __forceinline__ uint32_t ie_mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
__device__ __forceinline__ uint64_t ie_bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double ie_double(uint64_t x) { return __longlong_as_double((long long)x); }
#define IE_AS_FLOAT(u) __uint_as_float(u)
#define IE_FN __device__ __forceinline__
#define IE_SLOW static __device__ __noinline__
#else
// host versions, for the tests: the seeds with a settable error in units of
// the last place, since the device's approximations are not exact (at most 1
// unit for the reciprocal, 2^-22.9 or 2.1 units for the reciprocal root; the
// results are right up to 3)
#include <math.h>
#include <string.h>
static int ie_host_seed_ulps = 0;
static inline uint32_t ie_host_f(float y) {
  uint32_t u;
  memcpy(&u, &y, 4);
  return u + (uint32_t)ie_host_seed_ulps;
}
static inline float ie_host_as_float(uint32_t f) {
  float x;
  memcpy(&x, &f, 4);
  return x;
}
static inline uint32_t ie_rcp_seed(uint32_t f) { return ie_host_f((float)(1.0 / (double)ie_host_as_float(f))); }
static inline uint32_t ie_rsqrt_seed(uint32_t f) { return ie_host_f((float)(1.0 / sqrt((double)ie_host_as_float(f)))); }
static inline uint32_t ie_mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline uint64_t ie_bits(double x) {
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
}
static inline double ie_double(uint64_t u) {
  double x;
  memcpy(&x, &u, 8);
  return x;
}
#define IE_AS_FLOAT(u) ie_host_as_float(u)
#define IE_FN static inline
#define IE_SLOW static
#endif

// 2^32 times the seed with FP32 pattern f, less `ulps` units of its last place
// (at least 1/2, so never above a value of [1/2, 1) the seed approximates)
IE_FN uint32_t ie_fixed(uint32_t f, uint32_t ulps) {
  f -= ulps;
  f = f > 0x3f000000u ? f : 0x3f000000u;
  return (f << 8) | 0x80000000u;
}

// 2^32 / b, b = mb 2^-52 in [1, 2), from below (relative error under 2^-28)
IE_FN uint32_t ie_reciprocal(uint64_t mb) {
  const uint32_t bh = (uint32_t)(mb >> 21);  // b 2^31
  // seed from b rounded up to 24 bits, less 4 ulps: below 1/b
  const uint32_t y0 = ie_fixed(ie_rcp_seed(0x3f800000u + (((bh >> 8) & 0x7fffffu) + 1u)), 4u);
  const uint32_t e = 0x80000000u - ie_mulhi(bh, y0);  // (1 - b y) 2^31, positive
  return y0 + ie_mulhi(y0, 2u * e) - 8u;
}

// the mantissa of ma / mb, doubled first when ma < mb (lt), with y the
// reciprocal of mb: a 53-bit integer in [2^52, 2^53], correctly rounded
IE_FN uint64_t ie_quotient(uint64_t ma, uint64_t mb, uint32_t y, bool lt) {
  const uint64_t an = ma << (lt ? 1 : 0);                 // an / (2 mb) in [1/2, 1)
  const uint32_t ml = (uint32_t)mb, mh = (uint32_t)(mb >> 32);
  const uint32_t q1 = ie_mulhi((uint32_t)(an >> 22), y);  // 31 bits
  const uint64_t t = (an << 31) - (uint64_t)(2u * q1) * ml - ((uint64_t)(2u * q1 * mh) << 32);
  const uint32_t q2 = (ie_mulhi((uint32_t)(t >> 26), y) >> 4) | 1u;
  const uint64_t u = (t << 22) - (uint64_t)q2 * ml - ((uint64_t)(q2 * mh) << 32);
  return ((((uint64_t)q1 << 23) + q2) >> 1) + (uint64_t)(1u - (uint32_t)(u >> 63));
}

// the mantissa of the root of m (53-bit with the leading one), of 2 m when
// odd: correctly rounded, in [2^52, 2^53]
IE_FN uint64_t ie_root(uint64_t m, bool odd) {
  const uint64_t mo = m << (odd ? 1 : 0);    // x 2^52, x in [1, 4)
  const uint32_t xh = (uint32_t)(mo >> 22);  // x 2^30
  const uint32_t f = (odd ? 0x40000000u : 0x3f800000u) + ((uint32_t)(m >> 29) & 0x7fffffu) + 1u;
  const uint32_t y0 = ie_fixed(ie_rsqrt_seed(f), 8u);
  const uint32_t e = 0x40000000u - ie_mulhi(xh, ie_mulhi(y0, y0));  // (1 - x y^2) 2^30, positive
  const uint32_t y = y0 + ie_mulhi(y0, 2u * e) - 5u;                // 2^32 / sqrt(x), from below
  const uint32_t s1 = ie_mulhi(xh, y);                              // 31 bits
  const uint64_t t = (mo << 8) - (uint64_t)s1 * s1;
  const uint32_t q2 = ie_mulhi((uint32_t)(t >> 5), y) >> 3;
  const uint64_t h = (((uint64_t)s1 << 23) + q2) | 1u;
  const uint32_t hl = (uint32_t)h, hh = (uint32_t)(h >> 32);
  const uint64_t u = (mo << 54) - (uint64_t)hl * hl - ((uint64_t)(2u * hl * hh) << 32);
  return (h >> 1) + (uint64_t)(1u - (uint32_t)(u >> 63));
}

#define IE_MANTISSA 0xfffffffffffffull
#define IE_ONE 0x10000000000000ull

IE_SLOW double ie_div_slow(double a, double b) { return a / b; }
IE_SLOW double ie_sqrt_slow(double a) { return sqrt(a); }

// A divisor with its reciprocal, for several quotients by it.
struct IeDen {
  double b;
  uint32_t y;
};

IE_FN IeDen ie_den(double b) {
  IeDen d;
  d.b = b;
  d.y = ie_reciprocal((ie_bits(b) & IE_MANTISSA) | IE_ONE);
  return d;
}

// a / b without a branch; ok is false where the operands are outside the
// plain range and the value returned is not the quotient
IE_FN double ie_div_plain(double a, const IeDen& d, bool& ok) {
  const uint64_t x = ie_bits(a), z = ie_bits(d.b);
  const uint32_t xh = (uint32_t)(x >> 32), zh = (uint32_t)(z >> 32);
  const uint32_t ea = (xh >> 20) & 0x7ffu, eb = (zh >> 20) & 0x7ffu;
  const uint32_t sign = (xh ^ zh) & 0x80000000u;
  const uint32_t ex = ea - eb + 1022u;  // the quotient's biased exponent, less one, before normalisation
  const bool zero = (x << 1) == 0;
  ok = eb - 1u < 2046u && (zero || (ea - 1u < 2046u && ex - 2u < 2042u));
  const uint64_t ma = (x & IE_MANTISSA) | IE_ONE, mb = (z & IE_MANTISSA) | IE_ONE;
  const bool lt = ma < mb;
  const uint64_t q = ie_quotient(ma, mb, d.y, lt) + ((uint64_t)(ex - (lt ? 1u : 0u)) << 52);
  return ie_double((zero ? 0 : q) | ((uint64_t)sign << 32));
}

IE_FN double ie_div(double a, const IeDen& d) {
  bool ok;
  double q = ie_div_plain(a, d, ok);
  if (!ok) q = ie_div_slow(a, d.b);
  return q;
}

IE_FN double ie_div(double a, double b) { return ie_div(a, ie_den(b)); }

// two quotients by one divisor, side by side
IE_FN void ie_div2(double a0, double a1, const IeDen& d, double& q0, double& q1) {
  bool ok0, ok1;
  q0 = ie_div_plain(a0, d, ok0);
  q1 = ie_div_plain(a1, d, ok1);
  if (!(ok0 && ok1)) {
    q0 = ie_div_slow(a0, d.b);
    q1 = ie_div_slow(a1, d.b);
  }
}

IE_FN double ie_sqrt(double a) {
  const uint64_t x = ie_bits(a);
  const uint32_t e = (uint32_t)(x >> 52);
  const bool zero = (x << 1) == 0;
  const uint64_t s = ie_root((x & IE_MANTISSA) | IE_ONE, (e & 1u) == 0) + ((uint64_t)((e + 1021u) >> 1) << 52);
  double r = zero ? a : ie_double(s);
  if (!(zero || e - 1u < 2046u)) r = ie_sqrt_slow(a);  // negative, subnormal, infinite, NaN
  return r;
}

// The IEEE comparisons (false when an operand is NaN) from the bit patterns.
IE_FN int64_t ie_order(double a) {
  const int64_t x = (int64_t)ie_bits(a);
  return x < 0 ? (int64_t)(0x8000000000000000ull - (uint64_t)x) : x;
}
IE_FN bool ie_nan(double a) { return (ie_bits(a) << 1) > 0xffe0000000000000ull; }
IE_FN bool ie_lt(double a, double b) { return ie_order(a) < ie_order(b) && !ie_nan(a) && !ie_nan(b); }
IE_FN bool ie_le(double a, double b) { return ie_order(a) <= ie_order(b) && !ie_nan(a) && !ie_nan(b); }
// a <= b and a < b of operands with the sign bit clear
IE_FN bool ie_le_pos(double a, double b) { return ie_bits(a) <= ie_bits(b) && ie_bits(b) <= 0x7ff0000000000000ull; }
IE_FN bool ie_lt_pos(double a, double b) { return ie_bits(a) < ie_bits(b) && ie_bits(b) <= 0x7ff0000000000000ull; }
// a > 0
IE_FN bool ie_positive(double a) { return ie_bits(a) - 1ull < 0x7ff0000000000000ull; }
IE_FN double ie_abs(double a) { return ie_double(ie_bits(a) & 0x7fffffffffffffffull); }

// |a| in FP32, truncated (relative error under 2^-23); 0 below the FP32
// normal range, infinity above it and for NaN.  A conversion instruction
// would take the FP64 unit.
IE_FN uint32_t ie_float_bits(double a) {
  const uint64_t x = ie_bits(a);
  const uint32_t h = ((uint32_t)(x >> 32) & 0x7fffffffu) - 0x38000000u;  // exponent rebiased by 896
  const uint32_t f = (h << 3) | ((uint32_t)x >> 29);
  return (int32_t)h < 0x00100000 ? 0u : (h >= 0x0ff00000u ? 0x7f800000u : f);
}
IE_FN float ie_float(double a) { return IE_AS_FLOAT(ie_float_bits(a)); }
IE_FN float ie_float_signed(double a) {
  return IE_AS_FLOAT(ie_float_bits(a) | ((uint32_t)(ie_bits(a) >> 32) & 0x80000000u));
}

}  // namespace fc3dgpu
