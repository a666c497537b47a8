// Correctly rounded FP64 square root and quotient from 32-bit integer arithmetic.
//
// GB300's FP64 pipe takes one warp instruction per SM sub-partition every 76 cycles
// (measured: 152 SMs, 19.06 SM cycles per warp FMA whatever the number of active lanes), so
// an FP64 kernel leaves nine of ten issue slots empty, and a square root or a quotient costs
// a dozen such instructions. The functions here return the same IEEE results (round to
// nearest even) from integer multiplies and one FP32 special-function seed each, which run in
// those empty slots.
//
// Method: both are residual corrections of a short seed (Newton's iteration in fixed point):
// with y ~ 1/sqrt(x) or 1/d to 21 bits, s += y/2 (x - s^2) or q += y (n - d q) gains 20 bits a
// step, the residuals are exact modulo 2^64 (they are far smaller), and a last exact residual
// of the 53-bit result decides the rounding: x - R^2 against R, n - D Q against D/2. The
// results therefore do not depend on the seed's last bits.
//
// Domain: positive normal operands whose result is normal (the callers' ranges).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#ifndef __CUDA_ARCH__
#include <math.h>
#endif

namespace mbgb {
namespace dev {

__host__ __device__ __forceinline__ uint64_t f64_bits(const double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return b;
#endif
}
__host__ __device__ __forceinline__ double bits_f64(const uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}

// y x 2^23 for y = 1/sqrt(x) or 1/x of the float with bits `xb`, y in [0.5, 1]: the float sum
// 1 + y has ulp 2^-23, so its bits less 1.0's are the fixed-point value.
__host__ __device__ __forceinline__ uint32_t seed_rsqrt(const uint32_t xb) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(xb)));
  return __float_as_uint(1.0f + y) - 0x3f800000u;
#else
  float x, y;
  memcpy(&x, &xb, 4);
  y = 1.0f + 1.0f / sqrtf(x);
  uint32_t b;
  memcpy(&b, &y, 4);
  return b - 0x3f800000u;
#endif
}
__host__ __device__ __forceinline__ uint32_t seed_rcp(const uint32_t xb) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(xb)));
  return __float_as_uint(1.0f + y) - 0x3f800000u;
#else
  float x, y;
  memcpy(&x, &xb, 4);
  y = 1.0f + 1.0f / x;
  uint32_t b;
  memcpy(&b, &y, 4);
  return b - 0x3f800000u;
#endif
}

// sqrt(q) rounded to nearest: R is its 53-bit mantissa, `h` its exponent (R 2^(h - 52)), and
// X 2^104 - R^2 = t exactly, with q = X 4^h, X in [1, 4), A = X 2^60.
struct Sqrt64 {
  uint64_t R, A;
  int64_t t;
  int h;
};
__host__ __device__ __forceinline__ Sqrt64 sqrt_parts(const uint64_t qb, const uint32_t jitter = 0) {
  Sqrt64 r;
  const int e = (int)(qb >> 52) - 1023;
  const uint64_t m = (qb & 0xfffffffffffffull) | 0x10000000000000ull;
  const int odd = e & 1;
  r.h = (e - odd) >> 1;
  r.A = m << (8 + odd);
  const uint32_t xb = ((uint32_t)(127 + odd) << 23) | ((uint32_t)(m >> 29) & 0x7fffffu);
  const uint32_t y = seed_rsqrt(xb) + jitter;                       // 23 fraction bits
  const uint32_t s0 = (uint32_t)(((r.A >> 32) * (uint64_t)y) >> 21);   // 30 fraction bits
  const int32_t e0 = (int32_t)((int64_t)(r.A - (uint64_t)s0 * s0) >> 14);   // 46
  const uint64_t s1 = ((uint64_t)s0 << 16) + (uint64_t)(((int64_t)e0 * (int64_t)(int32_t)y) >> 24);   // 46
  const int32_t e1 = (int32_t)((int64_t)((r.A << 32) - s1 * s1) >> 26);   // 66
  uint64_t R = (s1 << 6) + (uint64_t)(((int64_t)e1 * (int64_t)(int32_t)y) >> 38);   // 52, within 1
  int64_t t = (int64_t)((r.A << 44) - R * R);                       // X 2^104 - R^2
  // (R + 1/2)^2 = R^2 + R + 1/4: R is the nearest iff -R < t <= R
  if (t > (int64_t)R) {
    t -= (int64_t)(2 * R + 1);
    R += 1;
  } else if (t <= -(int64_t)R) {
    t += (int64_t)(2 * R - 1);
    R -= 1;
  }
  r.R = R;
  r.t = t;
  return r;
}

// sqrt(q).
__host__ __device__ __forceinline__ double sqrt_exact(const double q, const uint32_t jitter = 0) {
  const Sqrt64 s = sqrt_parts(f64_bits(q), jitter);
  return bits_f64(((uint64_t)(s.h + 1022) << 52) + s.R);
}

// round(sqrt(q)^2) of the rounded square root: r * r for r = sqrt(q), from the residual
// (R^2 = X 2^104 - t) without a multiply.
__host__ __device__ __forceinline__ double sqrt_squared(const double q, const uint32_t jitter = 0) {
  const Sqrt64 s = sqrt_parts(f64_bits(q), jitter);
  uint64_t lo = s.A << 44, hi = s.A >> 20;   // X 2^104
  const uint64_t tl = (uint64_t)s.t;
  hi -= (uint64_t)(s.t >> 63) + (lo < tl ? 1u : 0u);
  lo -= tl;
  // the square lies in [2^104, 2^106]: 53 bits are left after sh places
  const int sh = 52 + (hi >> 41 ? 1 : 0) + (hi >> 42 ? 1 : 0);
  const uint64_t m = (hi << (64 - sh)) | (lo >> sh), rem = lo << (64 - sh);
  const uint64_t up = rem > 0x8000000000000000ull || (rem == 0x8000000000000000ull && (m & 1)) ? 1u : 0u;
  return bits_f64(((uint64_t)(2 * s.h + 1022 + sh - 52) << 52) + m + up);
}

// n / d.
__host__ __device__ __forceinline__ double div_exact(const double nd, const double dd, const uint32_t jitter = 0) {
  const uint64_t nb = f64_bits(nd), db = f64_bits(dd);
  uint64_t n = (nb & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint64_t d = (db & 0xfffffffffffffull) | 0x10000000000000ull;
  const int below = n < d ? 1 : 0;   // the quotient of the mantissas in [1, 2)
  n <<= below;
  const uint32_t y = seed_rcp(0x3f800000u | ((uint32_t)(d >> 29) & 0x7fffffu)) + jitter;   // 23 fraction bits
  const uint32_t q0 = (uint32_t)(((n >> 24) * (uint64_t)y) >> 23);                         // 28
  const int32_t e0 = (int32_t)((int64_t)((n << 28) - d * q0) >> 32);                       // 48
  const uint64_t q1 = ((uint64_t)q0 << 18) + (uint64_t)(((int64_t)e0 * (int64_t)(int32_t)y) >> 25);   // 46
  const int32_t e1 = (int32_t)((int64_t)((n << 46) - d * q1) >> 30);                       // 68
  uint64_t q = (q1 << 6) + (uint64_t)(((int64_t)e1 * (int64_t)(int32_t)y) >> 39);          // 52, within 1
  const int64_t t = (int64_t)((n << 52) - d * q);
  if (2 * t > (int64_t)d) q += 1;
  else if (2 * t < -(int64_t)d) q -= 1;
  const uint64_t sign = (nb ^ db) & 0x8000000000000000ull;
  const int ex = (int)((nb >> 52) & 0x7ff) - (int)((db >> 52) & 0x7ff) - below + 1022;
  return bits_f64((((uint64_t)ex << 52) + q) | sign);
}

// a * b (16 SM cycles a warp against the FP64 pipe's 20, and beside it).
__host__ __device__ __forceinline__ double mul_exact(const double a, const double b) {
  const uint64_t ab = f64_bits(a), bb = f64_bits(b);
  const uint64_t m = (ab & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint64_t k = (bb & 0xfffffffffffffull) | 0x10000000000000ull;
#ifdef __CUDA_ARCH__
  const uint64_t hi = __umul64hi(m << 11, k << 1), lo = (m << 11) * (k << 1);
#else
  const unsigned __int128 pr = (unsigned __int128)(m << 11) * (k << 1);
  const uint64_t hi = (uint64_t)(pr >> 64), lo = (uint64_t)pr;
#endif
  // the product x 2^12 lies in [2^116, 2^118): hi holds 53 or 54 bits, lo the rest
  const int big = (int)(hi >> 53);
  const uint64_t r = big ? hi >> 1 : hi;
  const uint64_t rest = big ? (hi << 63) | (lo >> 1) : lo;   // (the bit shifted out of lo is 0)
  const uint64_t up = rest > 0x8000000000000000ull || (rest == 0x8000000000000000ull && (r & 1)) ? 1u : 0u;
  const int ex = (int)((ab >> 52) & 0x7ff) + (int)((bb >> 52) & 0x7ff) - 1024 + big;
  return bits_f64((((uint64_t)ex << 52) + r + up) | ((ab ^ bb) & 0x8000000000000000ull));
}

#ifdef __CUDACC__
// The same for any operands: the integer forms where both operands lie in [2^-423, 2^377], so
// that every result is normal, the FP64 pipe elsewhere (zeros, huge and special values).
__device__ __forceinline__ bool int_range(const double a) {
  return ((uint32_t)(f64_bits(a) >> 52) & 0x7ffu) - 600u <= 800u;
}
// a * b with b in [2^-400, 2^400]
__device__ __forceinline__ double mul_int(const double a, const double b) {
  return int_range(a) ? mul_exact(a, b) : __dmul_rn(a, b);
}
// a * b for any two operands
__device__ __forceinline__ double mul2_int(const double a, const double b) {
  return int_range(a) && int_range(b) ? mul_exact(a, b) : __dmul_rn(a, b);
}
// 2 a
__device__ __forceinline__ double twice_int(const double a) {
  return int_range(a) ? bits_f64(f64_bits(a) + 0x10000000000000ull) : __dadd_rn(a, a);
}
__device__ __forceinline__ double square_int(const double a) {
  return int_range(a) ? mul_exact(a, a) : __dmul_rn(a, a);
}
__device__ __forceinline__ double div_int(const double n, const double d) {
  return int_range(n) && int_range(d) ? div_exact(n, d) : __ddiv_rn(n, d);
}
__device__ __forceinline__ double sqrt_int(const double q) {   // q >= 0
  return int_range(q) ? sqrt_exact(q) : __dsqrt_rn(q);
}
#endif

// copysign(p, x) - x for a power of two p and |x| > p / 2: an exact difference (both are
// multiples of the smaller one's last bit and the result is no longer than x), formed in units
// of x's last bit. |x| < 2^50 p.
__device__ __forceinline__ double fold_pow2(const double p, const double x) {
  const uint64_t b = f64_bits(x);
  const int ex = (int)(b >> 52) & 0x7ff, up = (int)(f64_bits(p) >> 52) - ex;
  const int64_t d = (int64_t)(1ull << (52 + up)) - (int64_t)((b & 0xfffffffffffffull) | 0x10000000000000ull);
  if (d == 0) return 0.0;
  const uint64_t a = d < 0 ? (uint64_t)-d : (uint64_t)d;
#ifdef __CUDA_ARCH__
  const int lz = __clzll((long long)a);   // 11 or more
#else
  const int lz = __builtin_clzll(a);
#endif
  const uint64_t r = ((uint64_t)(ex + 10 - lz) << 52) + (a << (lz - 11));
  return bits_f64(r | (((uint64_t)d ^ b) & 0x8000000000000000ull));
}

}  // namespace dev
}  // namespace mbgb
