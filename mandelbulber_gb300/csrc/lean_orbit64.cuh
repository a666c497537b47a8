// The Mandelbox orbit (formula 8, normal mode) of the FP64 policy, with the reference's
// results bit for bit at an eighth of the FP64 instructions of compute<double, 8, 0>.
//
// What bounds it: GB300's FP64 pipe, 20 SM cycles per warp instruction (exact64.cuh). The
// generic iteration (tglad_step) issues 61 of them; here the usual iteration issues 8, beside
// integer work of about as many cycles:
//   * The orbit needs r = sqrt(q), q = |z|^2, only inside the sphere fold's shell. The tests
//     r * r < mR2, r * r < fR2 and r > 1024 are monotone in q (square root and product round
//     monotonically), so each is q against a bound that the host derives exactly
//     (FractalT::boxQIn, boxQMid, boxQBail), and a comparison of positive doubles is one of
//     their bits: integer instructions. |x| > limit likewise.
//   * In the shell, r * r and fR2 / (r * r) come from integer multiplies (sqrt_squared and
//     div_exact, 33 SM cycles each in otherwise empty issue slots; on the pipe the root takes 156, its
//     square 20 and the quotient 90).
//   * With a scale and an inner fold factor that are powers of two (the usual 2 and 4) the
//     products are exact, so z * k * scale + c is one fused multiply-add. Other scales take the
//     two roundings.
//   * The fold against a power of two, the squares before the sphere fold and the shell's
//     products are integer too: moving them off the pipe took 2 M orbits of 15 iterations from
//     1.53 to 1.07 ms (fold 1.53 -> 1.33, products -> 1.17, squares -> 1.07). The bailout's
//     squares too: 25.3 -> 23.2 ms for a frame, whose stages have fewer active lanes and free issue
//     slots, but 1.07 -> 1.11 ms for that loop of full warps, which keeps them (FULL).
// Measured: 2,000,003 distances (N 15) 3.92 ms generic, 1.44 ms with the pipe for fold and
// products, 0.96 ms as it stands; a 481x271 Mandelbox frame 89.8 -> 22.6 ms.
// Not kept: leaving out the bailout test of the first five iterations, which a start point near
// the box cannot fail, made the loop slower in every form tried (1.17 -> 1.29 to 1.35 ms).
#pragma once

#include "exact64.cuh"
#include "kernel_params.h"

namespace mbgb {
namespace dev {

__device__ __forceinline__ bool abs_greater(const double x, const uint64_t bound) {
  return (f64_bits(x) & 0x7fffffffffffffffull) > bound;
}
// v with its sign flipped where x is negative
__device__ __forceinline__ double flip_sign(const double v, const double x) {
  return bits_f64(f64_bits(v) ^ (f64_bits(x) & 0x8000000000000000ull));
}

// |z|^2 in the reference's order: ((x x + y y) + z z), every operation rounded.
__device__ __forceinline__ double norm2_strict(const double x, const double y, const double z) {
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

// Distance r / |dr| at the bailout (q > boxQBail): integer forms within their domain.
__device__ __forceinline__ double box_dist_strict(const double q, const double dr) {
  if (f64_bits(q) >= 0x7ff0000000000000ull || f64_bits(dr) >= 0x7ff0000000000000ull)
    return __ddiv_rn(__dsqrt_rn(q), fabs(dr));
  return div_exact(sqrt_exact(q), dr);
}

// FULL: the caller's warps are full (a point cloud): the bailout's squares stay on the pipe.
template <bool FULL>
__device__ __forceinline__ double box_orbit_strict(const FractalT<double> &f, double x, double y, double z,
                                                   const double cx, const double cy, const double cz, const int N,
                                                   int &Lout, const double scale) {
  const uint64_t fl = f64_bits(f.mbFoldLimit), qIn = f64_bits(f.boxQIn), qMid = f64_bits(f.boxQMid),
                 qBail = f64_bits(f.boxQBail), far = f64_bits(f.boxFoldFar);
  const double fv = f.mbFoldValue, fR2 = __dmul_rn(f.mbFixedR, f.mbFixedR), k1 = f.boxK1;
  const uint64_t sb = f64_bits(scale);
  const bool pow2 = f.boxK1Pow2 && (sb & 0xfffffffffffffull) == 0 && (sb & 0x7fffffffffffffffull) >= 0x3ff0000000000000ull;
  const double ks1 = pow2 ? __dmul_rn(k1, scale) : scale;
  // box fold of one component: fold value - x beyond the limit (boxFoldFar: the integer form's
  // range, 0 where it does not apply)
  auto fold = [&](double &v) {
    const uint64_t av = f64_bits(v) & 0x7fffffffffffffffull;
    if (av > fl) v = av < far ? fold_pow2(fv, v) : __dsub_rn(flip_sign(fv, v), v);
  };
  double dr = 1.0;
  int L;
#pragma unroll 1
  for (L = 0; L < N; L++) {
    fold(x);
    fold(y);
    fold(z);
    const double q = __dadd_rn(__dadd_rn(square_int(x), square_int(y)), square_int(z));
    const uint64_t qb = f64_bits(q);
    double ks = scale;
    if (qb < qIn) {
      if (pow2) {
        ks = ks1;
      } else {
        x = __dmul_rn(x, k1);
        y = __dmul_rn(y, k1);
        z = __dmul_rn(z, k1);
        dr = __dmul_rn(dr, k1);
      }
    } else if (qb < qMid) {
      const double k = div_exact(fR2, sqrt_squared(q));
      x = mul_int(x, k);
      y = mul_int(y, k);
      z = mul_int(z, k);
      dr = mul_int(dr, k);
    }
    if (pow2) {
      x = __fma_rn(x, ks, cx);
      y = __fma_rn(y, ks, cy);
      z = __fma_rn(z, ks, cz);
      dr = __fma_rn(dr, fabs(ks), 1.0);
    } else {
      x = __dadd_rn(__dmul_rn(x, scale), cx);
      y = __dadd_rn(__dmul_rn(y, scale), cy);
      z = __dadd_rn(__dmul_rn(z, scale), cz);
      dr = __dadd_rn(__dmul_rn(dr, fabs(scale)), 1.0);
    }
    const double q2 = FULL ? norm2_strict(x, y, z)
                           : __dadd_rn(__dadd_rn(square_int(x), square_int(y)), square_int(z));
    if (f64_bits(q2) > qBail) {
      Lout = L;
      return box_dist_strict(q2, dr);
    }
  }
  Lout = N;
  return 0.0;
}

// Whether the orbit of a point may take box_orbit_strict: coordinates below 2^300 (no NaN, no
// overflow of their squares).
__device__ __forceinline__ bool box_strict_point(const double x, const double y, const double z) {
  const uint32_t lim = (uint32_t)(1023 + 300) << 20;
  return ((uint32_t)__double2hiint(x) & 0x7fffffffu) < lim && ((uint32_t)__double2hiint(y) & 0x7fffffffu) < lim &&
         ((uint32_t)__double2hiint(z) & 0x7fffffffu) < lim;
}

}  // namespace dev
}  // namespace mbgb
