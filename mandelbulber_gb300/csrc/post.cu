// Post-processing of a rendered frame on the device: CompileImage (src/cimage.cpp:132-214)
// into the 16-bit image, the screen-space ambient occlusion pass PostRendering_SSAO /
// ThreadSSAO (src/image.cpp:249-478) and the depth of field PostRendering_DOF
// (src/image.cpp:57-206), which the reference runs in that order after the render when
// post_SSAO_enabled / post_DOF_enabled are set (src/Render3D.cpp:1093-1106).
//
// Built with --fmad=false: the FP64 SSAO and the compile step follow the reference's
// double-precision operation order, so results match it to the last bit except where
// CUDA's atan / tanhf round differently from the host's libm.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <utility>
#include <vector>

#include "exact64.cuh"
#include "mbgb.h"
#include "mbgb_internal.h"

namespace {

constexpr double kPi = 3.14159265358979323846;

// CalculatePixel (src/cimage.cpp:132-171): brightness, contrast, optional tanh, clamp,
// x 65535 and the gamma table; without one, gamma 1, whose entry (int)(i / 65536 x 65535) is
// i - 1 (0 for i = 0).
__global__ void compile16_kernel(const float *__restrict__ image_float, int64_t n, double brightness,
                                 double contrast, int hdr, const int *__restrict__ gamma,
                                 uint16_t *__restrict__ image16) {
  // brightness and contrast 1 without HDR change no value above 2^-29 (v - 0.5 + 0.5 is exact there,
  // and smaller ones end as 0): the 24-bit product by 65535 is then one of integers
  const bool plain = brightness == 1.0 && contrast == 1.0 && !hdr;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n; i += (int64_t)gridDim.x * blockDim.x) {
    if (plain) {
      const float u = image_float[i];
      uint32_t r = 0;   // negative, NaN
      if (u >= 1.0f) {
        r = 65535u;
      } else if (u > 2e-6f) {
        const uint32_t b = __float_as_uint(u);
        r = (uint32_t)(((uint64_t)((b & 0x7fffffu) | 0x800000u) * 65535u) >> (150u - (b >> 23)));
      }
      image16[i] = gamma ? (uint16_t)gamma[r] : (uint16_t)(r ? r - 1 : 0);
      continue;
    }
    float v = (float)((double)image_float[i] * brightness);
    v = (float)(((double)v - 0.5) * contrast + 0.5);
    if (v < 0.0f) v = 0.0f;
    if (hdr) v = (float)tanh((double)v);   // the host's tanhf, to the float it rounds to
    if (v > 1.0f) v = 1.0f;
    const unsigned short q = (unsigned short)((double)v * 65535.0);
    image16[i] = gamma ? (uint16_t)gamma[q] : (uint16_t)(q ? q - 1 : 0);
  }
}

// One splat of PostRendering_DOF (src/image.cpp:148-182): the pixel at (x, y) spreads its
// original RGB16 / alpha over the pixels within `size` at opacity (blur - r) / factor.
struct DofSplat {
  int x, y, size, centre;   // centre: the pixel index of (x, y)
  double blur, factor;
};

constexpr int kDofTile = 16;

// Each CTA owns one 16 x 16 tile; each thread owns one pixel of it and applies, in the
// splat order, every splat of the tile's list that covers its pixel. A pixel's value after
// the pass is the reference's sequential in-place fold: splats change only pixels they cover
// and read only the frame's original values at their centres.
__global__ void dof_kernel(const DofSplat *__restrict__ splats, const int64_t *__restrict__ tileStart,
                           const int *__restrict__ tileList, const int tilesX, const int width, const int height,
                           const uint16_t *__restrict__ image0, const uint16_t *__restrict__ alpha0,
                           uint16_t *__restrict__ image16, uint16_t *__restrict__ alpha) {
  const int tile = blockIdx.x;
  const int xx = (tile % tilesX) * kDofTile + (int)(threadIdx.x % kDofTile);
  const int yy = (tile / tilesX) * kDofTile + (int)(threadIdx.x / kDofTile);
  if (xx >= width || yy >= height) return;
  const int64_t q = (int64_t)yy * width + xx;
  uint16_t v[3] = {image16[3 * q + 0], image16[3 * q + 1], image16[3 * q + 2]};
  uint16_t a = alpha[q];
  for (int64_t k = tileStart[tile]; k < tileStart[tile + 1]; k++) {
    const DofSplat sp = splats[tileList[k]];
    const int dx = xx - sp.x, dy = yy - sp.y;
    if (dx < -sp.size || dx > sp.size || dy < -sp.size || dy > sp.size) continue;
    const double r = (double)sqrtf((float)dx * dx + dy * dy);
    double op = (sp.blur - r) / sp.factor;
    if (op > 1.0) op = 1.0;
    if (op < 0.0) op = 0.0;
    if (op > 0.0) {
      const double opN = 1.0 - op;
      for (int c = 0; c < 3; c++) v[c] = (uint16_t)(v[c] * opN + image0[3 * (int64_t)sp.centre + c] * op);
      a = (uint16_t)(a * opN + alpha0[sp.centre] * op);
    }
  }
  image16[3 * q + 0] = v[0];
  image16[3 * q + 1] = v[1];
  image16[3 * q + 2] = v[2];
  alpha[q] = a;
}

// Screen position of a pixel sample (x, y may be fractional) at depth z in the plane
// the SSAO horizon search works in; perspective types as in ThreadSSAO. For the fish eye
// the centre pixel skips the projection where its radius is 0, while the samples test the
// search radius instead (always >= 1), as ThreadSSAO does.
template <typename T>
__device__ __forceinline__ void ssao_position(const int ptype, const T fx, const T fy, const T w, const T h,
                                              const T aspect, const T fov, const T z, const bool centre, T &ox,
                                              T &oy) {
  if (ptype == 1) {   // fish eye
    const T x2 = T(kPi) * (fx / w - T(0.5)) * aspect;
    const T y2 = T(kPi) * (fy / h - T(0.5));
    const T r = sqrt(x2 * x2 + y2 * y2);
    ox = x2;
    oy = y2;
    if (!centre || r != T(0)) {
      ox = x2 / r * sin(r * fov) * z;
      oy = y2 / r * sin(r * fov) * z;
    }
  } else if (ptype == 2) {   // equirectangular
    const T x2 = T(kPi) * (fx / w - T(0.5)) * aspect;
    const T y2 = T(kPi) * (fy / h - T(0.5));
    ox = sin(fov * x2) * cos(fov * y2) * z;
    oy = sin(fov * y2) * z;
  } else {
    ox = (fx / w - T(0.5)) * aspect;
    oy = (fy / h - T(0.5));
  }
}

// ThreadSSAO (src/image.cpp:249-417) for one pixel per thread: `quality` directions, each
// searching quality - 1 samples at radius r^2 * width / (2 quality^2) for the steepest
// horizon, ambient = mean over directions of 0.5 - atan(slope) / pi; the pixel's 16-bit
// value gains colour * ambient * intensity * (1 - opacity), clamped to 65535.
template <typename T>
__global__ void ssao_kernel(const float *__restrict__ zbuf, const uint16_t *__restrict__ opacity,
                            const uint8_t *__restrict__ colour, uint16_t *__restrict__ image16, const int width,
                            const int height, const T persp, const int quality, const int ptype, const T intensity,
                            const T *__restrict__ cs, const T *__restrict__ sn) {
  const int64_t n = (int64_t)width * height;
  const T w = (T)width, h = (T)height;
  const T scale = (T)width / (T)(quality * quality) / T(2);
  const T aspect = (T)width / (T)height;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % width), y = (int)(i / width);
    const T z = (T)zbuf[i];
    const T op = (T)opacity[i] / T(65535);
    T total = T(0);
    if (z < T(1e19)) {
      T x2, y2;
      ssao_position<T>(ptype, (T)x, (T)y, w, h, aspect, persp, z, true, x2, y2);
      if (ptype != 1 && ptype != 2) {
        x2 = x2 * z * persp;
        y2 = y2 * z * persp;
      }
      T ambient = T(0);
      for (int a = 0; a < quality; a++) {
        const T ca = cs[a], sa = sn[a];
        T maxDiff = T(-1e50);
        for (T r = T(1); r < (T)quality; r += T(1)) {
          const T rr = r * r * scale;
          const T xx = (T)x + rr * ca;
          const T yy = (T)y + rr * sa;
          if ((int)xx == x && (int)yy == y) continue;
          if (xx < T(0) || xx > (T)(width - 1) || yy < T(0) || yy > (T)(height - 1)) continue;
          const T z2 = (T)zbuf[(int64_t)(int)yy * width + (int)xx];
          T xx2, yy2;
          ssao_position<T>(ptype, xx, yy, w, h, aspect, persp, z2, false, xx2, yy2);
          if (ptype != 1 && ptype != 2) {
            xx2 = xx2 * (z2 * persp);
            yy2 = yy2 * (z2 * persp);
          }
          const T dx = xx2 - x2;
          const T dy = yy2 - y2;
          const T dz = z2 - z;
          const T dr = sqrt(dx * dx + dy * dy);
          const T diff = -dz / dr;
          if (diff > maxDiff) maxDiff = diff;
        }
        const T maxAngle = atan(maxDiff);
        ambient += -maxAngle / T(kPi) + T(0.5);
      }
      total = ambient / (T)quality;
      if (total < T(0)) total = T(0);
    }
    for (int c = 0; c < 3; c++) {
      T v = (T)image16[3 * i + c] + T(65535) * (T)colour[3 * i + c] / T(256) * total * intensity * (T(1) - op);
      if (v > T(65535)) v = T(65535);
      image16[3 * i + c] = (uint16_t)(unsigned short)v;
    }
  }
}

// Pairs of floats (value hi + lo, about 46 bits) for the horizon angles: Knuth's and Dekker's
// error-free sums, products with the residual of a fused multiply-add.
struct F2 {
  float h, l;
};
__device__ __forceinline__ F2 f2_quick(const float a, const float b) {   // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ F2 f2_sum(const float a, const float b) {     // exact
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ F2 f2_add(const F2 a, const F2 b) {
  const F2 s = f2_sum(a.h, b.h);
  return f2_quick(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ F2 f2_mul(const F2 a, const F2 b) {
  const float p = __fmul_rn(a.h, b.h);
  return f2_quick(p, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.h, -p))));
}
__device__ __forceinline__ F2 f2_of(const double v) {
  const float h = (float)v;
  return {h, (float)(v - (double)h)};
}

// One sample of the flat projection's horizon search (shared by every pixel): direction a,
// radius r. A pixel at integer x samples column trunc(fl(x + off)). With off = k + f, k integer
// and f in [1e-9, 1 - 1e-9], the rounded sum stays strictly between x + k and x + k + 1: column
// x + k, inside the picture up to width - 2. Other offsets (cos(pi / 2) = 6e-17 times a radius) are
// off = k + g, |g| < 1e-9, and the sum's rounding decides (near_column).
struct __align__(16) SsaoSample {
  float cx, cy;         // the offset in the projection plane at depth 1, off / w aspect persp
  uint32_t cc;          // float |cx| + |cy| rounded up to a multiple of 4 units; its low bits: kNearX,
                        // kNearY
  int16_t kx, ky;       // k of the offset
};
constexpr uint32_t kNearX = 1, kNearY = 2;
struct __align__(16) SsaoOffset {
  double x, y;          // r^2 scale cos, r^2 scale sin
  float cxl, cyl;       // what the floats cx, cy leave
  float gx, gy;         // g of the offset, its magnitude rounded up
};

// Column (or row) of fl(b + g), b = x + k, |g| < 1e-9, and whether it lies in [0, last]: the sum
// rounds to b where |g| is at most half the spacing of doubles on its side of b, 2^(e - 53) for b
// in [2^e, 2^(e+1)) and half that below a power of two (ties go to b, whose last bit is 0). A
// power of two compares with |g| as with |g| rounded up.
__device__ __forceinline__ bool near_column(const int b, const float g, const int last, int &at) {
  at = b;
  if (b < 0 || b > last) return false;
  if (g == 0.0f) return true;
  if (b == 0) return g > 0.0f && last > 0;
  const int e = 31 - __clz(b);
  const float half = __uint_as_float((uint32_t)(127 + e - 53) << 23);
  if (g < 0.0f) {
    if (-g > ((b & (b - 1)) ? half : 0.5f * half)) at = b - 1;
    return true;
  }
  return b < last || g <= half;
}

__global__ void ssao_table_kernel(SsaoSample *__restrict__ t, SsaoOffset *__restrict__ o, const int width,
                                  const int height, const double persp, const int quality,
                                  const double *__restrict__ cs, const double *__restrict__ sn) {
  const double w = (double)width, h = (double)height;
  const double scale = w / (double)(quality * quality) / 2.0, aspect = w / h;
  const int n = quality * (quality - 1);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int a = i / (quality - 1);
    const double r = (double)(i % (quality - 1) + 1), rr = r * r * scale;
    const double x = rr * cs[a], y = rr * sn[a];
    double kx = floor(x), ky = floor(y), gx = x - kx, gy = y - ky;
    const F2 cx = f2_of(x / w * aspect * persp), cy = f2_of(y / h * persp);
    uint32_t cc = (__float_as_uint(fabsf(cx.h) + fabsf(cy.h)) | 3u) + 1u;
    auto near = [&](const double v, double &k, double &g, const uint32_t flag) {
      if (g >= 1e-9 && g <= 1.0 - 1e-9) return;
      cc |= flag;
      k = rint(v);
      g = v - k;   // exact: v is next to k
    };
    near(x, kx, gx, kNearX);
    near(y, ky, gy, kNearY);
    t[i] = SsaoSample{cx.h, cy.h, cc, (int16_t)kx, (int16_t)ky};
    o[i] = SsaoOffset{x, y, cx.l, cy.l, (float)copysign((double)__double2float_ru(fabs(gx)), gx),
                      (float)copysign((double)__double2float_ru(fabs(gy)), gy)};
  }
}

// atan(k / 16), k = 0 .. 16, and pi / 2.
__device__ const F2 kAtan16[17] = {
    {0.0f, 0.0f}, {0.06241881102323532f, -1.0272779293885037e-09f}, {0.12435499578714371f, -1.240382241363136e-09f},
    {0.18534794449806213f, 5.49763257140512e-09f}, {0.244978666305542f, -3.1786777654474463e-09f}, {0.30288487672805786f, -8.353086222712136e-09f},
    {0.3587706685066223f, 1.7639498750554594e-09f}, {0.4124104380607605f, 3.5366267692182873e-09f}, {0.46364760398864746f, 5.01215868808913e-09f},
    {0.5123894810676575f, -2.0756919738573743e-08f}, {0.5585992932319641f, 2.2111597886009804e-08f}, {0.6022873520851135f, -5.950149262190507e-09f},
    {0.6435011029243469f, 5.868937336117597e-09f}, {0.6823165416717529f, 1.3202995141625706e-08f}, {0.7188299894332886f, 1.0188335508587443e-08f},
    {0.7531512975692749f, -1.660708015549517e-08f}, {0.7853981852531433f, -2.1855694143368964e-08f}};
constexpr F2 kHalfPi{1.5707963705062866f, -4.371138828673793e-08f};

// atan(t / d) for d > 0, both in [1e-10, 1e10] or t = 0, to 4e-12: the ratio n / m <= 1 of the two
// is turned by the nearest k / 16, s = (n - c m) / (m + c n) with |s| <= 1/32 + an ulp, and
// atan(s) is its series to s^7.
__device__ __forceinline__ F2 f2_atan(const F2 t, const F2 d) {
  const bool neg = t.h < 0.0f;
  const F2 u = neg ? F2{-t.h, -t.l} : t;
  const bool swap = u.h > d.h;
  const F2 n = swap ? d : u, m = swap ? u : d;
  const int k = __float2int_rn(16.0f * __fdividef(n.h, m.h));
  const float c = (float)k * 0.0625f;
  const F2 num = f2_add(n, f2_mul(F2{-c, 0.0f}, m)), den = f2_add(m, f2_mul(F2{c, 0.0f}, n));
  const float inv = __fdividef(1.0f, den.h), s0 = __fmul_rn(num.h, inv);
  const float s1 = __fmul_rn(__fadd_rn(__fmaf_rn(-s0, den.h, num.h), __fmaf_rn(-s0, den.l, num.l)), inv);
  const float ss = __fmul_rn(s0, s0);
  const float series = __fmul_rn(__fmul_rn(s0, ss), __fmaf_rn(ss, __fmaf_rn(ss, -1.0f / 7.0f, 0.2f), -1.0f / 3.0f));
  F2 r = f2_add(kAtan16[k], f2_add(F2{s0, s1}, F2{series, 0.0f}));
  if (swap) r = f2_add(kHalfPi, F2{-r.h, -r.l});
  return neg ? F2{-r.h, -r.l} : r;
}

// Error of the sum of a pixel's `quality` angles in pairs of floats: f2_add's three roundings of low
// parts are 2^-48 of its operands each, so the addition of angle i errs by 3 x 2^-48 (i + 1) pi / 2,
// 8.4e-15 q^2 + 2.5e-14 q in all.
__host__ __device__ inline double ssao_sum_error(const int quality) { return (1e-12 + 1e-14 * quality) * quality; }

// A sample's slope from a pixel at plane position (ax, ay) of depth zs 2^20, aa = |ax| + |ay|:
// lo <= slope <= up, infinite where FP32 does not tell (ssao_flat_kernel).
constexpr float kSsaoScale = 9.5367431640625e-07f;   // 2^-20
__device__ __forceinline__ void ssao_bracket(const SsaoSample &s, const float ax, const float ay, const float aa,
                                             const float zs, const float z2, float &lo, float &up) {
  const float t = fmaf(-z2, kSsaoScale, zs), cc = __uint_as_float(s.cc);
  const float dx = fmaf(ax + s.cx, -t, s.cx * zs), dy = fmaf(ay + s.cy, -t, s.cy * zs);
  const float inv = rsqrtf(fmaf(dx, dx, dy * dy)), slope = t * inv;
  const float e = fmaf(aa + cc, fabsf(t), cc * zs);
  const float rel = fmaf(e, 4.8e-7f * inv, 4e-6f), d = 1.15f * fabsf(slope) * rel;
  const bool known = rel < 0.1f && fabsf(slope) < 1e30f;   // (false for NaN)
  lo = known ? slope - d : -INFINITY;
  up = known ? slope + d : INFINITY;
}

// The depth from which a pixel's slopes are bracketed. Below it the squares of plane distances
// d = |c| z 2^-20 and less are subnormal floats, whose roundings (2 x 2^-150, so 7e-46 / d^2 of 1 / d)
// rel does not hold: known brackets have d > 4.8e-6 E, E = |c| z 2^-20, and leave 0.04 rel >=
// 0.04 x 4.8e-7 E / d, which covers them for E >= 9e-17. A sample's offset c is |persp| aspect /
// (2 quality^2) at least; the limit keeps E at twice that.
inline float ssao_least_depth(const int quality, const double persp, const double aspect) {
  return (float)std::max(1e-6, 4e-10 * quality * quality / (fabs(persp) * aspect));
}

// The flat horizon search's inputs and outputs. `open` receives the pixels that the FP32 pass
// leaves to ssao_exact_kernel, `opens` their number.
struct SsaoArgs {
  const float *zbuf;
  const uint16_t *opacity;
  const uint8_t *colour;
  uint16_t *image16;
  int width, height, quality;
  float zMin;                  // ssao_least_depth
  double persp, intensity;
  const SsaoSample *samples;   // [quality][quality - 1]
  const SsaoOffset *offsets;
  uint32_t *opens;
  uint32_t *open;
};

// Whether a sample of the pixel (x, y) lies inside the picture and off the pixel itself; its index.
__device__ __forceinline__ bool ssao_sample(const SsaoArgs &g, const SsaoSample &s, const int i, const int x,
                                            const int y, int &at) {
  int xi = x + s.kx, yi = y + s.ky;
  bool ok = xi >= 0 && xi <= g.width - 2 && yi >= 0 && yi <= g.height - 2;
  if (s.cc & (kNearX | kNearY)) {   // the same for every pixel: uniform
    const bool inX = (s.cc & kNearX) ? near_column(xi, g.offsets[i].gx, g.width - 1, xi) : xi >= 0 && xi <= g.width - 2;
    const bool inY = (s.cc & kNearY) ? near_column(yi, g.offsets[i].gy, g.height - 1, yi) : yi >= 0 && yi <= g.height - 2;
    ok = inX && inY;
  }
  ok = ok && !(xi == x && yi == y);
  at = (ok ? yi : y) * g.width + (ok ? xi : x);
  return ok;
}

// ThreadSSAO for the flat projection, the bytes of ssao_kernel<double>.
//
// What bounds it: in double the FP64 pipe (exact64.cuh): a sample's slope takes three quotients
// and a root there, 870 SM cycles a warp, a direction's atan 800. The output is 16 bits, so the
// horizon angles are formed in FP32 with proven errors, and only a pixel whose error interval
// holds a whole number is left to ssao_exact_kernel.
//   * Per direction a first pass brackets every sample's slope, lo <= slope <= up, in plain FP32:
//     with A(x) = (x / w - 1/2) aspect persp the plane distance is dx = A(xx) dz + c z (c the
//     offset's, dz the depth difference), whose FP32 error is below
//     e = 2^-21 ((|A(x)| + |c|) |dz| + |c z|); with y = 1 / distance the slope's relative error is
//     e y and 4e-6 for the root and the products. Where the largest lo passes every other sample's
//     up, that sample is the steepest for certain. Depths are scaled by 2^-20, which keeps the
//     squares of the background's 1e20 finite and those of 1e-6 normal.
//   * Its angle (or, where it is not certain, that of every sample whose bracket reaches the
//     largest lo) is computed in pairs of floats: distance error 2^-21 e, atan to 4e-12. To
//     these the double form's own rounding is added, 2^-49 of the plane positions.
//   * Columns and rows come from integers and a sample is one 16-byte load (SsaoSample). (An
//     instruction of the FP64 pipe costs its 20 cycles even with no lane active: the pass has none.)
// What bounds it now is the first pass's issue rate, about 40 instructions a sample.
// 1920x1080, quality 20, with the 16-bit step: every slope in double 70.6 ms, the steepest only
// in double 5.65 ms, as it stands 2.30 ms.
__global__ void __launch_bounds__(128) ssao_flat_kernel(const __grid_constant__ SsaoArgs g) {
  const int64_t n = (int64_t)g.width * g.height;
  const double w = (double)g.width, h = (double)g.height, aspect = w / h;
  const int steps = g.quality - 1;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % g.width), y = (int)(i / g.width);
    const float zf = g.zbuf[i];
    double total = 0.0, error = 0.0;
    if ((double)zf < 1e19) {
      if (!(zf > g.zMin && zf < 1e6f && g.intensity >= 0.0)) {   // outside the forms' range: no pass
        g.open[atomicAdd(g.opens, 1u)] = (uint32_t)i;
        continue;
      }
      const F2 axp = f2_of((mbgb::dev::div_int((double)x, w) - 0.5) * aspect * g.persp);
      const F2 ayp = f2_of((mbgb::dev::div_int((double)y, h) - 0.5) * g.persp);
      const float aa = fabsf(axp.h) + fabsf(ayp.h);
      bool open = !(aa < 1e3f);
      const float zs = zf * kSsaoScale;
      // a sample's angle and the bound of its error
      auto angle = [&](const SsaoSample &s, const int at, const float z2f, float &err) {
        // the background's depth is 1e20: the slope does not change with the scale
        const float scale = fabsf(z2f) > 1e6f ? 2.8421709430404007e-14f : 1.0f;   // 2^-45
        const float z2 = z2f * scale, z1 = zf * scale, cc = __uint_as_float(s.cc);
        const F2 dz = f2_sum(z2, -z1), z{z1, 0.0f}, cx{s.cx, g.offsets[at].cxl}, cy{s.cy, g.offsets[at].cyl};
        const F2 dx = f2_add(f2_mul(f2_add(axp, cx), dz), f2_mul(cx, z));
        const F2 dy = f2_add(f2_mul(f2_add(ayp, cy), dz), f2_mul(cy, z));
        const F2 q = f2_add(f2_mul(dx, dx), f2_mul(dy, dy));
        const float inv = rsqrtf(q.h), r0 = __fmul_rn(q.h, inv);
        const F2 dr = f2_quick(r0, __fmul_rn(__fmul_rn(0.5f, inv), __fadd_rn(__fmaf_rn(-r0, r0, q.h), q.l)));
        if (!(dr.h > 1e-10f && fabsf(dz.h) < 1e7f)) open = true;
        const float e = 4.8e-7f * fmaf(aa + cc, fabsf(dz.h), cc * z1);
        err = 4e-12f + __fdividef(fmaf(e, 4.8e-7f, 1.8e-15f * (aa + cc) * (z1 + fabsf(z2))), dr.h);
        return f2_atan(F2{-dz.h, -dz.l}, dr);
      };
      F2 sum{0.0f, 0.0f};
      float errSum = 0.0f;
      for (int a = 0; a < g.quality; a++) {
        const int first = a * steps;
        float bestLo = -INFINITY, bestUp = -INFINITY, otherUp = -INFINITY;
        int best = -1;
#pragma unroll 4
        for (int r = 0; r < steps; r++) {
          const SsaoSample s = g.samples[first + r];
          int at;
          const bool ok = ssao_sample(g, s, first + r, x, y, at);
          float lo, up;
          ssao_bracket(s, axp.h, ayp.h, aa, zs, g.zbuf[at], lo, up);
          lo = ok ? lo : -INFINITY;
          up = ok ? up : -INFINITY;
          const bool better = lo > bestLo;
          otherUp = fmaxf(otherUp, better ? bestUp : up);
          bestLo = better ? lo : bestLo;
          bestUp = better ? up : bestUp;
          best = better ? r : best;
        }
        F2 top{-kHalfPi.h, -kHalfPi.l};   // no sample: the slope -1e50
        float err = 0.0f;
        int at;
        if (best >= 0 && otherUp < bestLo) {
          const SsaoSample s = g.samples[first + best];
          ssao_sample(g, s, first + best, x, y, at);
          top = angle(s, first + best, g.zbuf[at], err);
        } else if (otherUp > -INFINITY) {
          for (int r = 0; r < steps; r++) {
            const SsaoSample s = g.samples[first + r];
            if (!ssao_sample(g, s, first + r, x, y, at)) continue;
            const float z2 = g.zbuf[at];
            float lo, up, er;
            ssao_bracket(s, axp.h, ayp.h, aa, zs, z2, lo, up);
            if (!(up >= bestLo)) continue;
            const F2 t = angle(s, first + r, z2, er);
            err = fmaxf(err, er);
            if (t.h > top.h || (t.h == top.h && t.l > top.l)) top = t;
          }
        }
        sum = f2_add(sum, top);
        errSum += err;
      }
      // the mean of 1/2 - angle / pi, and its error with that of the summation
      const double per = 1.0 / (kPi * g.quality);
      total = 0.5 - ((double)sum.h + (double)sum.l) * per;
      error = ((double)errSum * 1.001 + ssao_sum_error(g.quality)) * per;
      if (open || !(error < 1e-3)) error = 2.0;
    }
    const double op = (double)g.opacity[i] / 65535.0;
    const double gain = 65535.0 / 256.0 * g.intensity * (1.0 - op);
    const double lowT = fmax(total - error, 0.0), highT = fmax(total + error, 0.0);
    // (an error of 0 is the background's: its term is exactly 0)
    bool settled = error < 1.0;
    uint16_t out[3];
    for (int c = 0; c < 3; c++) {
      const uint16_t was = g.image16[3 * i + c];
      const double base = (double)was, k = error == 0.0 ? 0.0 : gain * (double)g.colour[3 * i + c];
      const double lo = fmin(base + k * lowT - 1e-9, 65535.0), hi = fmin(base + k * highT + 1e-9, 65535.0);
      out[c] = k > 0.0 ? (uint16_t)(unsigned short)hi : was;
      if (k > 0.0 && (uint16_t)(unsigned short)fmax(lo, 0.0) != out[c]) settled = false;
    }
    if (settled) {
      for (int c = 0; c < 3; c++) g.image16[3 * i + c] = out[c];
    } else {
      g.open[atomicAdd(g.opens, 1u)] = (uint32_t)i;
    }
  }
}

// The pixels that ssao_flat_kernel leaves open, every slope in double as ThreadSSAO forms it (the
// values of ssao_kernel<double> bit for bit): a lane takes a direction (every 32nd of more than 32),
// and the directions' terms are summed in the reference's order. A warp holds as many pixels as
// leave a lane to each direction: with one each, a frame whose depths all lie below the FP32 forms'
// range (a camera a millionth from the surface) took longer than ssao_kernel<double>: 1024x768 at
// quality 4 / 6 / 10 / 20 6.7 / 8.5 / 12.1 / 21.8 ms against 1.33 / 2.84 / 7.7 / 30.4, as it stands
// 0.88 / 2.13 / 5.9 / 20.8.
__global__ void __launch_bounds__(128) ssao_exact_kernel(const __grid_constant__ SsaoArgs g) {
  using mbgb::dev::div_int;
  using mbgb::dev::sqrt_int;
  const uint32_t n = *g.opens;
  const double w = (double)g.width, h = (double)g.height, aspect = w / h;
  const int lane = threadIdx.x & 31, steps = g.quality - 1;
  int lanes = 32;   // of a pixel
  while (lanes / 2 >= g.quality) lanes /= 2;
  const uint32_t per = 32u / lanes, own = (uint32_t)lane / lanes;
  const int sub = lane & (lanes - 1);
  const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t k0 = warp * per; k0 < n; k0 += warps * per) {
    const bool valid = k0 + own < n;   // (else the warp's first pixel again, unwritten)
    const int64_t i = g.open[valid ? k0 + own : k0];
    const int x = (int)(i % g.width), y = (int)(i / g.width);
    const double z = (double)g.zbuf[i];
    double ambient = 0.0;
    const double x2 = (div_int((double)x, w) - 0.5) * aspect * z * g.persp;
    const double y2 = (div_int((double)y, h) - 0.5) * z * g.persp;
    for (int a0 = 0; a0 < g.quality; a0 += lanes) {
      double term = 0.0;
      if (a0 + sub < g.quality) {
        const int first = (a0 + sub) * steps;
        double maxDiff = -1e50;
        for (int r = 0; r < steps; r++) {
          int at;
          if (!ssao_sample(g, g.samples[first + r], first + r, x, y, at)) continue;
          const double xx = (double)x + g.offsets[first + r].x, yy = (double)y + g.offsets[first + r].y;
          const double z2 = (double)g.zbuf[at], q = z2 * g.persp;
          const double dx = (div_int(xx, w) - 0.5) * aspect * q - x2;
          const double dy = (div_int(yy, h) - 0.5) * q - y2;
          const double diff = div_int(-(z2 - z), sqrt_int(dx * dx + dy * dy));
          if (diff > maxDiff) maxDiff = diff;
        }
        term = div_int(-atan(maxDiff), kPi) + 0.5;
      }
      for (int l = 0; l < lanes && a0 + l < g.quality; l++) ambient += __shfl_sync(0xffffffffu, term, l, lanes);
    }
    double total = ambient / (double)g.quality;
    if (total < 0.0) total = 0.0;
    if (!valid) continue;
    for (int c = sub; c < 3; c += lanes) {
      const double op = (double)g.opacity[i] / 65535.0;
      double v = (double)g.image16[3 * i + c] +
                 65535.0 * (double)g.colour[3 * i + c] / 256.0 * total * g.intensity * (1.0 - op);
      if (v > 65535.0) v = 65535.0;
      g.image16[3 * i + c] = (uint16_t)(unsigned short)v;
    }
  }
}

int grid_for(int64_t work, int block) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t want = (work + block - 1) / block;
  const int64_t cap = (int64_t)(sms > 0 ? sms : 1) * 16;
  return (int)(want < cap ? (want > 0 ? want : 1) : cap);
}

}  // namespace

namespace mbgb {

// CompileImage on the device (gamma table from the host's pow, as CalculateGammaTable).
mbgb_status compile16_device(const mbgb_scene &scene, const float *image_float, int width, int height,
                             uint16_t *image16, int *gamma_dev, cudaStream_t s) {
  // gamma 1 (the default) needs no table: pow(x, 1) is x, and its 65536 calls on the host with
  // the copy took 1.9 ms, several times the kernel
  const bool table = scene.imageGamma != 1.0;
  std::vector<int> gamma(table ? 65536 : 0);
  for (size_t i = 0; i < gamma.size(); i++) gamma[i] = (int)(pow(i / 65536.0, 1.0 / scene.imageGamma) * 65535);
  cudaError_t e = cudaSuccess;
  if (table) e = cudaMemcpyAsync(gamma_dev, gamma.data(), sizeof(int) * 65536, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return set_error(MBGB_ERR_CUDA, std::string("gamma table: ") + cudaGetErrorString(e));
  const int64_t n = (int64_t)width * height;
  compile16_kernel<<<grid_for(3 * n, 256), 256, 0, s>>>(image_float, n, scene.brightness, scene.contrast,
                                                        scene.hdrEnabled ? 1 : 0, table ? gamma_dev : nullptr, image16);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);   // the host table is released on return
  if (e != cudaSuccess) return set_error(MBGB_ERR_CUDA, std::string("compile kernel: ") + cudaGetErrorString(e));
  return MBGB_OK;
}

// Whether ssao_flat_kernel takes a frame: the flat projection, offsets of at most 16 bits and pixel
// indices of at most 31.
static bool ssao_flat(const mbgb_scene &scene, int width, int64_t npix) {
  return scene.perspectiveType != MBGB_PERSP_FISH_EYE && scene.perspectiveType != MBGB_PERSP_EQUIRECT &&
         width <= 64000 && npix < (int64_t)1 << 31;
}

// Scratch of ssao_device: cos and sin of the directions, and for the flat kernel their samples and
// the open pixels.
struct SsaoScratch {
  SsaoSample *samples;
  SsaoOffset *offsets;
  uint32_t *opens, *open;
  size_t bytes;
};
static SsaoScratch ssao_scratch(void *base, int quality, int64_t npix) {
  const size_t q = (size_t)std::max(quality, 0), n = q > 0 ? q * (q - 1) : 0;
  size_t at = (sizeof(double) * 2 * q + 15) & ~(size_t)15;
  SsaoScratch m;
  m.samples = (SsaoSample *)((char *)base + at);
  at += sizeof(SsaoSample) * n;
  m.offsets = (SsaoOffset *)((char *)base + at);
  at += sizeof(SsaoOffset) * n;
  m.opens = (uint32_t *)((char *)base + at);
  m.open = m.opens + 4;
  m.bytes = at + 16 + sizeof(uint32_t) * (size_t)npix;
  return m;
}
size_t ssao_scratch_bytes(int quality, int64_t npix) { return ssao_scratch(nullptr, quality, npix).bytes; }
size_t ssao_scratch_bytes(const mbgb_scene &scene, int width, int64_t npix) {
  return ssao_flat(scene, width, npix) ? ssao_scratch_bytes(scene.SSAOQuality, npix)
                                       : sizeof(double) * 2 * (size_t)std::max(scene.SSAOQuality, 0);
}

// PostRendering_SSAO on the device, in double (the reference's arithmetic): the sample
// positions x + r^2 s cos(a) land on the neighbouring pixel or not depending on the last
// bits of cos(a) near 0 (cos(pi / 2) = 6e-17), which float arithmetic does not keep.
// `tables`: device scratch of ssao_scratch_bytes.
mbgb_status ssao_device(const mbgb_scene &scene, const mbgb_image &layers, uint16_t *image16, void *tables,
                        cudaStream_t s) {
  const int q = scene.SSAOQuality;
  if (q < 1) return MBGB_OK;   // the loops of ThreadSSAO run no direction: nothing changes
  std::vector<double> t(2 * (size_t)q);
  for (int i = 0; i < q; i++) {
    t[q + i] = sin((double)i / q * 2.0 * kPi);
    t[i] = cos((double)i / q * 2.0 * kPi);
  }
  const int64_t n = (int64_t)layers.width * layers.height;
  const int block = 128;
  const double *cs = (const double *)tables, *sn = cs + q;
  cudaError_t e = cudaMemcpyAsync(tables, t.data(), sizeof(double) * 2 * q, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    if (!ssao_flat(scene, layers.width, n)) {
      ssao_kernel<double><<<grid_for(n, block), block, 0, s>>>(
          layers.zbuffer, layers.opacity, layers.colour, image16, layers.width, layers.height, scene.persp, q,
          scene.perspectiveType, scene.globalIlum, cs, sn);
    } else {
      const SsaoScratch m = ssao_scratch(tables, q, n);
      const SsaoArgs g{layers.zbuffer, layers.opacity, layers.colour, image16, layers.width, layers.height, q,
                       ssao_least_depth(q, scene.persp, (double)layers.width / layers.height),
                       scene.persp, scene.globalIlum, m.samples, m.offsets, m.opens, m.open};
      e = cudaMemsetAsync(m.opens, 0, sizeof(uint32_t), s);
      ssao_table_kernel<<<grid_for((int64_t)q * (q - 1), block), block, 0, s>>>(m.samples, m.offsets, layers.width,
                                                                                layers.height, scene.persp, q, cs, sn);
      ssao_flat_kernel<<<grid_for(n, block), block, 0, s>>>(g);
      ssao_exact_kernel<<<grid_for(n, block), block, 0, s>>>(g);
    }
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return set_error(MBGB_ERR_CUDA, std::string("SSAO kernel: ") + cudaGetErrorString(e));
  return MBGB_OK;
}

}  // namespace mbgb

namespace {

struct SortZ {
  float z;
  int i;
};

// QuickSortZBuffer (src/common_math.h:53-84): Hoare partition around the middle element, on
// [l, p]; an explicit stack instead of recursion (the two parts are disjoint).
void quicksort_z(std::vector<SortZ> &d, int l0, int p0) {
  std::vector<std::pair<int, int>> stack{{l0, p0}};
  while (!stack.empty()) {
    const int l = stack.back().first, p = stack.back().second;
    stack.pop_back();
    int i = l, j = p;
    const SortZ x = d[(size_t)((l + p) / 2)];
    do {
      while (d[(size_t)i].z < x.z) i++;
      while (x.z < d[(size_t)j].z) j--;
      if (i <= j) {
        std::swap(d[(size_t)i], d[(size_t)j]);
        i++;
        j--;
      }
    } while (i <= j);
    if (i < p) stack.push_back({i, p});
    if (l < j) stack.push_back({l, j});
  }
}

}  // namespace

namespace mbgb {

// PostRendering_DOF (src/image.cpp:57-206). The host sorts the z-buffer with the
// reference's quicksort (element 0 stays in place, as there), shuffles it with its Random()
// swaps (rand() seeded with `seed`; the reference continues the process's rand() stream),
// and lists, per 16 x 16 tile, the splats that reach it in splat order (far to near); the
// device applies the splats (dof_kernel).
mbgb_status dof_device(const mbgb_scene &scene, const mbgb_image &layers, uint16_t *image16, uint32_t seed,
                       cudaStream_t s) {
  const int width = layers.width, height = layers.height;
  const int64_t n = (int64_t)width * height;
  if (n <= 0 || n > (int64_t)1 << 30) return set_error(MBGB_ERR_BAD_PARAM, "DOF: image size out of range");
  const double deep = scene.DOFRadius * width / 1000.0;
  const double neutral = pow(10, scene.DOFFocus / 10.0 - 16.0);
  std::vector<SortZ> sortz((size_t)n);
  std::vector<float> zb((size_t)n);
  cudaError_t e = cudaMemcpyAsync(zb.data(), layers.zbuffer, sizeof(float) * n, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return set_error(MBGB_ERR_CUDA, std::string("DOF z-buffer: ") + cudaGetErrorString(e));
  for (int64_t p = 0; p < n; p++) sortz[(size_t)p] = SortZ{zb[(size_t)p], (int)p};
  if (n > 2) quicksort_z(sortz, 1, (int)n - 1);
  // randomise the order within similar blur sizes (src/image.cpp:96-138)
  GlibcRand rng(seed);
  for (int64_t i = n - 1; i >= 0; i--) {
    const SortZ temp = sortz[(size_t)i];
    const double z1 = temp.z;
    const double size1 = (z1 - neutral) / z1 * deep;
    int randomStep = (int)i;
    bool done = false;
    int64_t ii;
    do {
      ii = i - rng.random(randomStep);
      if (ii <= 0) ii = 0;
      const double z2 = sortz[(size_t)ii].z;
      const double size2 = (z2 - neutral) / z2 * deep;
      if (size1 == 0 && size2 == 0) done = true;
      if (size1 * size2 > 0) {
        const double sizeCompare = size1 > 0 ? size2 / size1 : size1 / size2;
        done = sizeCompare > 0.7;
      } else {
        done = false;
      }
      randomStep = (int)(randomStep * 0.7 - 1);
      if (randomStep <= 0) done = true;
    } while (!done);
    sortz[(size_t)i] = sortz[(size_t)ii];
    sortz[(size_t)ii] = temp;
  }
  // splats in order, and the tiles each reaches
  const int tilesX = (width + kDofTile - 1) / kDofTile, tilesY = (height + kDofTile - 1) / kDofTile;
  std::vector<DofSplat> splats((size_t)n);
  std::vector<int64_t> count((size_t)tilesX * tilesY + 1, 0);
  for (int64_t k = 0; k < n; k++) {
    const int ii = sortz[(size_t)(n - k - 1)].i;
    const int x = ii % width, y = ii / width;
    const double z = zb[(size_t)ii];
    double blur = fabs(z - neutral) / z * deep;
    if (blur > 100) blur = 100.0;
    const int size = (int)blur;
    splats[(size_t)k] = DofSplat{x, y, size, ii, blur, blur * blur * sqrt(blur) * kPi / 3.0};
    const int tx0 = std::max(0, x - size) / kDofTile, tx1 = std::min(width - 1, x + size) / kDofTile;
    const int ty0 = std::max(0, y - size) / kDofTile, ty1 = std::min(height - 1, y + size) / kDofTile;
    for (int ty = ty0; ty <= ty1; ty++)
      for (int tx = tx0; tx <= tx1; tx++) count[(size_t)ty * tilesX + tx + 1]++;
  }
  for (size_t t = 1; t < count.size(); t++) count[t] += count[t - 1];
  std::vector<int> list((size_t)count.back());
  std::vector<int64_t> fill(count.begin(), count.end() - 1);
  for (int64_t k = 0; k < n; k++) {
    const DofSplat &sp = splats[(size_t)k];
    const int tx0 = std::max(0, sp.x - sp.size) / kDofTile, tx1 = std::min(width - 1, sp.x + sp.size) / kDofTile;
    const int ty0 = std::max(0, sp.y - sp.size) / kDofTile, ty1 = std::min(height - 1, sp.y + sp.size) / kDofTile;
    for (int ty = ty0; ty <= ty1; ty++)
      for (int tx = tx0; tx <= tx1; tx++) list[(size_t)fill[(size_t)ty * tilesX + tx]++] = (int)k;
  }
  // device buffers: splats, tile starts, lists, original image and alpha
  const size_t bSplat = sizeof(DofSplat) * (size_t)n, bStart = sizeof(int64_t) * count.size(),
               bList = sizeof(int) * list.size(), bImg = sizeof(uint16_t) * 3 * (size_t)n,
               bAlpha = sizeof(uint16_t) * (size_t)n;
  char *buf = nullptr;
  e = cudaMallocAsync((void **)&buf, bSplat + bStart + bList + bImg + bAlpha + 64, s);
  if (e != cudaSuccess) return set_error(MBGB_ERR_CUDA, std::string("DOF buffers: ") + cudaGetErrorString(e));
  char *pSplat = buf, *pStart = pSplat + bSplat, *pList = pStart + bStart, *pImg = pList + bList;
  pImg = (char *)(((uintptr_t)pImg + 15) & ~(uintptr_t)15);
  char *pAlpha = pImg + bImg;
  e = cudaMemcpyAsync(pSplat, splats.data(), bSplat, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(pStart, count.data(), bStart, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && bList) e = cudaMemcpyAsync(pList, list.data(), bList, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(pImg, image16, bImg, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(pAlpha, layers.alpha, bAlpha, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess)
    dof_kernel<<<tilesX * tilesY, kDofTile * kDofTile, 0, s>>>(
        (const DofSplat *)pSplat, (const int64_t *)pStart, (const int *)pList, tilesX, width, height,
        (const uint16_t *)pImg, (const uint16_t *)pAlpha, image16, layers.alpha);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFreeAsync(buf, s);
  cudaStreamSynchronize(s);
  if (e != cudaSuccess) return set_error(MBGB_ERR_CUDA, std::string("DOF kernel: ") + cudaGetErrorString(e));
  return MBGB_OK;
}

}  // namespace mbgb
