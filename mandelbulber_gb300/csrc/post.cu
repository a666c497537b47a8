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
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n; i += (int64_t)gridDim.x * blockDim.x) {
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

// One sample of the flat projection's horizon search (shared by every pixel): direction a,
// radius r. A pixel at integer x samples column trunc(x + off): with off = k + f, k integer, the
// rounded sum stays strictly between x + k and x + k + 1 for f in [1e-9, 1 - 1e-9] and is x + k
// for f = 0, so the column is x + k and the bounds test one of integers; other offsets (`sure`
// false: cos(pi / 2) = 6e-17 times a radius) are added in double.
struct SsaoSample {
  double offX, offY;    // r^2 scale cos, r^2 scale sin
  int kx, ky;           // floor of the offsets
  int maxX, maxY;       // largest column and row inside the picture: size - 2, size - 1 for f = 0
  float cx, cy;         // the offsets in the projection plane at depth 1: off / w aspect persp
  int sure;
};

__global__ void ssao_table_kernel(SsaoSample *__restrict__ t, const int width, const int height, const double persp,
                                  const int quality, const double *__restrict__ cs, const double *__restrict__ sn) {
  const double w = (double)width, h = (double)height;
  const double scale = w / (double)(quality * quality) / 2.0, aspect = w / h;
  const int n = quality * (quality - 1);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int a = i / (quality - 1);
    const double r = (double)(i % (quality - 1) + 1), rr = r * r * scale;
    SsaoSample s;
    s.offX = rr * cs[a];
    s.offY = rr * sn[a];
    const double fx = floor(s.offX), fy = floor(s.offY), rx = s.offX - fx, ry = s.offY - fy;
    s.kx = (int)fx;
    s.ky = (int)fy;
    s.maxX = width - (rx == 0.0 ? 1 : 2);
    s.maxY = height - (ry == 0.0 ? 1 : 2);
    s.cx = (float)(s.offX / w * aspect * persp);
    s.cy = (float)(s.offY / h * persp);
    s.sure = (rx == 0.0 || (rx >= 1e-9 && rx <= 1.0 - 1e-9)) && (ry == 0.0 || (ry >= 1e-9 && ry <= 1.0 - 1e-9));
    t[i] = s;
  }
}

// ThreadSSAO for the flat projection, the values of ssao_kernel<double> bit for bit.
//
// What bounds it: the FP64 pipe (exact64.cuh). A sample's slope takes three quotients and a root
// there, 870 SM cycles a warp, and of the quality - 1 samples of a direction only the steepest
// counts. So a first pass brackets every slope in FP32, lo <= slope <= up, and keeps the largest
// lo and the largest up of the other samples: where that lies below, one sample is the steepest
// for certain and only it is computed in double (otherwise every sample whose bracket reaches the
// largest lo). The brackets: with A(x) = (x / w - 1/2) aspect persp the plane distance is
// dx = A(xx) dz + c z (c the offset's, dz the depth difference, exact in FP32 up to its
// rounding), so FP32's error is below 2^-21 ((|A(x)| + |c|) |dz| + |c z|), far above the double
// form's own; the root and quotients add 4e-6 relative. Columns and rows come from integers
// (SsaoSample). What is left is mostly atan, once a direction.
// 1920x1080, quality 20 (with the 16-bit step): 70.6 -> 5.65 ms.
__global__ void __launch_bounds__(128) ssao_flat_kernel(
    const float *__restrict__ zbuf, const uint16_t *__restrict__ opacity, const uint8_t *__restrict__ colour,
    uint16_t *__restrict__ image16, const int width, const int height, const double persp, const int quality,
    const double intensity, const SsaoSample *__restrict__ table) {
  using mbgb::dev::div_int;
  using mbgb::dev::sqrt_int;
  const int64_t n = (int64_t)width * height;
  const double w = (double)width, h = (double)height, aspect = w / h;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % width), y = (int)(i / width);
    const float zf = zbuf[i];
    const double z = (double)zf;
    double total = 0.0;
    if (z < 1e19) {
      const double px = (div_int((double)x, w) - 0.5) * aspect, py = div_int((double)y, h) - 0.5;
      const double x2 = px * z * persp, y2 = py * z * persp;
      const float ax = (float)(px * persp), ay = (float)(py * persp);
      // the depth of sample s, or false outside the picture and on the pixel itself
      auto depth_at = [&](const SsaoSample &s, float &z2) {
        int xi = x + s.kx, yi = y + s.ky;
        if (s.sure) {
          if (xi < 0 || xi > s.maxX || yi < 0 || yi > s.maxY) return false;
        } else {
          const double xx = (double)x + s.offX, yy = (double)y + s.offY;
          if (xx < 0.0 || xx > (double)(width - 1) || yy < 0.0 || yy > (double)(height - 1)) return false;
          xi = (int)xx;
          yi = (int)yy;
        }
        if (xi == x && yi == y) return false;
        z2 = zbuf[(int64_t)yi * width + xi];
        return true;
      };
      auto bracket = [&](const SsaoSample &s, const float z2, float &lo, float &up) {
        const float dz = z2 - zf, gx = ax + s.cx, gy = ay + s.cy, bx = s.cx * zf, by = s.cy * zf;
        const float dx = fabsf(fmaf(gx, dz, bx)), dy = fabsf(fmaf(gy, dz, by));
        const float e = 4.8e-7f * ((fabsf(ax) + fabsf(s.cx) + fabsf(ay) + fabsf(s.cy)) * fabsf(dz) + fabsf(bx) + fabsf(by));
        const float m = fmaxf(dx, dy), q = __fdividef(fminf(dx, dy), m);
        const float dr = m * sqrtf(fmaf(q, q, 1.0f));
        const float drLo = fmaf(dr, 1.0f - 4e-6f, -e), drUp = fmaf(dr, 1.0f + 4e-6f, e);
        if (!(m > 1e-25f) || !(drLo > 1e-25f)) {   // nothing certain
          lo = -INFINITY;
          up = INFINITY;
          return;
        }
        const float near = __fdividef(-dz, drLo), wide = __fdividef(-dz, drUp);
        lo = dz < 0.0f ? wide * (1.0f - 4e-6f) : near * (1.0f + 4e-6f);
        up = dz < 0.0f ? near * (1.0f + 4e-6f) : wide * (1.0f - 4e-6f);
      };
      auto slope = [&](const SsaoSample &s, const float z2f) {
        const double xx = (double)x + s.offX, yy = (double)y + s.offY, z2 = (double)z2f;
        const double g = z2 * persp;
        const double dx = (div_int(xx, w) - 0.5) * aspect * g - x2;
        const double dy = (div_int(yy, h) - 0.5) * g - y2;
        return div_int(-(z2 - z), sqrt_int(dx * dx + dy * dy));
      };
      double ambient = 0.0;
      for (int a = 0; a < quality; a++) {
        const SsaoSample *dir = table + (int64_t)a * (quality - 1);
        float bestLo = -INFINITY, bestUp = -INFINITY, otherUp = -INFINITY;
        int best = -1;
        for (int r = 0; r < quality - 1; r++) {
          float z2, lo, up;
          if (!depth_at(dir[r], z2)) continue;
          bracket(dir[r], z2, lo, up);
          if (lo > bestLo || best < 0) {
            otherUp = fmaxf(otherUp, bestUp);
            bestLo = lo;
            bestUp = up;
            best = r;
          } else {
            otherUp = fmaxf(otherUp, up);
          }
        }
        double maxDiff = -1e50;
        if (best >= 0) {
          if (otherUp < bestLo) {
            float z2;
            depth_at(dir[best], z2);
            const double diff = slope(dir[best], z2);
            if (diff > maxDiff) maxDiff = diff;
          } else {
            for (int r = 0; r < quality - 1; r++) {
              float z2, lo, up;
              if (!depth_at(dir[r], z2)) continue;
              bracket(dir[r], z2, lo, up);
              if (!(up >= bestLo)) continue;
              const double diff = slope(dir[r], z2);
              if (diff > maxDiff) maxDiff = diff;
            }
          }
        }
        ambient += div_int(-atan(maxDiff), kPi) + 0.5;
      }
      total = ambient / (double)quality;
      if (total < 0.0) total = 0.0;
    }
    const double op = (double)opacity[i] / 65535.0;
    for (int c = 0; c < 3; c++) {
      double v = (double)image16[3 * i + c] + 65535.0 * (double)colour[3 * i + c] / 256.0 * total * intensity * (1.0 - op);
      if (v > 65535.0) v = 65535.0;
      image16[3 * i + c] = (uint16_t)(unsigned short)v;
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

size_t ssao_scratch_bytes(int quality) {
  const size_t q = (size_t)std::max(quality, 0);
  return sizeof(double) * 2 * q + (q > 0 ? sizeof(SsaoSample) * q * (q - 1) : 0) + 64;
}

// PostRendering_SSAO on the device, in double (the reference's arithmetic): the sample
// positions x + r^2 s cos(a) land on the neighbouring pixel or not depending on the last
// bits of cos(a) near 0 (cos(pi / 2) = 6e-17), which float arithmetic does not keep.
// `tables` (ssao_scratch_bytes) receives cos and sin of the `quality` directions and, for the
// flat projection, the directions' samples.
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
    if (scene.perspectiveType == MBGB_PERSP_FISH_EYE || scene.perspectiveType == MBGB_PERSP_EQUIRECT) {
      ssao_kernel<double><<<grid_for(n, block), block, 0, s>>>(
          layers.zbuffer, layers.opacity, layers.colour, image16, layers.width, layers.height, scene.persp, q,
          scene.perspectiveType, scene.globalIlum, cs, sn);
    } else {
      SsaoSample *table = (SsaoSample *)(cs + 2 * q);
      ssao_table_kernel<<<grid_for((int64_t)q * (q - 1), block), block, 0, s>>>(table, layers.width, layers.height,
                                                                                scene.persp, q, cs, sn);
      ssao_flat_kernel<<<grid_for(n, block), block, 0, s>>>(layers.zbuffer, layers.opacity, layers.colour, image16,
                                                            layers.width, layers.height, scene.persp, q,
                                                            scene.globalIlum, table);
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
