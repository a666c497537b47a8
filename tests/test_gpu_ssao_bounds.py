"""The flat projection's SSAO against the same unit's double kernel, and the error bounds that let
it answer in FP32 (needs a GPU; csrc/post.cu is compiled into the test with its probes)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from mandelbulber_gb300 import _build

pytestmark = pytest.mark.gpu
SOURCE = r"""
#include "post.cu"
namespace mbgb {
// what the unit takes from the library's others
mbgb_status set_error(mbgb_status s, const std::string &) { return s; }
GlibcRand::GlibcRand(uint32_t) {}
int GlibcRand::random(int) { return 0; }
}
namespace {
// lo <= slope <= up of samples at plane offset (cx, cy) from pixels at (ax, ay): 1 where not
__global__ void bracket_kernel(const int n, const float *z, const float *z2, const double *ax, const double *ay,
                               const double *cx, const double *cy, int *outside) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    SsaoSample s;
    s.cx = f2_of(cx[i]).h;
    s.cy = f2_of(cy[i]).h;
    s.cc = (__float_as_uint(fabsf(s.cx) + fabsf(s.cy)) | 3u) + 1u;
    const float x = f2_of(ax[i]).h, y = f2_of(ay[i]).h;
    float lo, up;
    ssao_bracket(s, x, y, fabsf(x) + fabsf(y), z[i] * kSsaoScale, z2[i], lo, up);
    const double z1 = z[i], zz = z2[i], dz = zz - z1;
    const double dx = ax[i] * dz + cx[i] * zz, dy = ay[i] * dz + cy[i] * zz;
    const double slope = -dz / sqrt(dx * dx + dy * dy);
    outside[i] = !((double)lo <= slope && slope <= (double)up);
  }
}
// the sum of q equal angles in pairs of floats against q c, in units of its bound
__global__ void sum_kernel(const int n, const double *c, const int quality, double *ratio) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const F2 a = f2_of(c[i]);
    F2 sum{0.0f, 0.0f};
    for (int k = 0; k < quality; k++) sum = f2_add(sum, a);
    const double v = (double)a.h + (double)a.l;
    ratio[i] = fabs(((double)sum.h + (double)sum.l) - quality * v) / ssao_sum_error(quality);
  }
}
}
extern "C" int sums(int n, const double *c, int quality, double *ratio) {
  sum_kernel<<<256, 128>>>(n, c, quality, ratio);
  return (int)cudaDeviceSynchronize();
}
extern "C" float least_depth(int quality, double persp, double aspect) { return ssao_least_depth(quality, persp, aspect); }
extern "C" int brackets(int n, const float *z, const float *z2, const double *ax, const double *ay, const double *cx,
                        const double *cy, int *outside) {
  bracket_kernel<<<256, 128>>>(n, z, z2, ax, ay, cx, cy, outside);
  return (int)cudaDeviceSynchronize();
}
extern "C" long scratch_bytes(int quality, long npix) { return (long)mbgb::ssao_scratch_bytes(quality, npix); }
// ms of `a` by ssao_device and of `b` by ssao_kernel<double>, the least of five
extern "C" int ssao_times(int width, int height, int quality, float *z, uint16_t *opacity, uint8_t *colour, uint16_t *a,
                          uint16_t *b, void *scratch, float *ms) {
  mbgb_scene *scene = (mbgb_scene *)calloc(1, sizeof(mbgb_scene));
  scene->SSAOQuality = quality;
  scene->persp = 0.5;
  scene->globalIlum = 0.5;
  mbgb_image img{};
  img.width = width;
  img.height = height;
  img.zbuffer = z;
  img.opacity = opacity;
  img.colour = colour;
  const double *cs = (const double *)scratch;
  cudaEvent_t e[3];
  for (auto &v : e) cudaEventCreate(&v);
  ms[0] = ms[1] = 1e30f;
  int st = 0;
  for (int k = 0; k < 6 && !st; k++) {
    cudaEventRecord(e[0]);
    st = mbgb::ssao_device(*scene, img, a, scratch, 0);
    cudaEventRecord(e[1]);
    ssao_kernel<double><<<grid_for((int64_t)width * height, 128), 128>>>(z, opacity, colour, b, width, height, 0.5, quality,
                                                                      0, 0.5, cs, cs + quality);
    cudaEventRecord(e[2]);
    if (!st) st = (int)cudaDeviceSynchronize();
    float t[2];
    cudaEventElapsedTime(&t[0], e[0], e[1]);
    cudaEventElapsedTime(&t[1], e[1], e[2]);
    for (int j = 0; j < 2 && k > 0; j++) ms[j] = t[j] < ms[j] ? t[j] : ms[j];
  }
  for (auto &v : e) cudaEventDestroy(v);
  free(scene);
  return st;
}
// image `a` by ssao_device, image `b` by ssao_kernel<double>
extern "C" int ssao_both(int width, int height, double persp, int quality, double intensity, float *z, uint16_t *opacity,
                         uint8_t *colour, uint16_t *a, uint16_t *b, void *scratch) {
  mbgb_scene *scene = (mbgb_scene *)calloc(1, sizeof(mbgb_scene));
  scene->SSAOQuality = quality;
  scene->persp = persp;
  scene->globalIlum = intensity;
  mbgb_image img{};
  img.width = width;
  img.height = height;
  img.zbuffer = z;
  img.opacity = opacity;
  img.colour = colour;
  const int st = mbgb::ssao_device(*scene, img, a, scratch, 0);
  free(scene);
  const double *cs = (const double *)scratch;   // ssao_device leaves the directions there
  ssao_kernel<double><<<grid_for((int64_t)width * height, 128), 128>>>(z, opacity, colour, b, width, height, persp, quality,
                                                                    0, intensity, cs, cs + quality);
  return st ? st : (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("ssao")
    (d / "t.cu").write_text(SOURCE)
    command = next(c for u, c in _build._units(_build._cuda_home()) if u == "post.cu")
    subprocess.check_call([*command, "-shared", str(d / "t.cu"), "-o", str(d / "t.so")])
    out = ctypes.CDLL(str(d / "t.so"))
    out.least_depth.restype = ctypes.c_float
    out.least_depth.argtypes = [ctypes.c_int, ctypes.c_double, ctypes.c_double]
    out.scratch_bytes.restype = ctypes.c_long
    out.scratch_bytes.argtypes = [ctypes.c_int, ctypes.c_long]
    return out


def _cuda(*arrays):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]
    torch.cuda.synchronize()
    return t, [ctypes.c_void_p(v.data_ptr()) for v in t]


@pytest.mark.parametrize("quality", [2, 20, 200, 1000])
@pytest.mark.parametrize("persp", [2.0, 0.5, 1e-2, 1e-3, 1e-4])
def test_brackets_hold_the_slope(lib, quality, persp):
    """Every bracket holds the slope in double, from the least depth on (seven digits of depth
    differences, so that plane distances cancel too), wide and narrow views."""
    n, rng, aspect = 400000, np.random.default_rng(quality), 4 / 3
    z = (lib.least_depth(quality, persp, aspect) * 10 ** rng.uniform(0.001, 2, n)).astype(np.float32)
    z2 = (z * (1 + 10 ** rng.uniform(-7, 0, n) * rng.choice([-1, 1], n))).astype(np.float32)
    ax, ay = rng.uniform(-0.5, 0.5, n) * aspect * persp, rng.uniform(-0.5, 0.5, n) * persp
    r, a = rng.integers(1, min(quality, 40), n), rng.integers(0, quality, n) * (2 * np.pi / quality)
    rr = r * r * aspect * persp / (2 * quality ** 2)
    outside = np.zeros(n, np.int32)
    t, p = _cuda(z, z2, ax, ay, rr * np.cos(a), rr * np.sin(a), outside)
    assert lib.brackets(n, *p) == 0
    assert int(t[6].sum()) == 0


@pytest.mark.parametrize("quality", [1, 2, 20, 333, 1000])
def test_angle_sum_stays_in_its_bound(lib, quality):
    """Equal angles, whose roundings add up, over the angles' whole range."""
    n = 400000
    c = np.random.default_rng(quality).uniform(-np.pi / 2, np.pi / 2, n)
    t, p = _cuda(c, np.zeros(n))
    assert lib.sums(n, p[0], quality, p[1]) == 0
    assert float(t[1].max()) <= 1.0


def _depth(kind, w, h, rng):
    y, x = np.mgrid[0:h, 0:w]
    if kind == "plane":
        return 3.0 + 0.01 * x + 0.02 * y
    if kind == "steps":
        z = 2.0 + rng.integers(0, 4, (h, w)) * 0.5
        z[rng.random((h, w)) < 0.3] = 1e20
        return z
    if kind == "tiny":
        z = rng.random((h, w)) * 10.0 ** rng.uniform(-30, 9, (h, w))
        z[0, 0] = 0.0
        return z
    if kind == "deep":   # a camera a millionth from the surface, on both sides of the FP32 forms' range
        return 1e-6 * (1 + 0.3 * np.sin(x * 0.3) + 0.2 * rng.random((h, w)))
    return 5.0 + np.sin(x * 0.3) + np.cos(y * 0.2) + 0.05 * rng.normal(size=(h, w))


@pytest.mark.parametrize("kind", ["plane", "steps", "tiny", "deep", "waves"])
@pytest.mark.parametrize("w,h,quality,persp", [(33, 32, 1, 0.5), (1, 40, 7, 0.5), (64, 48, 2, 3.0), (61, 47, 3, 0.5),
                                               (97, 55, 5, 0.01), (96, 54, 6, 0.9), (70, 41, 8, 0.5), (64, 64, 9, 0.5),
                                               (131, 67, 16, 1e-3), (131, 67, 17, 0.5), (257, 101, 20, 0.9),
                                               (48, 200, 33, 0.5), (40, 30, 200, 0.5), (31, 23, 1000, 0.7),
                                               (31, 23, 1000, 1e-3)])
def test_flat_ssao_is_the_double_kernel(lib, w, h, quality, persp, kind):
    """The bytes of ssao_kernel<double>."""
    import torch
    rng = np.random.default_rng(w * 100 + quality)
    image = rng.integers(0, 65536, (h, w, 3)).astype(np.uint16).view(np.int16)
    t, p = _cuda(_depth(kind, w, h, rng).astype(np.float32), rng.integers(0, 65536, (h, w)).astype(np.uint16).view(np.int16),
                 rng.integers(0, 256, (h, w, 3)).astype(np.uint8), image, image.copy())
    scratch = torch.zeros(lib.scratch_bytes(quality, w * h), dtype=torch.uint8, device="cuda")
    for intensity in (0.8, -0.4)[:2 if quality <= 33 else 1]:
        assert lib.ssao_both(w, h, ctypes.c_double(persp), quality, ctypes.c_double(intensity), *p,
                             ctypes.c_void_p(scratch.data_ptr())) == 0
        assert torch.equal(t[3], t[4])


@pytest.mark.parametrize("quality", [4, 6, 10, 20])
def test_depths_below_the_fp32_range_cost_no_more_than_the_double_kernel(lib, quality):
    """A camera half a millionth from the surface: every pixel is the double form's. The call with its
    tables and synchronisation may take 1.1 times the one kernel."""
    import torch
    w, h = 1024, 768
    y, x = np.mgrid[0:h, 0:w]
    z = 5e-7 * (1 + 0.3 * np.sin(x * 0.05) + 0.2 * np.cos(y * 0.03))
    t, p = _cuda(z.astype(np.float32), np.zeros((h, w), np.int16), np.full((h, w, 3), 128, np.uint8),
                 np.zeros((h, w, 3), np.int16), np.zeros((h, w, 3), np.int16))
    scratch = torch.zeros(lib.scratch_bytes(quality, w * h), dtype=torch.uint8, device="cuda")
    ms = (ctypes.c_float * 2)()
    assert lib.ssao_times(w, h, quality, *p, ctypes.c_void_p(scratch.data_ptr()), ms) == 0
    print(quality, "call", ms[0], "double kernel", ms[1])
    assert ms[0] <= 1.1 * ms[1], (ms[0], ms[1])
    assert torch.equal(t[3], t[4])
