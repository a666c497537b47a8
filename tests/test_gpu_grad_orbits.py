"""The gradient stage's value-only orbits against the orbits with tangents (needs a GPU;
csrc/grad_core.cuh is compiled into the test with its probes). An orbit first runs as the value alone
and is taken as bounded by that, so both must round alike: points around the set's surface, where
orbits of hundreds of iterations escape or not by their last bits."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from mandelbulber_gb300 import _build

pytestmark = pytest.mark.gpu
SOURCE = r"""
#include "grad_core.cuh"
using namespace mbgb;
using namespace mbgb::dev;
namespace {
template <typename T>
FractalT<T> fractal(const int formula, const int N) {
  FractalT<T> f{};
  f.formula = formula;
  f.N = N;
  f.constantFactor = T(1);
  f.bailout = T(formula == 2 ? 100 : 1024);
  f.mbFoldLimit = T(1);
  f.mbFoldValue = T(2);
  f.mbMinR = T(0.5);
  f.mbFixedR = T(1);
  return f;
}
// counts: [0] points, [1] orbits of more than kGradHead iterations that escape, [2] bounded orbits,
// differences of [3] de_dual_policy and the plain dual orbit, [4] escapes and the FP32 dual orbit,
// [5] escapes and the FP64 orbit of the level set
template <int FORMULA>
__global__ void compare_kernel(const ParamsT<float> p, const FractalT<double> fd, const double fparam, const int n,
                               const double *points, unsigned long long *count) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const V3<double> P{points[3 * i], points[3 * i + 1], points[3 * i + 2]};
    const V3<float> q{(float)P.x, (float)P.y, (float)P.z};
    int L, M;
    const Dual<double, 4> a = de_dual_policy<float, FORMULA>(p, fd, P, fd.N, L, (float)fparam, fparam);
    const Dual<float, 4> b = de_dual<float, FORMULA>(p.f, q, fd.N, M, (float)fparam);
    bool finite = isfinite(b.v), same = L == M && a.v == (double)b.v;
    for (int k = 0; k < 4; k++) {
      finite = finite && isfinite(b.d[k]);
      same = same && a.d[k] == (double)b.d[k];
    }
    atomicAdd(count + 0, 1ull);
    if (M > kGradHead && M < fd.N) atomicAdd(count + 1, 1ull);
    if (M == fd.N) atomicAdd(count + 2, 1ull);
    if (finite && !same) atomicAdd(count + 3, 1ull);
    if (escapes<float, FORMULA>(p.f, q, fd.N, (float)fparam) != (M < fd.N)) atomicAdd(count + 4, 1ull);
    if (i % 8 == 0) {
      de_along<double, FORMULA>(fd, P, V3<double>{0.3, 0.9, -0.2}, fd.N, M, fparam);
      if (escapes<double, FORMULA>(fd, P, fd.N, fparam) != (M < fd.N)) atomicAdd(count + 5, 1ull);
    }
  }
}
}
extern "C" int compare(int formula, int N, double fparam, int n, const double *points, unsigned long long *count) {
  ParamsT<float> p{};
  p.f = fractal<float>(formula, N);
  const FractalT<double> fd = fractal<double>(formula, N);
  if (formula == 2) compare_kernel<2><<<608, 128>>>(p, fd, fparam, n, points, count);
  else compare_kernel<8><<<608, 128>>>(p, fd, fparam, n, points, count);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("grad")
    (d / "t.cu").write_text(SOURCE)
    command = next(c for u, c in _build._units(_build._cuda_home()) if u == "wave_f32.cu")
    subprocess.check_call([*command, "-shared", str(d / "t.cu"), "-o", str(d / "t.so")])
    return ctypes.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("formula,N,fparam", [(2, 250, 8.0), (2, 1250, 8.0), (2, 250, 6.3), (2, 250, 9.7), (8, 150, 2.0),
                                              (8, 150, -1.5)])
def test_value_only_orbits_are_the_dual_orbits(lib, formula, N, fparam):
    import torch
    rng, n = np.random.default_rng(N), 400000
    if formula == 2:   # a shell about the bulb's surface
        p = rng.normal(size=(n, 3))
        p *= (rng.uniform(0.85, 1.2, n) / np.linalg.norm(p, axis=1))[:, None]
    else:
        p = rng.uniform(-6.0, 6.0, (n, 3))
        p[: n // 2] *= 0.2
    points = torch.tensor(p, device="cuda")
    count = torch.zeros(6, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert lib.compare(formula, N, ctypes.c_double(fparam), n, ctypes.c_void_p(points.data_ptr()),
                       ctypes.c_void_p(count.data_ptr())) == 0
    total, late, bounded, policy, fp32, fp64 = count.tolist()
    assert total == n and bounded > 0 and (formula == 8 or late > 100)
    assert (policy, fp32, fp64) == (0, 0, 0)
