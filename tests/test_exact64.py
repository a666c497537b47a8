"""The integer FP64 operations (csrc/exact64.cuh) and the strict Mandelbox orbit built on them.

The operations are held to the host's IEEE square root, quotient and product bit for bit, with
the seed off by as much as four of its last bits (the device's approximate reciprocal and
reciprocal square root stay within two). The orbit is held to the FP64 oracle bit for bit over
the scales, folds and radii that choose between its forms, and at points where a form's range
ends: zeros, subnormals, the far field, infinities and NaN.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import mandelbulber_gb300 as mb
from mandelbulber_gb300 import _build
from mandelbulber_gb300 import workloads as W
from tests import oracle_lib

SOURCE = r"""
#include "exact64.cuh"
#include <math.h>
using namespace mbgb::dev;
// counts of results that differ from the host's: sqrt, sqrt^2, quotient, product, square, fold
extern "C" void compare(const double *x, const double *y, long n, int jitter, long *bad) {
  for (long i = 0; i < n; i++) {
    const double s = sqrt(x[i]), p = exp2((double)(ilogb(y[i]) - 1)) * 2;
    bad[0] += f64_bits(s) != f64_bits(sqrt_exact(x[i], (uint32_t)jitter));
    bad[1] += f64_bits(s * s) != f64_bits(sqrt_squared(x[i], (uint32_t)jitter));
    bad[2] += f64_bits(x[i] / y[i]) != f64_bits(div_exact(x[i], y[i], (uint32_t)jitter));
    bad[3] += f64_bits(-x[i] * y[i]) != f64_bits(mul_exact(-x[i], y[i]));
    bad[4] += f64_bits(x[i] * x[i]) != f64_bits(mul_exact(x[i], x[i]));
    // |x| > p / 2 and below 2^50 p: x scaled next to p
    const double v = (i & 1 ? -1.0 : 1.0) * x[i] * exp2((double)(ilogb(p) - ilogb(x[i]) + i % 49));
    const double w = fabs(v) > 0.5 * p ? v : p;
    bad[5] += f64_bits(copysign(p, w) - w) != f64_bits(fold_pow2(p, w));
  }
}
"""


@pytest.fixture(scope="module")
def compare(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact64")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I", _build.CSRC, "-I",
                           os.path.join(_build._cuda_home(), "include"), str(d / "t.cpp"), "-o", str(d / "t.so")])
    lib = ctypes.CDLL(str(d / "t.so"))

    def run(x, y, jitter):
        bad = np.zeros(6, np.int64)
        vp = ctypes.c_void_p
        lib.compare(x.ctypes.data_as(vp), y.ctypes.data_as(vp), ctypes.c_long(len(x)), jitter, bad.ctypes.data_as(vp))
        return bad
    return run


def _mantissas(rng, n):
    """Doubles of random, short and all-ones mantissas and exponents from 2^-60 to 2^60."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    k = rng.integers(0, 53, n).astype(np.uint64)
    kind = rng.integers(0, 4, n)
    m = np.where(kind == 1, (m >> k) << k, m)
    m = np.where(kind == 2, m | ((np.uint64(1) << np.uint64(52)) - (np.uint64(1) << np.minimum(k, np.uint64(51)))), m)
    e = rng.integers(1023 - 60, 1023 + 60, n).astype(np.uint64)
    return ((e << np.uint64(52)) | (m & np.uint64((1 << 52) - 1))).view(np.float64)


@pytest.mark.parametrize("jitter", [-4, -1, 0, 1, 4])
def test_integer_operations_equal_ieee(compare, jitter):
    rng = np.random.default_rng(7 + jitter)
    x, y = _mantissas(rng, 400000), _mantissas(rng, 400000)
    # squares and their neighbours, where the root's rounding is nearly a tie
    r = _mantissas(rng, 100000)
    near = (r * r).view(np.int64) + rng.integers(-2, 3, len(r))
    x[:len(r)] = near.view(np.float64)
    assert not compare(x, y, jitter).any()


BOXES = [{}, {"mandelbox_scale": -1.5}, {"mandelbox_scale": -2.0}, {"mandelbox_scale": 3.0}, {"mandelbox_scale": 0.5},
         {"mandelbox_folding_min_radius": 0.25}, {"mandelbox_folding_min_radius": 0.4},
         {"mandelbox_folding_min_radius": 1.0}, {"mandelbox_folding_min_radius": 1.5},
         {"mandelbox_folding_fixed_radius": 1.3}, {"mandelbox_folding_value": 1.0},
         {"mandelbox_folding_limit": 0.7, "mandelbox_folding_value": 1.4},
         {"mandelbox_folding_limit": 0.6, "mandelbox_folding_value": 2.0},
         {"mandelbox_folding_value": -2.0}, {"mandelbox_folding_limit": 0.0},
         {"julia_mode": 1, "julia_a": 0.3, "julia_b": -0.7, "julia_c": 0.0}, {"fractal_constant_factor": 0.5},
         {"N": 1}, {"N": 250}, {"interior_mode": 1}, {"iteration_threshold_mode": 1},
         {"limits_enabled": 1, "x_min": -3, "x_max": 2.5, "y_min": -4, "y_max": 1, "z_min": -5, "z_max": 5}]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 4133])
@pytest.mark.parametrize("keys", BOXES, ids=[",".join(f"{k.split('_')[-1]}={v}" for k, v in b.items()) or "usual" for b in BOXES])
def test_strict_box_distance_equals_oracle(gpu_ctx, oracle, keys, n):
    import torch
    sc = W.workload("mandelbox_1080p", 64, 48, **keys)
    rng = np.random.default_rng(11)
    pts = rng.uniform(-6.5, 6.5, (4133, 3))
    pts[:64] *= 0.05
    edge = [0.0, -0.0, 1.0, -1.0, 0.5, 2.0, 3.0, 1e-200, -1e-310, 0.25, 1e15, -4e15, 1e30, 1e95, 1e200, -1e300, np.inf,
            np.nan]
    pts[64:64 + 2000] = rng.choice(edge, (2000, 3))
    pts = np.ascontiguousarray(pts[:n])
    det = np.full(len(pts), 1e-3)
    ref, ref_it, ref_mi = oracle_lib.distance(oracle, sc, pts, det)
    p, d = torch.tensor(pts, device="cuda"), torch.tensor(det, device="cuda")
    out = torch.zeros(len(pts), dtype=torch.float64, device="cuda")
    it = torch.zeros(len(pts), dtype=torch.int32, device="cuda")
    mi = torch.zeros(len(pts), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    gpu_ctx.distance(sc, p.data_ptr(), d.data_ptr(), len(pts), out.data_ptr(), it.data_ptr(), mi.data_ptr(), mb.PREC_FP64)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    # beyond the limit box no orbit runs: itersOut stays as it was (the oracle's -1, the kernel's 0)
    np.testing.assert_array_equal(it.cpu().numpy(), np.where(ref_it == -1, 0, ref_it))
    np.testing.assert_array_equal(mi.cpu().numpy(), ref_mi)


@pytest.mark.gpu
@pytest.mark.parametrize("formula", [3, 4, 5, 6])
@pytest.mark.parametrize("keys", [{}, {"linear_DE_mode": 1, "N": 3}, {"julia_mode": 1, "julia_a": -0.6, "julia_b": 0.3, "julia_c": 0.1},
                                  {"fractal_constant_factor": 0.7, "N": 1}, {"minN": 5}], ids=str)
def test_strict_finite_difference_equals_oracle(gpu_ctx, oracle, formula, keys):
    # iterations equal and distances to log()'s last bits: the radii and their differences are
    # the reference's doubles, and only the logarithm may round differently (2 ulp of 1e-16)
    import torch
    sc = W.workload("mandelbulb_640x480", 64, 48, formula=formula, analityc_DE_mode=0, **{"N": 60, **keys})
    rng = np.random.default_rng(formula)
    pts = rng.uniform(-1.6, 1.6, (3000, 3))
    edge = [0.0, -0.0, 1.0, -1.0, 0.25, 1e-200, -1e-310, 3.0, -50.0, 1e9, 1e20, 1e160, np.inf, np.nan]
    pts[:600] = rng.choice(edge, (600, 3))
    det = np.full(len(pts), 1e-3)
    ref, ref_it, ref_mi = oracle_lib.distance(oracle, sc, pts, det)
    p, d = torch.tensor(pts, device="cuda"), torch.tensor(det, device="cuda")
    out = torch.zeros(len(pts), dtype=torch.float64, device="cuda")
    it = torch.zeros(len(pts), dtype=torch.int32, device="cuda")
    mi = torch.zeros(len(pts), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    gpu_ctx.distance(sc, p.data_ptr(), d.data_ptr(), len(pts), out.data_ptr(), it.data_ptr(), mi.data_ptr(), mb.PREC_FP64)
    np.testing.assert_array_equal(it.cpu().numpy(), ref_it)
    np.testing.assert_array_equal(mi.cpu().numpy(), ref_mi)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=1e-15, atol=0.0, equal_nan=True)
