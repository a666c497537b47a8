"""Mandelbox settings at the ends of what the strict and lean orbits accept (needs a GPU)."""
import numpy as np
import pytest

import mandelbulber_gb300 as mb
from mandelbulber_gb300 import workloads as W
from tests import oracle_lib

pytestmark = pytest.mark.gpu
LAYERS = ["image_float", "zbuffer", "alpha", "opacity", "colour", "hit", "iters", "depth"]


@pytest.mark.parametrize("value", [0.0, 2.0])
def test_fold_limit_of_negative_zero_folds(gpu_ctx, oracle, value):
    """-0 is a limit of 0: |x| > 0 folds. The distances are the oracle's bit for bit and the frames
    those of a limit of +0 (value 0: the lean FP32 orbit and its FP64 polish)."""
    import torch
    sc, plus = (W.workload("mandelbox_1080p", 97, 55, mandelbox_folding_limit=v, mandelbox_folding_value=value)
                for v in (-0.0, 0.0))
    pts = np.random.default_rng(3).uniform(-6.5, 6.5, (501, 3))
    det = np.full(len(pts), 1e-3)
    ref, ref_it, _ = oracle_lib.distance(oracle, sc, pts, det)
    p, d = torch.tensor(pts, device="cuda"), torch.tensor(det, device="cuda")
    out = torch.zeros(len(pts), dtype=torch.float64, device="cuda")
    it = torch.zeros(len(pts), dtype=torch.int32, device="cuda")
    mi = torch.zeros(len(pts), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    gpu_ctx.distance(sc, p.data_ptr(), d.data_ptr(), len(pts), out.data_ptr(), it.data_ptr(), mi.data_ptr(), mb.PREC_FP64)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    np.testing.assert_array_equal(it.cpu().numpy(), ref_it)
    for o in ({"precision": mb.PREC_FP64}, {"precision": mb.PREC_FP32_FIX, "polish_all": True}):
        got, want = gpu_ctx.render(sc, **o), gpu_ctx.render(plus, **o)
        for k in LAYERS:
            np.testing.assert_array_equal(getattr(got, k), getattr(want, k), err_msg=f"{o} layer {k}")


@pytest.mark.parametrize("radius", [2.0, 1.2])
def test_min_radius_beyond_the_fixed_one_has_no_sign(gpu_ctx, oracle, radius):
    """The sphere fold squares its radii: a min radius of -2 is the frame of 2, whose fold is no
    clamp, so the lean FP32 orbit applies to neither."""
    minus, plus = (W.workload("mandelbox_1080p", 96, 54, mandelbox_folding_min_radius=r) for r in (-radius, radius))
    ref, _ = oracle_lib.render(oracle, minus)
    for o in ({}, {"polish_all": True}, {"precision": mb.PREC_FP64}):
        got, want = gpu_ctx.render(minus, **o), gpu_ctx.render(plus, **o)
        for k in LAYERS:
            np.testing.assert_array_equal(getattr(got, k), getattr(want, k), err_msg=f"{o} layer {k}")
        np.testing.assert_array_equal(got.hit, ref.hit)
