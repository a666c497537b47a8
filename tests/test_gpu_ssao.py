"""The flat projection's SSAO kernel against the oracle over synthetic depth maps (needs a GPU):
odd sizes, the smallest and largest qualities, planes (many equal slopes), steps to the
background, zero and tiny depths. The oracle's slopes and sums are the reference's doubles; only
atan may round differently, so values agree to +-1 on at most 0.5 % (as the fixtures' test)."""
import ctypes

import numpy as np
import pytest

import mandelbulber_gb300 as mb
from mandelbulber_gb300 import workloads as W
from tests import oracle_lib
from tests.test_post import _within_one

pytestmark = pytest.mark.gpu


def _depth(kind, w, h, rng):
    y, x = np.mgrid[0:h, 0:w]
    if kind == "plane":
        return 3.0 + 0.01 * x + 0.02 * y
    if kind == "flat":
        return np.full((h, w), 2.5)
    if kind == "steps":
        z = 2.0 + rng.integers(0, 4, (h, w)) * 0.5
        z[rng.random((h, w)) < 0.3] = 1e20
        return z
    if kind == "tiny":
        z = rng.random((h, w)) * 10.0 ** rng.uniform(-30, 2, (h, w))
        z[0, 0] = 0.0
        return z
    return 5.0 + np.sin(x * 0.3) + np.cos(y * 0.2) + 0.05 * rng.normal(size=(h, w))


@pytest.mark.parametrize("w,h,quality", [(33, 32, 1), (1, 40, 7), (64, 48, 2), (97, 55, 5), (131, 67, 20), (48, 200, 33)])
@pytest.mark.parametrize("kind", ["plane", "flat", "steps", "tiny", "waves"])
def test_flat_ssao_equals_oracle(gpu_ctx, oracle, w, h, quality, kind):
    import torch
    rng = np.random.default_rng(w * 100 + quality)
    z = np.ascontiguousarray(_depth(kind, w, h, rng), np.float32)
    opacity = rng.integers(0, 65536, (h, w)).astype(np.uint16)
    colour = rng.integers(0, 256, (h, w, 3)).astype(np.uint8)
    image = rng.integers(0, 65536, (h, w, 3)).astype(np.uint16)
    sc = W.workload("mandelbox_1080p", w, h, post_SSAO_quality=quality)
    sc.image_width, sc.image_height, sc.SSAOQuality, sc.globalIlum = w, h, quality, 0.8
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    oracle.oracle_ssao.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p,
                                   ctypes.c_double, ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_void_p]
    want = image.copy()
    oracle.oracle_ssao(w, h, p(z), p(opacity), p(colour), sc.persp, quality, sc.perspectiveType, sc.globalIlum, p(want))
    t = [torch.tensor(a, device="cuda") for a in (z, opacity.view(np.int16), colour, image.view(np.int16))]
    torch.cuda.synchronize()
    v = [ctypes.c_void_p(a.data_ptr()) for a in t]
    layers = mb.mbgb_image(w, h, None, v[0], None, v[1], v[2], None, None, None)
    lib = mb.library()
    assert lib.mbgb_ssao_device(gpu_ctx._h, ctypes.byref(sc), ctypes.byref(layers), t[3].data_ptr()) == 0
    _within_one(t[3].cpu().numpy().view(np.uint16), want, kind)
