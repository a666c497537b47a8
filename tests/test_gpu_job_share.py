"""Frames with fewer rays than the machine has lanes: the stages hand a warp fewer jobs and let
the first warps take them (job_share), which moves rays between lanes and changes no pixel."""
import numpy as np
import pytest

import mandelbulber_gb300 as mb
from mandelbulber_gb300 import workloads as W

pytestmark = pytest.mark.gpu
LAYERS = ["image_float", "zbuffer", "alpha", "opacity", "colour", "hit", "iters", "depth"]


@pytest.mark.parametrize("name,precision", [("mandelbulb_640x480", mb.PREC_FP32_FIX), ("mandelbulb_640x480", mb.PREC_FP64),
                                            ("mandelbox_1080p", mb.PREC_FP32_FIX), ("mandelbox_1080p", mb.PREC_FP64)])
@pytest.mark.parametrize("w,h", [(32, 32), (33, 37), (71, 45), (160, 121)])
def test_small_frames_do_not_depend_on_the_sharing(gpu_ctx, name, precision, w, h):
    sc = W.workload(name, w, h, N=12)
    ref = gpu_ctx.render(sc, precision=precision)
    n = gpu_ctx.stats().de_calls
    for o in ({"ctas_per_sm": 1}, {"threads_per_cta": 32}, {"threads_per_cta": 64, "ctas_per_sm": 3}, {"refill_min": 1}):
        got = gpu_ctx.render(sc, precision=precision, **o)
        assert gpu_ctx.stats().de_calls == n, o
        for k in LAYERS:
            np.testing.assert_array_equal(getattr(ref, k), getattr(got, k), err_msg=f"{o} layer {k}")
