"""The lean Mandelbulb's fast AO (needs a GPU): the shadow stage's values (orbit-granular refill) are
the composition's (without), bit for bit, up to the quality whose last weights 2^-i underflow."""
import numpy as np
import pytest

from mandelbulber_gb300 import workloads as W

pytestmark = pytest.mark.gpu
LAYERS = ["image_float", "zbuffer", "alpha", "opacity", "colour"]


@pytest.mark.parametrize("quality", [1, 2, 4, 12, 13])
@pytest.mark.parametrize("keys", [{}, {"interior_mode": 1}, {"quality": 0.3, "ambient_occlusion_fast_tune": 0.3}], ids=str)
def test_fast_ao_does_not_depend_on_the_stage(gpu_ctx, quality, keys):
    sc = W.workload("mandelbulb_640x480", 83, 61, ambient_occlusion_enabled=1, fast_ambient_occlusion_mode=1,
                    ambient_occlusion_quality=quality, **keys)
    got, want = gpu_ctx.render(sc), gpu_ctx.render(sc, orbit_refill=-1)
    for k in LAYERS:
        np.testing.assert_array_equal(getattr(got, k), getattr(want, k), err_msg=k)
