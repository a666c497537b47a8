"""The FP64 polish at the faces of a limit box (needs a GPU). CalculateDistance returns early beyond a
face and leaves itersOut as the last orbit set it; a hit has run an orbit of at least one iteration
(minN 1), so no hit's iteration count is 0."""
import numpy as np
import pytest

import mandelbulber_gb300 as mb
from mandelbulber_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polish_all", [False, True])
@pytest.mark.parametrize("quality", [1, 30, 300])
@pytest.mark.parametrize("formula", [2, 7])
def test_hits_at_a_limit_face_keep_their_iterations(gpu_ctx, formula, quality, polish_all):
    sc = W.workload("mandelbulb_640x480", 320, 180, formula=formula, quality=quality, limits_enabled=1, x_min=-0.7,
                    x_max=0.5, y_min=-0.6, y_max=1, z_min=-0.4, z_max=0.4)
    img = gpu_ctx.render(sc, precision=mb.PREC_FP32_FIX, polish_all=polish_all)
    hit = img.hit == 1
    assert hit.any() and (img.iters[hit] > 0).all(), int((img.iters[hit] == 0).sum())
