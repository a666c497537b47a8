"""Device memory that a context takes for a call (needs a GPU): buffers that only some scenes read are
held by those alone."""
import ctypes

import pytest

import mandelbulber_gb300 as mb
from mandelbulber_gb300 import workloads as W

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def _held(call):
    """Bytes that a new context holds after `call(context)`."""
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with mb.Context(0) as ctx:
        call(ctx)
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0]


def test_hit_values_are_held_where_the_shadow_stage_writes_them(gpu_ctx):
    """A value per hit of colour, normal and fast AO, [5][pixels] floats: the lean Mandelbulb with
    orbit-granular refill; not without it, and not the Mandelbox."""
    import torch
    w, h = 1920, 1080
    image = torch.zeros((h, w, 3), device="cuda")

    def frame(precision=mb.PREC_FP32_FIX, formula=2, **opts):
        sc = W.workload("mandelbulb_640x480", w, h, formula=formula, N=10)
        call = lambda ctx: ctx.render_device(sc, {"image_float": image.data_ptr()}, precision=precision, **opts)  # noqa: E731
        call(gpu_ctx)   # code and stacks are loaded by the first call
        return _held(call)
    with_jobs = frame()
    values = 5 * 4 * w * h
    assert with_jobs - frame(orbit_refill=-1) > values - 4 * MIB
    assert with_jobs - frame(formula=8) > values - 4 * MIB
    # FP64: every array at most twice as wide, without the values
    assert frame(precision=mb.PREC_FP64) < 2 * (with_jobs - values) + 4 * MIB


def test_ssao_of_other_projections_holds_its_directions_alone(gpu_ctx):
    """The flat kernel's samples (48 bytes x quality (quality - 1)) and open list (4 bytes a pixel):
    fish eye and equirectangular frames run ssao_kernel<double>, which reads neither."""
    import torch
    w, h, quality = 64, 48, 1000
    t = [torch.zeros((h, w), device="cuda") + 2.0, torch.zeros((h, w), dtype=torch.int16, device="cuda"),
         torch.zeros((h, w, 3), dtype=torch.uint8, device="cuda"), torch.zeros((h, w, 3), dtype=torch.int16, device="cuda")]
    t[0][:] = 1e20   # background: no search
    p = [ctypes.c_void_p(v.data_ptr()) for v in t]
    layers = mb.mbgb_image(w, h, None, p[0], None, p[1], p[2], None, None, None)

    def call(ptype):
        sc = W.workload("mandelbulb_640x480", w, h, post_SSAO_quality=quality)
        sc.SSAOQuality, sc.perspectiveType = quality, ptype

        def run(ctx):
            assert mb.library().mbgb_ssao_device(ctx._h, ctypes.byref(sc), ctypes.byref(layers), t[3].data_ptr()) == 0
        run(gpu_ctx)
        return _held(run)
    flat = call(0)
    for ptype in (1, 2):
        assert flat - call(ptype) > 48 * quality * (quality - 1) - 4 * MIB
