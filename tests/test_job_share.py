"""How a stage's warps share its jobs (csrc/job_share.cuh, the code that the kernels run), on the
CPU: main launches of 152 SMs and the overflow pass's 2048 threads."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from mandelbulber_gb300 import _build

SOURCE = r"""
#include "job_share.cuh"
extern "C" void share(unsigned jobs, unsigned spread, unsigned launched, unsigned refill, unsigned *out) {
  const mbgb::dev::JobShare s = mbgb::dev::job_share(jobs, mbgb::dev::launch_spread(spread, launched), refill, 0, 0);
  out[0] = s.lanes; out[1] = s.warps; out[2] = s.refill;
}
"""


@pytest.fixture(scope="module")
def share(tmp_path_factory):
    d = tmp_path_factory.mktemp("share")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", _build.CSRC, "-I",
                           os.path.join(_build._cuda_home(), "include"), str(d / "t.cpp"), "-o", str(d / "t.so")])
    lib = ctypes.CDLL(str(d / "t.so"))

    def run(jobs, spread, launched, refill=8):
        out = (ctypes.c_uint * 3)()
        lib.share(jobs, spread, launched, refill, out)
        return tuple(out)
    return run


JOBS = sorted({*range(0, 70), 300, 607, 608, 609, 1999, 2000, 2001, 2431, 2432, 2433, 3000, 19455, 19456, 77824, 100000, 4000000000})


@pytest.mark.parametrize("spread", [152, 304, 608, 2432])
@pytest.mark.parametrize("launched", [16, 32, 64, 608, 4864])
def test_every_job_finds_a_lane_where_there_are_enough(share, spread, launched):
    for jobs in JOBS:
        lanes, warps, _ = share(jobs, spread, launched)
        assert 1 <= lanes <= 32 and (warps - 1) * lanes < max(jobs, 1)
        assert lanes * min(warps, launched) >= min(jobs, 32 * launched), (jobs, lanes, warps)


@pytest.mark.parametrize("refill", [1, 4, 8, 16, 32])
def test_full_warps_claim_at_the_threshold_that_was_asked_for(share, refill):
    assert share(2_000_000, 2432, 4864, refill) == (32, 62500, refill)
    lanes, _, got = share(19200, 2432, 4864, refill)   # 160x120: eight lanes a warp
    assert (lanes, got) == (8, max(1, refill // 4))
