"""Launches that advance several subcycles (k_sl_run, k_fwd_run: LINEAR and the other interpolators
without B-splines) against one launch per subcycle (CFD2LCS_B200_RUN=0 at cfd2lcs_init): the same
expressions, so flow maps and FTLE must be bitwise equal.  Sizes at the edges of the 32 x 8 and
32 x 2 x 4 tiles, one tile and several, with flags and without, more subcycles than one launch takes
(16), both parities of the flow-map buffers, and the batched form's streams."""
import os

import numpy as np
import pytest

from tests import scenarios as SC
from tests import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_dp():
    import libcfd2lcs_b200 as L
    return L.Cfd2lcs("dp")


def _run(gpu, run, g, vel, dirs, integ, interp, dt, steps, h, mixed=False):
    # SL_TILE=0: on three-dimensional grids the reference side gathers too
    env = {"CFD2LCS_B200_RUN": "1" if run else "0", "CFD2LCS_B200_SL_TILE": "0"}
    os.environ.update(env)
    try:
        gpu.reset()
        if mixed:
            gpu.set_option("MIXED_PRECISION", 1)
        gpu.init(g.n, g.x, g.y, g.z, g.flag)
        hs = [gpu.diagnostic_init(d, 0, 2 * h, h, f"d{d}") for d in dirs]
        gpu.set_option("INTEGRATOR", integ)
        gpu.set_option("INTERPOLATOR", interp)
        for k in range(steps):
            gpu.update(*vel(k * dt), k * dt)
    finally:
        for k in env:
            os.environ.pop(k, None)
    assert gpu.error()[0] == 0, gpu.error()
    return [f(h) for h in hs for f in (gpu.flowmap, gpu.ftle)], gpu.counters()


BOTH = (SC.FTLE_FWD, SC.FTLE_BKWD)


@pytest.mark.parametrize("case, n, integ, interp, dt, steps, mixed", [
    ("dg", 32, 2, 1, 0.125, 9, False),     # one column of tiles in y, 1 to 3 subcycles
    ("dg", 66, 3, 1, 0.125, 9, False),     # partial tiles in x and y
    ("dg", 200, 2, 1, 0.5, 5, False),      # more subcycles than one launch holds
    ("abc", 16, 2, 1, 0.125, 9, False),    # 3-D tiles without flags
    ("abc", 33, 4, 1, 0.125, 9, True),     # partial 3-D tiles, FP32 velocity
    ("channel", None, 1, 1, 0.125, 9, False),
    ("mixed_bc", None, 0, 1, 0.125, 9, False),
    ("mixed_bc", None, 2, 0, 0.125, 9, False),  # NEAREST: forward only takes the longer launches
    ("curv_box", 12, 2, 6, 0.125, 9, False),
])
def test_run_equals_single_launches(gpu_dp, case, n, integ, interp, dt, steps, mixed):
    g, vel, _ = SC.make_case(case, n)
    a, ca = _run(gpu_dp, True, g, vel, BOTH, integ, interp, dt, steps, 4 * dt, mixed)
    b, cb = _run(gpu_dp, False, g, vel, BOTH, integ, interp, dt, steps, 4 * dt, mixed)
    for key in ("integrations_fwd", "integrations_bkwd", "ftle_frames"):
        assert ca[key] == cb[key]
    assert ca["kernel_launches"] <= cb["kernel_launches"]
    for x, y in zip(a, b):
        assert np.array_equal(x, y), np.max(np.abs(x - y))
    gpu_dp.reset()
