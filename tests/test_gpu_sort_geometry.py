"""The staged forward kernel reads the tiles of the last sort, so a sort made for another kernel ends its
use until the particles are sorted for it again.  INTERPOLATOR may change between updates: LINEAR
updates sort into the gathering kernels' tiles, and the CUBIC update after one has to sort first."""
import os

import numpy as np
import pytest

from tests import scenarios as SC
from tests import workloads as W

pytestmark = pytest.mark.gpu

N = 24
DT = 1.5 * 0.5 * (2 * np.pi / N) / 7.2  # two subcycles (the ABC flow's sum of |u_a| is up to 7.2)


def _run(api, staged):
    env = {"CFD2LCS_B200_SL_TILE": "2" if staged else "0", "CFD2LCS_B200_SORT_EVERY": "3"}
    os.environ.update(env)
    try:
        api.reset()
        g = W.abc_grid(N)
        api.init(g.n, g.x, g.y, g.z, g.flag)
    finally:
        for k in env:
            os.environ.pop(k, None)
    h = api.diagnostic_init(SC.FTLE_FWD, 0, 4.5 * DT, 4.5 * DT, "f")
    api.set_option("INTEGRATOR", 2)
    launches = []
    for k, interp in enumerate((1, 3, 1, 3, 3)):  # LINEAR, CUBIC, LINEAR, CUBIC, and a frame
        api.set_option("INTERPOLATOR", interp)
        before = api.counters()["kernel_launches"]
        api.update(*W.abc_velocity(g), k * DT if k < 4 else 5 * DT)
        launches.append(api.counters()["kernel_launches"] - before)
        if 0 < k < 4:
            assert api.counters()["nsub_fwd"] == 2
    assert api.error()[0] == 0, api.error()
    out = api.flowmap(h), api.ftle(h)
    n = api.staged_launches()["fwd"]
    api.reset()
    return launches, out, n


def test_a_sort_for_another_kernel_ends_the_staged_one():
    import libcfd2lcs_b200 as L
    api = L.Cfd2lcs("dp")
    launches, a, n = _run(api, True)
    assert n > 0
    # subcycles since the last sort: 1, then the first CUBIC update sorts (2); the LINEAR update sorts
    # after its first subcycle (1), so the second CUBIC update has to sort again: the same launches
    assert launches[3] == launches[1], launches
    _, b, n = _run(api, False)
    assert n == 0
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [(162, 162, 162), (40, 330, 330), (1030, 1024, 1)])
def test_large_grid_tiles_keep_bits(n):
    """The 64 x 2 x 2 (32 x 4 x 2 on short rows) tiles of large FP64 grids against particles that are
    never sorted: particles are advanced one by one, so the order of their slots changes nothing."""
    import libcfd2lcs_b200 as L
    api = L.Cfd2lcs("dp")
    out = []
    for every in ("1", "1000000"):
        env = {"CFD2LCS_B200_SL_TILE": "0", "CFD2LCS_B200_SORT_EVERY": every}
        os.environ.update(env)
        try:
            api.reset()
            g = W.double_gyre_grid(*n[:2]) if n[2] == 1 else W.abc_grid(n[0], nj=n[1], nk=n[2])
            api.init(g.n, g.x, g.y, g.z, g.flag)
        finally:
            for k in env:
                os.environ.pop(k, None)
        dt = (40 if n[2] == 1 else 14) / max(n)  # the second update passes 32 subcycles, where the tiles change
        h = api.diagnostic_init(SC.FTLE_FWD, 0, 2 * dt, 2 * dt, "f")
        api.set_option("INTEGRATOR", 2)
        api.set_option("INTERPOLATOR", 3)
        vel = W.double_gyre_velocity if n[2] == 1 else W.abc_velocity
        for k in range(3):
            api.update(*vel(g, 0.0), k * dt)
        assert api.error()[0] == 0, api.error()
        out.append((api.flowmap(h), api.counters()["kernel_launches"]))
    api.reset()
    assert out[0][1] > out[1][1]  # it was sorted
    assert np.array_equal(out[0][0], out[1][0])
