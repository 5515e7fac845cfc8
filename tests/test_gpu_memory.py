"""Device memory that only saves time -- the blend buffers beyond those a subcycle needs, and what the
adjoint keeps between calls -- is taken while half of the device stays free, and given back when one of
the library's own allocations would fail otherwise."""
import os

import numpy as np
import pytest

from tests import scenarios as SC
from tests import workloads as W

pytestmark = pytest.mark.gpu

N = 120
FIELD = (N + 2) ** 3 * 8  # bytes of one padded FP64 component
SLACK = 8 << 20           # allocation granularity


def _used():
    import torch
    free, total = torch.cuda.mem_get_info()
    return total - free


def _fill(leave):
    """Device memory taken so that `leave` bytes stay free."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")


def _drop():
    import torch
    torch.cuda.empty_cache()


def _instance():
    """A LINEAR RK2 instance with one forward set whose stages are blended fields."""
    import libcfd2lcs_b200 as L
    os.environ["CFD2LCS_B200_LINEAR_BLEND_MIN"] = "0"
    try:
        a = L.Cfd2lcs("dp")
        a.reset()
        g = W.abc_grid(N)
        a.init(g.n, g.x, g.y, g.z, g.flag)
    finally:
        os.environ.pop("CFD2LCS_B200_LINEAR_BLEND_MIN", None)
    a.diagnostic_init(SC.FTLE_FWD, 0, 100.0, 100.0, "f")
    a.set_option("INTEGRATOR", 2)
    a.set_option("INTERPOLATOR", 1)
    a.grid = g
    return a


@pytest.fixture(scope="module")
def loaded():
    """The kernels' code and stacks in device memory before anything is counted."""
    a = _instance()
    _update(a, 0.0)
    _update(a, LARGE)
    a.reset()
    _gradient()
    a.reset()
    _drop()


@pytest.fixture
def api(loaded):
    a = _instance()
    yield a
    a.reset()
    _drop()


def _update(a, t):
    a.update(*W.abc_velocity(a.grid), t)
    assert a.error()[0] == 0, a.error()


SMALL, LARGE = 0.25 * 2 * np.pi / N / 4.0, 6.0 * 2 * np.pi / N / 4.0  # one subcycle, several


def test_one_subcycle_takes_the_blends_it_needs(api):
    before = _used()
    _update(api, 0.0)
    _update(api, SMALL)
    assert api.counters()["nsub_fwd"] == 1
    assert _used() - before <= 2 * 3 * FIELD + SLACK  # RK2: two stage fractions


def test_several_subcycles_take_the_rest_only_with_room(api):
    before = _used()
    _update(api, 0.0)
    hog = _fill(2 << 30)
    held = _used()
    _update(api, LARGE)
    assert api.counters()["nsub_fwd"] > 2
    assert _used() - held <= 3 * FIELD + SLACK
    del hog
    _drop()
    assert _used() - before <= 2 * 3 * FIELD + SLACK


def test_blends_make_room_for_a_diagnostic(api):
    """With the optional buffers taken, a diagnostic that fits only in their place."""
    _update(api, 0.0)
    before = _used()
    _update(api, LARGE)
    optional = _used() - before
    assert optional >= 4 * 3 * FIELD
    before = _used()
    api.diagnostic_init(SC.FTLE_FWD, 0, 100.0, 100.0, "g")
    diag = _used() - before
    hog = _fill(diag - optional // 2)
    api.diagnostic_init(SC.FTLE_FWD, 0, 100.0, 100.0, "h")
    assert api.error()[0] == 0, api.error()
    del hog
    _drop()
    _update(api, 2 * LARGE)


def _gradient(n=40, levels=4):
    import torch

    import libcfd2lcs_b200 as L
    g = W.abc_grid(n)
    base = [torch.from_numpy(np.ascontiguousarray(a.ravel(order="F"))).cuda() for a in W.abc_velocity(g)]
    weight = torch.ones(g.npts, dtype=torch.float64, device="cuda")
    out = L.adjoint_ftle(g, *([a] * levels for a in base), [0.05 * k for k in range(levels)], weight)
    torch.cuda.synchronize()
    return out


def test_adjoint_keeps_memory_only_with_room(loaded):
    import torch

    import libcfd2lcs_b200 as L
    L.Cfd2lcs("dp").reset()
    torch.cuda.empty_cache()
    _gradient()
    torch.cuda.empty_cache()
    kept = _used()
    L.Cfd2lcs("dp").reset()
    assert kept - _used() >= 32 << 20  # the pool is kept between calls, and given back
    hog = _fill(2 << 30)
    held = _used()
    out = _gradient()
    del out
    torch.cuda.empty_cache()
    assert _used() - held <= 2 * SLACK
    del hog
    _drop()
