"""Pairs of kernels that share a dispatch, each pair run on both sides of its rule:

* the marching LINEAR backward kernel (tensor-map and element copies) against the gathering kernel
  k_sl_subcycle itself: CFD2LCS_B200_RUN=0 beside SL_TILE=0, since small grids otherwise advance
  several subcycles per launch with the marching kernel's own node routine;
* several subcycles per launch: fewer launches, the single library, the batched form on either side of
  its limit;
* lines too long for the chunked fits, in the library and in the adjoint;
* the composition of a cubic plane with its orders fixed at compile time and with general ones."""
import os

import numpy as np
import pytest

from tests import scenarios as SC
from tests import workloads as W

pytestmark = pytest.mark.gpu


def _api(prec="dp"):
    import libcfd2lcs_b200 as L
    return L.Cfd2lcs(prec)


def _case(api, env, case, integ, interp, n=None, steps=None, dirs=(SC.FTLE_BKWD,), mixed=False):
    env = {"CFD2LCS_B200_" + k: str(v) for k, v in env.items()}
    os.environ.update(env)
    try:
        api.reset()
        if mixed:
            api.set_option("MIXED_PRECISION", 1)
        _, hs = SC.run(api, case, dirs, integ, interp, n=n, steps=steps)
    finally:
        for k in env:
            os.environ.pop(k, None)
    assert api.error()[0] == 0, api.error()
    out = [f(h) for h in hs for f in (api.flowmap, api.ftle)]
    c, s = api.counters(), api.staged_launches()
    api.reset()
    return out, c, s


def _equal(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x, y), float(np.max(np.abs(x - y)))


@pytest.mark.parametrize("prec, case, n, integ, mixed, env", [
    ("dp", "abc", 38, 2, False, {}),                                           # box copies
    ("dp", "abc", 38, 3, False, {"SL_MARCH_KC": 7}),
    ("dp", "abc", 37, 2, False, {}),                                           # element copies: rows of 39 values
    ("dp", "abc", 37, 4, False, {"SL_MARCH_KC": 1}),
    ("dp", "abc", 70, 3, False, {"TMA_TENSOR": 0, "SL_MARCH_KC": 3}),          # three columns in x, partial ones
    ("dp", "abc_unsteady", 37, 3, False, {"SL_MARCH_KC": 64}),
    ("dp", "abc_unsteady", 38, 2, True, {"SL_MARCH_KC": 3}),                   # FP32 velocity beside FP64 maps
    ("dp", "channel", None, 3, False, {"TMA_TENSOR": 0, "SL_MARCH_KC": 4}),    # flags
    ("dp", "mixed_bc", None, 2, False, {}),
    ("sp", "abc", 38, 2, False, {}),
    ("sp", "turb", 37, 3, False, {"SL_MARCH_KC": 3}),
])
def test_march_against_the_gathering_kernel(prec, case, n, integ, mixed, env):
    api = _api(prec)
    steps = 10 if n and n > 30 else None
    a, _, s = _case(api, dict(env, SL_TILE=2), case, integ, 1, n, steps, mixed=mixed)
    assert s["sl_march"] == s["sl"] > 0
    b, _, s = _case(api, dict(RUN=0, SL_TILE=0), case, integ, 1, n, steps, mixed=mixed)
    assert s["sl"] == 0
    _equal(a, b)


@pytest.mark.parametrize("prec", ["dp", "sp"])
@pytest.mark.parametrize("case, n, integ", [("dg", 66, 2), ("abc", 33, 3)])
@pytest.mark.parametrize("direction", [SC.FTLE_FWD, SC.FTLE_BKWD])
def test_runs_take_fewer_launches(prec, case, n, integ, direction):
    api = _api(prec)
    a, ca, _ = _case(api, dict(SL_TILE=0), case, integ, 1, n, 9, dirs=(direction,))
    b, cb, _ = _case(api, dict(SL_TILE=0, RUN=0), case, integ, 1, n, 9, dirs=(direction,))
    key = "integrations_fwd" if direction == SC.FTLE_FWD else "integrations_bkwd"
    assert ca[key] == cb[key] > 9 * np.prod(a[1].shape)  # more than one subcycle per update
    assert ca["kernel_launches"] < cb["kernel_launches"]
    _equal(a, b)


def test_batched_runs_on_either_side_of_their_limit():
    """8 and 91 tiles of 32 x 8: within half the SMs of the device, and beyond (one launch per
    subcycle); the same instances alone run several subcycles per launch."""
    import torch

    import libcfd2lcs_b200 as L
    sizes, steps, dt = ((64, 32), (200, 100)), 9, 0.25
    grids = [W.double_gyre_grid(*s) for s in sizes]
    ref = []
    for g in grids:
        api = _api()
        api.reset()
        api.init(g.n, g.x, g.y, g.z, g.flag)
        h = api.diagnostic_init(SC.FTLE_BKWD, 0, 4 * dt, 2 * dt, "b")
        for k in range(steps):
            api.update(*W.double_gyre_velocity(g, k * dt), k * dt)
        assert api.error()[0] == 0, api.error()
        ref.append((api.flowmap(h), api.ftle(h)))
        api.reset()
    b = L.Batch("dp")
    b.reset()
    ids = [b.add(g.n, g.x, g.y, g.z, g.flag) for g in grids]
    hs = [b.diagnostic_init(i, SC.FTLE_BKWD, 4 * dt, 2 * dt) for i in ids]
    for k in range(steps):
        lev = [[torch.from_numpy(np.ascontiguousarray(a.ravel(order="F"))).cuda() for a in W.double_gyre_velocity(g, k * dt)] for g in grids]
        assert b.update_device(ids, *([v[c].data_ptr() for v in lev] for c in range(3)), [k * dt] * 2) == 0, b.error()
    for i, h, r in zip(ids, hs, ref):
        _equal((b.flowmap(i, h), b.ftle(i, h)), r)
    small, large = (b.counters(i)["kernel_launches"] for i in ids)
    assert small < large
    b.reset()


@pytest.mark.parametrize("prec, n", [("dp", 1800), ("sp", 3600)])
def test_lines_too_long_for_the_chunks(prec, n, oracle_dp, oracle_sp):
    """Past 1792 (FP32: 3584) padded points the x axis is swept as whole lines."""
    oracle = oracle_dp if prec == "dp" else oracle_sp
    g = W.abc_grid(n, nj=4, nk=4)
    vel = W.abc_velocity(g)
    api, maps = _api(prec), []
    for a in (api, oracle):
        a.reset()
        a.init(g.n, g.x, g.y, g.z, g.flag)
        hs = [a.diagnostic_init(d, 0, 0.02, 0.01, f"d{d}") for d in (SC.FTLE_FWD, SC.FTLE_BKWD)]
        a.set_option("INTEGRATOR", 2)
        a.set_option("INTERPOLATOR", 3)
        for k in range(5):
            a.update(*vel, k * 0.005)
        maps.append([a.flowmap(h) for h in hs])
    assert api.error()[0] == 0, api.error()
    # the suite's bounds on composed maps: 1e-12 of the domain in FP64, 2e-5 in FP32
    bound = (1e-12 if prec == "dp" else 2e-5) * 2 * np.pi
    for x, y in zip(*maps):
        assert np.max(np.abs(x - y)) <= bound
    api.reset()
    oracle.reset()


def test_cubic_adjoint_on_lines_too_long_for_the_chunks():
    """The transposed whole-line solve: dJ of the tangent model equals <gradient, d>."""
    import torch

    import libcfd2lcs_b200 as L
    g, nl, dt = W.abc_grid(1800, nj=4, nk=4), 4, 0.002
    rng = np.random.default_rng(7)
    base = W.abc_velocity(g)
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a.ravel(order="F"))).cuda()
    lev = [[cuda(b + 0.05 * rng.standard_normal(b.shape)) for _ in range(nl)] for b in base]
    d = [[cuda(rng.standard_normal(b.shape)) for _ in range(nl)] for b in base]
    weight, times = cuda(rng.random(g.n) / g.npts), [k * dt for k in range(nl)]
    J, *grad = L.adjoint_ftle(g, *lev, times, weight, interpolator=3, checkpoint_every=2)
    Jt, dJ = L.tangent_ftle(g, *lev, times, weight, *d, interpolator=3)
    assert Jt == J
    ad = sum(float(torch.dot(grad[c][k], d[c][k])) for c in range(3) for k in range(nl))
    size = sum(float((grad[c][k] * d[c][k]).abs().sum()) for c in range(3) for k in range(nl))
    assert abs(dJ - ad) <= 1e-11 * size, (dJ, ad)


@pytest.mark.parametrize("n, steps", [(64, 40), (97, 12)])
def test_composition_of_a_cubic_plane(n, steps):
    """Steps with re-sorted particles and general orders (what planes of 2^20 points and more take)
    against the node-ordered composition with orders 4, 4 and 2: the same sums in the same order."""
    api = _api()
    both = (SC.FTLE_BKWD, SC.FTLE_FWD)
    a, ca, _ = _case(api, dict(COMPOSE_SORT_MIN=0), "dg", 2, 3, n, steps, dirs=both)
    b, cb, _ = _case(api, dict(COMPOSE_SORT_MIN=1 << 40), "dg", 2, 3, n, steps, dirs=both)
    assert ca["slots_composed"] == cb["slots_composed"] > ca["ftle_frames"]
    _equal(a, b)
