"""The chunked spline fits (k_fit_block) against the oracle's whole-line solves: CUBIC and QUADRATIC
runs whose axes fall on either side of the kernel's line widths (32, 16 and 8 lines per block),
with fewer points than chunks, and with velocity and flow-map lines that are constant along an axis
(the lines whose chunks are swept again)."""
import numpy as np
import pytest

from tests import scenarios as SC
from tests import workloads as W

pytestmark = pytest.mark.gpu


def _run(api, g, vel, interp, steps=6, dt=0.05):
    api.reset()
    api.init(g.n, g.x, g.y, g.z, g.flag)
    hd = [api.diagnostic_init(d, 0, 0.2, 0.1, f"d{d}") for d in (SC.FTLE_FWD, SC.FTLE_BKWD)]
    api.set_option("INTEGRATOR", 2)
    api.set_option("INTERPOLATOR", interp)
    for k in range(steps):
        api.update(*vel(k * dt), k * dt)
    return hd


def _shear(g, t):
    """u(z) only: its lines, and those of the displacement it makes, are constant in x and y."""
    u = np.asfortranarray(0.3 + 0.2 * np.sin(g.z) + 0.0 * g.x)
    return u, np.asfortranarray(0.0 * g.x), np.asfortranarray(0.0 * g.x)


@pytest.mark.parametrize("n, flow, interp", [
    ((25, 4, 5), "abc", 3),       # 7 and 6 points on the short axes: fewer than chunks
    ((24, 26, 31), "shear", 3),   # constant lines; 26 and 28 points: edge of the y / z rule
    ((24, 23, 22), "abc", 2),     # order 3: two off-diagonal factors on every row
    ((448, 5, 4), "abc", 3),      # 16 lines per block in FP64
    ((900, 4, 4), "shear", 3),    # 8 lines per block
    ((1700, 4, 4), "abc", 3),     # too long to stage: whole-line sweeps
])
def test_fit_against_oracle(n, flow, interp, oracle_dp):
    import libcfd2lcs_b200 as L
    g = W.abc_grid(n[0], nj=n[1], nk=n[2])
    vel = (lambda t: _shear(g, t)) if flow == "shear" else (lambda t: tuple(0.02 * a for a in W.abc_velocity(g, t)))
    gpu = L.Cfd2lcs("dp")
    hg = _run(gpu, g, vel, interp)
    ho = _run(oracle_dp, g, vel, interp)
    assert gpu.error()[0] == 0, gpu.error()
    for a, b in zip(hg, ho):
        # the suite's FP64 B-spline bound on composed maps, 1e-12 of the domain
        assert np.max(np.abs(gpu.flowmap(a) - oracle_dp.flowmap(b))) <= 1e-12 * 2 * np.pi
    gpu.reset()
    oracle_dp.reset()
