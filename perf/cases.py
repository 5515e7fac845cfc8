"""The workloads whose speed is watched, each run through the library's public entry points.

A pass is what a flow solver has the library do over one whole integration time T: the velocity
field of every solver step handed to update(), and the FTLE field read at the end.  A case names
its grid and flow, the options a user sets (precision, integrator, interpolator, direction), how
many solver steps lie between two sub-flow maps (`per_h`) and how many sub-flow maps one frame
composes (`slots`), so a pass is per_h * slots updates and its last frame composes every sub-map
of the pass.  The reference keeps one library instance per process, so the states of one case
share it: the instance is the handle a user's program keeps, a state holds the velocity fields.

Two choices make a pass repeatable.  Times are multiples of a power of two, so the subcycle
counts and stage fractions do not drift with the solver time.  And the velocity of a seed,
base + s(t) * (its own disturbance), has s = 0 at both ends of a pass, so a pass starts from the
same velocity level whatever ran before it.
"""
import math
import types

import numpy as np
import torch

import libcfd2lcs_b200 as L

INTEGRATORS = {"rk2": L.RK2, "rk3": L.RK3, "rk4": L.RK4}
INTERPOLATORS = {"linear": L.LINEAR, "cubic": L.CUBIC}
DIRECTIONS = {"backward": (L.FTLE_BKWD,), "forward": (L.FTLE_FWD,), "both": (L.FTLE_FWD, L.FTLE_BKWD)}
STAGES = {"rk2": 2, "rk3": 3, "rk4": 4}
CFL = 0.5  # the reference's default subcycle limit
TWO_PI = 2.0 * math.pi
DEV = "cuda"

# Largest sum over the axes of |u_a| * (points per unit length along a), per point along an axis
# of the flow's domain: what sets the number of subcycles.  Only work() and draw() use it.
RATE = {"gyre": 0.42, "abc": 0.95, "turbulence": 1.25, "duct": 0.75, "channel": 0.62}


def listed():
    return [
        # a small two-dimensional solver on the host: the drop-in call with host arrays, the
        # smallest call there is; what counts is the time of one update, not bandwidth
        dict(name="gyre small, host arrays", kind="flow", flow="gyre", ni=64, nj=32, nk=1, dt_log2=-3, per_h=4, slots=4,
             precision="dp", integrator="rk2", interpolator="linear", direction="backward", host=True),
        # the double gyre at the benchmark's size: two-dimensional fields that fit in the cache
        dict(name="gyre 512x256", kind="flow", flow="gyre", ni=512, nj=256, nk=1, dt_log2=-3, per_h=4, slots=5,
             precision="dp", integrator="rk2", interpolator="linear", direction="backward", host=False),
        # a plane of odd sizes with the smooth interpolator, both directions
        dict(name="gyre ragged cubic", kind="flow", flow="gyre", ni=1001, nj=487, nk=1, dt_log2=-4, per_h=2, slots=3,
             precision="dp", integrator="rk3", interpolator="cubic", direction="both", host=False),
        # a solver with inflow, outflow, slip walls and masked nodes that hands over host arrays
        dict(name="duct, host arrays", kind="flow", flow="duct", ni=101, nj=75, nk=50, dt_log2=-5, per_h=4, slots=2,
             precision="dp", integrator="rk3", interpolator="cubic", direction="both", host=True),
        # walls and a stretched grid, the classical integrator
        dict(name="channel ragged rk4", kind="flow", flow="channel", ni=191, nj=129, nk=95, dt_log2=-5, per_h=4, slots=2,
             precision="dp", integrator="rk4", interpolator="linear", direction="both", host=False),
        # the benchmark's default: ABC flow, both directions, cubic B-splines in FP64
        dict(name="abc 256 cubic", kind="flow", flow="abc", ni=256, nj=256, nk=256, dt_log2=-6, per_h=3, slots=2,
             precision="dp", integrator="rk3", interpolator="cubic", direction="both", host=False),
        # the same flow with the reference's default interpolator
        dict(name="abc 256 linear", kind="flow", flow="abc", ni=256, nj=256, nk=256, dt_log2=-6, per_h=4, slots=2,
             precision="dp", integrator="rk2", interpolator="linear", direction="both", host=False),
        # the mixed-precision option on an odd-sized box
        dict(name="abc ragged mixed cubic", kind="flow", flow="abc", ni=173, nj=160, nk=147, dt_log2=-5, per_h=3, slots=2,
             precision="mixed", integrator="rk3", interpolator="cubic", direction="both", host=False),
        # the single-precision library on turbulence
        dict(name="turbulence single", kind="flow", flow="turbulence", ni=200, nj=200, nk=200, dt_log2=-6, per_h=4, slots=3,
             precision="sp", integrator="rk2", interpolator="linear", direction="both", host=False),
        # turbulence in FP64, the largest grid here: fields of 0.45 GB per component
        dict(name="turbulence 384", kind="flow", flow="turbulence", ni=384, nj=384, nk=384, dt_log2=-7, per_h=4, slots=2,
             precision="dp", integrator="rk2", interpolator="linear", direction="backward", host=False),
        # many small instances advanced together, gyres and cubes of uneven sizes
        dict(name="batch of 16", kind="batch", gyres=8, cubes=8, largest=96, mix=64, updates=6, precision="dp",
             interpolator="linear"),
        # gradient of a mean FTLE with respect to the velocity at every level, single precision
        dict(name="gradient 80", kind="gradient", n=80, dt_log2=-5, levels=11, checkpoint=4, precision="sp", integrator="rk2",
             interpolator="linear"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dt_log2(rate, subcycles):
    """The power of two nearest to the step that takes about this many subcycles."""
    return int(round(math.log2(subcycles * CFL / rate)))


def draw(rng):
    kind = rng.choice(["gyre", "gyre", "duct", "channel", "cube", "cube", "cube", "batch", "gradient"])
    interp, integ = rng.choice(["linear", "cubic"]), rng.choice(["rk2", "rk3"])
    if kind == "batch":
        return dict(kind="batch", gyres=rng.randint(2, 10), cubes=rng.randint(2, 10), largest=_log_int(rng, 32, 96),
                    mix=rng.randint(1, 10**6), updates=6, precision=rng.choice(["dp", "mixed"]), interpolator=interp)
    if kind == "gradient":
        n, prec = _log_int(rng, 20, 72), rng.choice(["sp", "sp", "dp"])
        return dict(kind="gradient", n=n, dt_log2=_dt_log2(RATE["abc"] * n, rng.uniform(2, 5)), levels=rng.randint(5, 10),
                    checkpoint=rng.randint(2, 6), precision=prec, integrator=rng.choice(["rk2", "rk3"]), interpolator=interp)
    case = dict(kind="flow", precision=rng.choice(["dp", "dp", "sp", "mixed"]), integrator=integ, interpolator=interp,
                direction=rng.choice(["backward", "forward", "both"]), host=False, slots=rng.randint(2, 4), per_h=rng.randint(2, 4))
    if kind == "gyre":
        ni = _log_int(rng, 64, 1024)
        case.update(flow="gyre", ni=ni, nj=ni // 2 + rng.randint(-9, 9), nk=1, host=ni < 400 and rng.random() < 0.5)
    elif kind == "duct":
        n = _log_int(rng, 40, 140)
        case.update(flow="duct", ni=n, nj=n - rng.randint(0, n // 4), nk=n - rng.randint(0, n // 2), host=rng.random() < 0.5)
    elif kind == "channel":
        n = _log_int(rng, 40, 190)
        case.update(flow="channel", ni=n, nj=n - rng.randint(0, n // 3), nk=n - rng.randint(0, n // 2), interpolator="linear",
                    integrator=rng.choice(["rk2", "rk4"]))
    else:
        n = _log_int(rng, 32, 224)
        case.update(flow=rng.choice(["abc", "turbulence"]), ni=n, nj=max(24, n - rng.randint(0, n // 5)),
                    nk=max(24, n - rng.randint(0, n // 5)))
    case["dt_log2"] = _dt_log2(RATE[case["flow"]] * max(case["ni"], case["nj"], case["nk"]), rng.uniform(2, 7))
    return case


# ------------------------------------------------------------------------------- grids
def _grid(xl, yl, zl, flag=None):
    n = (len(xl), len(yl), len(zl))
    g = types.SimpleNamespace(n=n, lines=(xl, yl, zl))
    g.x, g.y, g.z = (np.empty(n, order="F") for _ in range(3))
    g.x[...], g.y[...], g.z[...] = xl[:, None, None], yl[None, :, None], zl[None, None, :]
    g.flag = np.zeros(n, dtype=np.int32, order="F") if flag is None else np.asfortranarray(flag)
    return g


def _flow_grid(flow, n):
    ni, nj, nk = n
    if flow == "gyre":  # node-centred [0,2] x [0,1] with slip walls
        flag = np.zeros(n, dtype=np.int32)
        flag[[0, -1], :, :] = L.LCS_SLIP
        flag[:, [0, -1], :] = L.LCS_SLIP
        return _grid(np.arange(ni) * (2.0 / (ni - 1)), np.arange(nj) * (1.0 / (nj - 1)), np.zeros(1), flag)
    if flow in ("abc", "turbulence"):  # cell-centred and periodic in every direction
        return _grid(*((np.arange(m) + 0.5) * (TWO_PI / m) for m in n))
    if flow == "duct":  # inflow and outflow in x, periodic in y, slip walls in z, a masked block
        flag = np.zeros(n, dtype=np.int32)
        flag[0], flag[-1] = L.LCS_INFLOW, L.LCS_OUTFLOW
        flag[:, :, [0, -1]] = L.LCS_SLIP
        flag[ni // 2:ni // 2 + 3, nj // 2:nj // 2 + 2, nk // 2:nk // 2 + 2] = L.LCS_MASK
        return _grid(np.arange(ni) * (1.0 / (ni - 1)), (np.arange(nj) + 0.5) / nj, np.arange(nk) * (0.9 / (nk - 1)), flag)
    flag = np.zeros(n, dtype=np.int32)  # channel: periodic in x and z, walls in y, points drawn towards them
    flag[:, [0, -1], :] = L.LCS_WALL
    y = 0.5 * (1.0 + np.tanh(1.6 * np.linspace(-1.0, 1.0, nj)) / math.tanh(1.6))
    return _grid((np.arange(ni) + 0.5) * (2.0 / ni), y, (np.arange(nk) + 0.5) * (1.0 / nk), flag)


# ------------------------------------------------------------------------------- velocities
def _modes(seed, count, kmax):
    """Divergence-free Fourier modes on [0, 2 pi)^3 with a k^-5/3 spectrum and unit rms."""
    rng = np.random.default_rng(seed)
    k = np.empty((0, 3))
    while len(k) < count:
        c = rng.integers(-kmax, kmax + 1, size=(4 * count, 3))
        m = np.linalg.norm(c, axis=1)
        k = np.concatenate([k, c[(m >= 1) & (m <= kmax)]])
    k = k[:count]
    km = np.linalg.norm(k, axis=1, keepdims=True)
    a = rng.normal(size=(count, 3))
    a -= (a * k).sum(1, keepdims=True) * k / km**2
    a *= km ** (-5.0 / 6.0) / np.linalg.norm(a, axis=1, keepdims=True)
    return k, a / math.sqrt(0.5 * (a * a).sum() / 3.0), rng.uniform(0.0, TWO_PI, count)


def _mode_field(g, seed, count, kmax):
    """Three components as (nk, nj, ni) tensors, from modes stretched to the grid's box."""
    k, a, phase = (torch.as_tensor(v, dtype=torch.float64, device=DEV) for v in _modes(seed, count, kmax))
    x, y, z = (torch.as_tensor(v, dtype=torch.float64, device=DEV) for v in g.lines)
    if g.box != (TWO_PI,) * 3:
        x, y, z = (v * (TWO_PI / b) for v, b in zip((x, y, z), g.box))
    plane = (k[:, 0, None, None] * x + k[:, 1, None, None] * y[:, None] + phase[:, None, None]).reshape(count, -1)
    up = k[:, 2, None] * z
    cp, sp, cz, sz = plane.cos(), plane.sin(), up.cos(), up.sin()
    n = (len(z), len(y), len(x))
    return [((cz * a[:, c, None]).T @ cp - (sz * a[:, c, None]).T @ sp).reshape(n) for c in range(3)]


def _levels(flow, g, seed, steps, dt):
    """Velocity of the levels 0 .. steps (level 0 and the last are the base flow), each three
    (nk, nj, ni) tensors."""
    X, Y, Z = (torch.as_tensor(v, dtype=torch.float64, device=DEV) for v in g.lines)
    X, Y, Z = X[None, None, :], Y[None, :, None], Z[:, None, None]
    n = (len(g.lines[2]), len(g.lines[1]), len(g.lines[0]))
    rng = np.random.default_rng(seed)
    s = [math.sin(math.pi * j / steps) ** 2 for j in range(steps)] + [0.0]
    if flow == "gyre":
        eps, A = rng.uniform(0.1, 0.3), 0.1
        out = []
        for j in range(steps + 1):
            e = eps * math.sin(TWO_PI * j / steps) if 0 < j < steps else 0.0
            f, df = e * X * X + (1.0 - 2.0 * e) * X, 2.0 * e * X + (1.0 - 2.0 * e)
            u = -math.pi * A * torch.sin(math.pi * f) * torch.cos(math.pi * Y)
            v = math.pi * A * torch.cos(math.pi * f) * torch.sin(math.pi * Y) * df
            out.append([t.expand(n).contiguous() for t in (u, v, torch.zeros_like(u))])
        return out
    if flow == "abc":
        A, B, C = math.sqrt(3.0), math.sqrt(2.0), 1.0
        base = [A * torch.sin(Z) + C * torch.cos(Y), B * torch.sin(X) + A * torch.cos(Z), C * torch.sin(Y) + B * torch.cos(X)]
        more, window = [0.2 * t for t in _mode_field(g, seed, 8, 3)], (1.0, 1.0, 1.0)
    elif flow == "turbulence":
        # wavenumbers up to 32, fewer on a grid that would not resolve them
        kmax = max(3, min(32, min(g.n) // 8))
        base = _mode_field(g, 20261203, 64, kmax)
        more, window = [0.3 * t for t in _mode_field(g, seed, 32, kmax)], (1.0, 1.0, 1.0)
    elif flow == "duct":
        wall = torch.sin(math.pi * Z / 0.9)
        base = [0.4 + 0.1 * wall, 0.08 * torch.sin(TWO_PI * X) + 0.05 * torch.cos(TWO_PI * Y), 0.05 * wall * torch.sin(TWO_PI * Y)]
        more, window = [0.03 * t for t in _mode_field(g, seed, 8, 3)], (1.0, 1.0, wall)
    else:
        wall = 4.0 * Y * (1.0 - Y)
        base = [0.6 * wall + 0.1 * torch.sin(TWO_PI * Z) * wall, 0.0125 * wall**2 * torch.cos(math.pi * X), 0.025 * wall * torch.cos(math.pi * X)]
        more, window = [0.05 * t for t in _mode_field(g, seed, 8, 3)], (wall, wall**2, wall)
    base = [t.expand(n) for t in base]
    return [[(b + s[j] * w * m).contiguous() for b, w, m in zip(base, window, more)] for j in range(steps + 1)]


# ------------------------------------------------------------------------------- the library
_HELD = {"key": None}  # the library instance in use: one per process, as the reference has


def _release():
    if _HELD["key"] is not None:
        _HELD["api"].reset()
        _HELD.clear()
        _HELD["key"] = None


def _lib(case):
    return "sp" if case["precision"] == "sp" else "dp"


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def _check(api):
    code, text = api.error()
    if code:
        raise RuntimeError(text)


class _DeviceArray:
    """A device buffer of the library for torch.as_tensor."""

    def __init__(self, ptr, count, double):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8" if double else "<f4", "data": (ptr, False), "version": 3}


def _hold_flow(case, g, first):
    """The library set up for the case's grid and options, at solver time 0 with the velocity
    level `first`."""
    if _HELD["key"] == _key(case):
        return
    _release()
    api = L.Cfd2lcs(_lib(case))
    api.reset()
    _HELD.update(key=_key(case), api=api, step=0)
    dt = 2.0 ** case["dt_log2"]
    if case["precision"] == "mixed":
        api.set_option("MIXED_PRECISION", L.LCS_TRUE)
    api.init(g.n, g.x, g.y, g.z, g.flag)
    h = dt * case["per_h"]
    _HELD["handles"] = [api.diagnostic_init(d, 0, h * case["slots"], h) for d in DIRECTIONS[case["direction"]]]
    api.set_option("INTEGRATOR", INTEGRATORS[case["integrator"]])
    api.set_option("INTERPOLATOR", INTERPOLATORS[case["interpolator"]])
    api.set_param("CFL", CFL)
    (api.update if case["host"] else api.update_device)(*first, 0.0)
    _check(api)


def _feed(case, g, level):
    """One velocity level as update() takes it: host arrays, or device pointers of the tensors
    returned beside them."""
    kind = torch.float32 if _lib(case) == "sp" else torch.float64
    flat = [t.reshape(-1).to(kind) for t in level]
    if case["host"]:
        return [t.cpu().numpy().reshape(g.n, order="F") for t in flat], None
    return [t.data_ptr() for t in flat], flat


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    if case["kind"] == "gradient":
        return _prepare_gradient(case, seed)
    n, steps = (case["ni"], case["nj"], case["nk"]), case["per_h"] * case["slots"]
    held = _HELD["key"] == _key(case)
    g = _HELD["grid"] if held else _flow_grid(case["flow"], n)
    g.box = (2.0, 1.0, 1.0) if case["flow"] == "channel" else (1.0, 1.0, 0.9) if case["flow"] == "duct" else (TWO_PI,) * 3
    levels = [_feed(case, g, v) for v in _levels(case["flow"], g, seed, steps, 2.0 ** case["dt_log2"])]
    torch.cuda.synchronize()
    _hold_flow(case, g, levels[0][0])
    _HELD["grid"] = g
    return {"case": case, "grid": g, "levels": levels}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        return _run_batch(state)
    if case["kind"] == "gradient":
        return _run_gradient(state)
    _hold_flow(case, state["grid"], state["levels"][0][0])
    api, dt = _HELD["api"], 2.0 ** case["dt_log2"]
    update = api.update if case["host"] else api.update_device
    for fields, _ in state["levels"][1:]:
        _HELD["step"] += 1
        update(*fields, _HELD["step"] * dt)
    _check(api)
    out = {}
    for d, h in zip(DIRECTIONS[case["direction"]], _HELD["handles"]):
        name = "forward" if d == L.FTLE_FWD else "backward"
        if case["host"]:
            out[name + " ftle"], out[name + " map"] = api.ftle(h), api.flowmap(h)
        else:  # the library's own buffer, as a program that goes on working on the GPU reads it
            count = case["ni"] * case["nj"] * case["nk"]
            out[name + " ftle"] = torch.as_tensor(_DeviceArray(api.ftle_device_ptr(h), count, _lib(case) == "dp"), device=DEV)
    return out


# ------------------------------------------------------------------------------- many instances
def _batch_specs(case):
    """Sizes, directions and time steps of the instances: gyres from 64 x 32, cubes from 32^3."""
    rng, specs = np.random.default_rng(case["mix"]), []
    for _ in range(case["gyres"]):
        ni = int(round(2.0 ** rng.uniform(6.0, 9.0)))
        specs.append(("gyre", (ni, ni // 2, 1), int(rng.integers(0, 2))))
    for _ in range(case["cubes"]):
        n = int(round(32.0 * (case["largest"] / 32.0) ** rng.uniform()))
        specs.append(("abc", (n, n, n), int(rng.integers(0, 2))))
    return [(f, n, d, _dt_log2(RATE[f] * max(n), 3.0 + 2.0 * rng.uniform())) for f, n, d in specs]


def _hold_batch(state):
    case = state["case"]
    if _HELD["key"] == _key(case):
        return
    _release()
    api = L.Batch(_lib(case))
    api.reset()
    _HELD.update(key=_key(case), api=api, step=0)
    ids, handles = [], []
    for (_, n, d, e), g in zip(state["specs"], state["grids"]):
        ids.append(api.add(g.n, g.x, g.y, g.z, g.flag, L.RK2, INTERPOLATORS[case["interpolator"]], CFL, case["precision"] == "mixed"))
        handles.append(api.diagnostic_init(ids[-1], d, 2.0**e * case["updates"], 2.0**e * case["updates"] / 2))
    _check(api)
    _HELD.update(ids=ids, handles=handles)
    api.update_device(ids, *state["levels"][0][0], [0.0] * len(ids))
    _check(api)


def _prepare_batch(case, seed):
    specs, steps = _batch_specs(case), case["updates"]
    grids = [_flow_grid(f, n) for f, n, _, _ in specs]
    per, kind = [], torch.float32 if _lib(case) == "sp" else torch.float64
    for q, ((f, _, _, e), g) in enumerate(zip(specs, grids)):
        g.box = (TWO_PI,) * 3
        per.append([[t.reshape(-1).to(kind) for t in v] for v in _levels(f, g, seed * 1000 + q, steps, 2.0**e)])
    levels = []
    for j in range(steps + 1):
        levels.append(([[p[j][c].data_ptr() for p in per] for c in range(3)], [p[j] for p in per]))
    torch.cuda.synchronize()
    state = {"case": case, "specs": specs, "grids": grids, "levels": levels}
    _hold_batch(state)
    return state


def _run_batch(state):
    _hold_batch(state)
    api, ids = _HELD["api"], _HELD["ids"]
    for fields, _ in state["levels"][1:]:
        _HELD["step"] += 1
        api.update_device(ids, *fields, [_HELD["step"] * 2.0**e for _, _, _, e in state["specs"]])
    _check(api)
    return {"ftle": [api.ftle(i, h) for i, h in zip(ids, _HELD["handles"])]}


# ------------------------------------------------------------------------------- gradients
def _prepare_gradient(case, seed):
    _release()
    g = _flow_grid("abc", (case["n"],) * 3)
    g.box = (TWO_PI,) * 3
    kind = torch.float32 if _lib(case) == "sp" else torch.float64
    levels = [[t.reshape(-1).to(kind) for t in v] for v in _levels("abc", g, seed, case["levels"] - 1, 2.0 ** case["dt_log2"])]
    # noise on every level, as measured or modelled velocities carry it
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    levels = [[t + 0.01 * torch.randn(t.shape, generator=gen, device=DEV, dtype=t.dtype) for t in v] for v in levels]
    axes = [torch.as_tensor((a > 0.25 * TWO_PI) & (a < 0.75 * TWO_PI), device=DEV) for a in g.lines]
    box = (axes[2][:, None, None] & axes[1][None, :, None] & axes[0][None, None, :]).reshape(-1)
    weight = (box.to(torch.float64) / box.sum()).to(kind)  # J is the mean FTLE over the middle of the box
    torch.cuda.synchronize()
    return {"case": case, "grid": g, "levels": [[v[c] for v in levels] for c in range(3)], "weight": weight,
            "times": [j * 2.0 ** case["dt_log2"] for j in range(case["levels"])]}


def _run_gradient(state):
    case = state["case"]
    J, gu, gv, gw = L.adjoint_ftle(state["grid"], *state["levels"], state["times"], state["weight"],
                                   integrator=INTEGRATORS[case["integrator"]], cfl=CFL, checkpoint_every=case["checkpoint"],
                                   precision=_lib(case), interpolator=INTERPOLATORS[case["interpolator"]])
    return {"J": J, "u": gu, "v": gv, "w": gw}


# ------------------------------------------------------------------------------- least work
def _sample_flops(interp):
    """Multiplications and additions of one three-component sample."""
    return 3 * 2 * 8 + 20 if interp == "linear" else 3 * 2 * (64 + 16 + 4) + 60


def _flow_work(flow, n, dt_log2, updates, frames, slots, stages, interp, ways, size):
    """Least bytes and operations: every velocity level read once, the flow map or the particles
    read and written and the two velocity levels read in each subcycle, each frame's sub-maps
    read and its field written."""
    points = n[0] * n[1] * n[2]
    subcycles = updates * max(1, math.ceil(RATE[flow] * max(n) * 2.0**dt_log2 / CFL))
    per_point = size * (6 + 6) * subcycles + size * (3 * slots + 4) * frames
    flops = subcycles * (stages * _sample_flops(interp) + 6 * stages) + frames * slots * _sample_flops(interp)
    return points * (3 * size * updates + ways * per_point), points * ways * flops


def work(case):
    size = 4 if case["precision"] == "sp" else 8
    if case["kind"] == "batch":
        each = [_flow_work(f, n, e, case["updates"], 2, 2, 2, case["interpolator"], 1, size) for f, n, _, e in _batch_specs(case)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    if case["kind"] == "gradient":
        # the forward sweep, once more for the recomputed segments, and the reverse one, which
        # reads and writes the adjoints beside the fields
        b, f = _flow_work("abc", (case["n"],) * 3, case["dt_log2"], case["levels"] - 1, 1, 0, STAGES[case["integrator"]],
                          case["interpolator"], 1, size)
        return {"bytes": 4 * b, "flops": 5 * f}
    b, f = _flow_work(case["flow"], (case["ni"], case["nj"], case["nk"]), case["dt_log2"], case["per_h"] * case["slots"], case["slots"],
                      case["slots"], STAGES[case["integrator"]], case["interpolator"], len(DIRECTIONS[case["direction"]]), size)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------- in 64 bits
class _Box:
    """A periodic box in 64 bits: the case's coordinate lines as the library gets them, padded by
    a node on either side, and samples of periodic fields (3, nk, nj, ni) at points (3 tensors)."""

    def __init__(self, g, single, interp):
        self.n, self.interp = g.n, interp
        self.lines = []
        for a in g.lines:
            a = torch.as_tensor(np.asarray(a, dtype=np.float32 if single else np.float64), device=DEV).double()
            self.lines.append(torch.cat([(2 * a[0] - a[1])[None], a, (2 * a[-1] - a[-2])[None]]))
        self.period = [a[-1] - a[1] for a in self.lines]
        z, y, x = torch.meshgrid(self.lines[2][1:-1], self.lines[1][1:-1], self.lines[0][1:-1], indexing="ij")
        self.nodes = [x.reshape(-1), y.reshape(-1), z.reshape(-1)]
        if interp == "cubic":
            self.knots, self.inverse = zip(*(self._fit(a) for a in self.lines))

    @staticmethod
    def _basis(t, l, x):
        """The four cubic B-splines that are not zero at x in [t(l), t(l+1))."""
        b = [torch.ones_like(x)]
        for j in range(1, 4):
            new, carry = [], 0.0
            for m in range(j):
                right, left = t[l + m + 1], t[l + m + 1 - j]
                v = b[m] / (right - left)
                new.append(carry + v * (right - x))
                carry = v * (x - left)
            b = new + [carry]
        return b

    def _fit(self, a):
        """Not-a-knot knots (the right end moved out by a tenth of a cell) and the inverse of the
        collocation matrix at the nodes."""
        m = len(a)
        t = torch.cat([a[:1].repeat(4), a[2:-2], (a[-1] + 0.1 * (a[-1] - a[-2])).repeat(4)])
        l = (torch.searchsorted(t, a, right=True) - 1).clamp(3, m - 1)
        A = torch.zeros(m, m, dtype=torch.float64, device=DEV)
        for j, v in enumerate(self._basis(t, l, a)):
            A[torch.arange(m, device=DEV), l - 3 + j] = v
        return t, torch.linalg.inv(A)

    def coefficients(self, f):
        """What sample() takes for a field (3, N): itself, or its spline coefficients on the
        padded box."""
        if self.interp == "linear":
            return f
        ni, nj, nk = self.n
        f = torch.nn.functional.pad(f.reshape(3, nk, nj, ni), (1,) * 6, mode="circular")
        for axis, inv in ((3, self.inverse[0]), (2, self.inverse[1]), (1, self.inverse[2])):
            f = torch.movedim(torch.movedim(f, axis, 3) @ inv.T, 3, axis)
        return f.reshape(3, -1)

    def sample(self, c, x):
        out, taps = 0.0, []
        for a in range(3):
            if self.interp == "linear":
                i = (torch.searchsorted(self.lines[a], x[a].detach(), right=True) - 1).clamp(0, self.n[a])
                t = (x[a] - self.lines[a][i]) / (self.lines[a][i + 1] - self.lines[a][i])
                taps.append([((i - 1) % self.n[a], 1.0 - t), (i % self.n[a], t)])
            else:
                l = (torch.searchsorted(self.knots[a], x[a], right=True) - 1).clamp(3, self.n[a] + 1)
                taps.append([(l - 3 + j, v) for j, v in enumerate(self._basis(self.knots[a], l, x[a]))])
        pad = 0 if self.interp == "linear" else 2
        sx, sxy = self.n[0] + pad, (self.n[0] + pad) * (self.n[1] + pad)
        for k, wk in taps[2]:
            for j, wj in taps[1]:
                for i, wi in taps[0]:
                    out = out + wk * wj * wi * c[:, i + sx * j + sxy * k]
        return out

    def wrap(self, x):
        """Points back to the image whose nearest node is inside the box."""
        out = []
        for a in range(3):
            p, L_ = self.lines[a], self.period[a]
            lo, hi = 0.5 * (p[0] + p[1]), 0.5 * (p[-2] + p[-1])
            out.append(torch.where(x[a] < lo, x[a] + L_, torch.where(x[a] >= hi, x[a] - L_, x[a])))
        return out

    def subcycles(self, u, dt):
        rate = sum(u[a].abs() / (self.lines[a][2] - self.lines[a][1]) for a in range(3)).max()
        return max(1, math.ceil(float(rate) * dt / CFL))

    def step(self, integrator, velocity, x, t, dt):
        """One Runge-Kutta step (the reference's third-order form has its last stage at x + 2 k2)."""
        u = lambda y, s: dt * velocity(y, s)  # noqa: E731
        k1 = u(x, t)
        k2 = u([a + 0.5 * b for a, b in zip(x, k1)], t + 0.5 * dt)
        if integrator == "rk2":
            return [a + b for a, b in zip(x, k2)]
        if integrator == "rk3":
            k3 = u([a + 2.0 * b for a, b in zip(x, k2)], t + dt)
            return [a + b / 6 + 2 * c / 3 + d / 6 for a, b, c, d in zip(x, k1, k2, k3)]
        k3 = u([a + 0.5 * b for a, b in zip(x, k2)], t + 0.5 * dt)
        k4 = u([a + b for a, b in zip(x, k3)], t + dt)
        return [a + (b + 2 * c + 2 * d + e) / 6 for a, b, c, d, e in zip(x, k1, k2, k3, k4)]

    def maps(self, integrator, levels, dt, forward):
        """Displacement over the levels' span of the nodes, and of one direction's subcycles."""
        d, x = torch.zeros_like(levels[0]), list(self.nodes)
        coef = [self.coefficients(u) for u in levels]
        for j in range(1, len(levels)):
            m = self.subcycles(levels[j].detach(), dt)
            old, new = coef[j - 1], coef[j]
            vel = lambda y, s: self.sample((1 - s) * old + s * new, y)  # noqa: E731
            for q in range(m):
                if forward:
                    y = self.step(integrator, lambda p, s: vel(p, s / dt), x, q * dt / m, dt / m)
                    d = d + torch.stack([a - b for a, b in zip(y, x)])
                    x = self.wrap(y)
                else:
                    y = self.step(integrator, lambda p, s: vel(p, s / dt), self.nodes, dt - q * dt / m, -dt / m)
                    d = self.sample(self.coefficients(d), y) + torch.stack([a - b for a, b in zip(y, self.nodes)])
        return d

    def compose(self, maps):
        x, d = list(self.nodes), 0.0
        for m in maps:
            up = self.sample(self.coefficients(m), x)
            d, x = d + up, self.wrap([a + b for a, b in zip(x, up)])
        return d

    def ftle(self, d, T):
        d = d.reshape(3, self.n[2], self.n[1], self.n[0])
        G = []
        for a, axis in ((0, 3), (1, 2), (2, 1)):
            p = self.lines[a]
            shape = [1, 1, 1, 1]
            shape[axis] = -1
            G.append((torch.roll(d, -1, axis) - torch.roll(d, 1, axis)) / (p[2:] - p[:-2]).reshape(shape))
        C = [[(G[a] * G[b]).sum(0) for b in range(3)] for a in range(3)]
        # largest eigenvalue of a symmetric matrix by the trigonometric solution of its cubic
        m = (C[0][0] + C[1][1] + C[2][2]) / 3
        D = [C[a][a] - m for a in range(3)]
        off = C[0][1] ** 2 + C[0][2] ** 2 + C[1][2] ** 2
        p = torch.sqrt((D[0] ** 2 + D[1] ** 2 + D[2] ** 2 + 2 * off) / 6)
        det = (D[0] * (D[1] * D[2] - C[1][2] ** 2) - C[0][1] * (C[0][1] * D[2] - C[1][2] * C[0][2])
               + C[0][2] * (C[0][1] * C[1][2] - D[1] * C[0][2]))
        r = (det / (2 * p**3)).clamp(-1 + 1e-14, 1 - 1e-14)
        lam = m + 2 * p * torch.cos(torch.acos(r) / 3)
        return (0.5 * torch.log(lam) / T).reshape(-1)


def exact(case, seed):
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed) if case["interpolator"] == "linear" else None
    # walls, masks and planes go by the reference's rules node by node: no plain form of them here
    if case["kind"] == "batch" or case["flow"] not in ("abc", "turbulence"):
        return None
    n, steps, dt = (case["ni"], case["nj"], case["nk"]), case["per_h"] * case["slots"], 2.0 ** case["dt_log2"]
    ways = DIRECTIONS[case["direction"]]
    # the cubic's 64 taps per sample take over 20 seconds on the large grids
    cost = _flow_work(case["flow"], n, case["dt_log2"], steps, 1, case["slots"], STAGES[case["integrator"]], case["interpolator"],
                      len(ways), 8)[1]
    if case["interpolator"] == "cubic" and cost > 5e11:
        return None
    with torch.no_grad():
        g = _flow_grid(case["flow"], n)
        g.box = (TWO_PI,) * 3
        box = _Box(g, case["precision"] == "sp", case["interpolator"])
        levels = []
        for v in _levels(case["flow"], g, seed, steps, dt):
            v = torch.stack([t.reshape(-1) for t in v])
            levels.append(v.float().double() if case["precision"] == "sp" else v)
        out = {}
        for d in ways:
            fwd = d == L.FTLE_FWD
            parts = [box.maps(case["integrator"], levels[q * case["per_h"]:(q + 1) * case["per_h"] + 1], dt, fwd) for q in range(case["slots"])]
            out[("forward" if fwd else "backward") + " ftle"] = box.ftle(box.compose(parts if fwd else parts[::-1]), steps * dt)
        return out


def _exact_gradient(case, seed):
    state = _prepare_gradient(case, seed)
    box = _Box(state["grid"], case["precision"] == "sp", "linear")
    u = [torch.stack([state["levels"][c][j].double() for c in range(3)]).requires_grad_() for j in range(case["levels"])]
    dt = 2.0 ** case["dt_log2"]
    field = box.ftle(box.maps(case["integrator"], u, dt, False), (case["levels"] - 1) * dt)
    J = (state["weight"].double() * field).sum()
    J.backward()
    # the first level is never interpolated with a weight of its own where a pass has one level only
    grads = [v.grad if v.grad is not None else torch.zeros_like(v) for v in u]
    return {"J": float(J.detach()), "u": [v[0] for v in grads], "v": [v[1] for v in grads], "w": [v[2] for v in grads]}
