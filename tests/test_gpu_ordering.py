"""Calls that take device arrays start after the work their caller has queued: levels, weight and
direction computed behind tens of milliseconds of queued work, and gradient buffers that reuse a
freed temporary that queued work still writes, give what the synchronised call gives -- on the default
stream and on another current stream."""
import numpy as np
import pytest

from tests import workloads as W

pytestmark = pytest.mark.gpu

SPIN = 60_000_000  # cycles of queued work: 30 ms at 2 GHz, many times the host side of a call
N, LEVELS, DT = 12, 5, 0.05


def _streams():
    import torch
    return {"default": torch.cuda.default_stream(), "side": torch.cuda.Stream()}


def _problem():
    import torch
    g = W.abc_grid(N)
    rng = np.random.default_rng(3)
    base = W.abc_velocity(g)
    lev = [[torch.from_numpy((base[c] + 0.05 * rng.standard_normal(g.n)).ravel(order="F")).cuda() for _ in range(LEVELS)] for c in range(3)]
    weight = torch.from_numpy(rng.random(g.npts)).cuda()
    return g, lev, [k * DT for k in range(LEVELS)], weight


def _late(tensors):
    """Copies that hold other values until the queued work reaches them."""
    import torch
    late = [-2.0 * t for t in tensors]
    torch.cuda.synchronize()
    torch.cuda._sleep(SPIN)
    for a, t in zip(late, tensors):
        a.copy_(t)
    return late


def _late_levels(lev, more):
    flat = _late([t for comp in lev for t in comp] + [more])
    return [flat[c * LEVELS:(c + 1) * LEVELS] for c in range(3)], flat[-1]


@pytest.mark.parametrize("stream", ["default", "side"])
@pytest.mark.parametrize("interp", [1, 3])
def test_adjoint_waits_for_its_inputs_and_buffers(stream, interp):
    import torch

    import libcfd2lcs_b200 as L
    g, lev, times, weight = _problem()
    torch.cuda.synchronize()
    J, *ref = L.adjoint_ftle(g, *lev, times, weight, interpolator=interp)
    with torch.cuda.stream(_streams()[stream]):
        late, late_w = _late_levels(lev, weight)
        # freed while queued work still writes them: the gradients are given the same blocks
        junk = [torch.empty_like(weight) for _ in range(3 * LEVELS)]
        for t in junk:
            t.fill_(float("nan"))
        del junk, t
        Jl, *out = L.adjoint_ftle(g, *late, times, late_w, interpolator=interp)
        assert Jl == J
        for a, b in zip(ref, out):
            for x, y in zip(a, b):
                # (the scatters' atomics add in any order)
                assert float((x - y).abs().max()) <= 1e-12 * float(x.abs().max())


@pytest.mark.parametrize("stream", ["default", "side"])
def test_tangent_waits_for_its_inputs(stream):
    import torch

    import libcfd2lcs_b200 as L
    g, lev, times, weight = _problem()
    d = [[torch.sin(7.0 * t) for t in comp] for comp in lev]
    torch.cuda.synchronize()
    ref = L.tangent_ftle(g, *lev, times, weight, *d)
    with torch.cuda.stream(_streams()[stream]):
        late, late_w = _late_levels(lev, weight)
        late_d, _ = _late_levels(d, weight)
        assert L.tangent_ftle(g, *late, times, weight, *late_d) == ref
        late, late_w = _late_levels(lev, weight)
        assert L.tangent_ftle(g, *late, times, late_w, *d) == ref


@pytest.mark.parametrize("stream", ["default", "side"])
def test_update_device_waits_for_its_level(stream):
    import torch

    import libcfd2lcs_b200 as L
    g, lev, times, weight = _problem()

    def frame(late):
        api = L.Cfd2lcs("dp")
        api.reset()
        api.init(g.n, g.x, g.y, g.z, g.flag)
        h = [api.diagnostic_init(d, 0, times[-1], times[-1], "d") for d in (0, 1)]
        for k in range(LEVELS):
            u = [lev[c][k] for c in range(3)]
            u = _late(u) if late else u
            api.update_device(*(t.data_ptr() for t in u), times[k])
        assert api.error()[0] == 0, api.error()
        out = [api.flowmap(q) for q in h]
        api.reset()
        return out

    torch.cuda.synchronize()
    ref = frame(False)
    with torch.cuda.stream(_streams()[stream]):
        for a, b in zip(ref, frame(True)):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("stream", ["default", "side"])
def test_batch_update_waits_for_its_levels(stream):
    import torch

    import libcfd2lcs_b200 as L
    g, lev, times, weight = _problem()

    def frame(late):
        api = L.Batch("dp")
        api.reset()
        ids = [api.add(g.n, g.x, g.y, g.z, g.flag) for _ in range(2)]
        h = [api.diagnostic_init(i, 1, times[-1], times[-1]) for i in ids]
        for k in range(LEVELS):
            u = [lev[c][k] for c in range(3)]
            u = _late(u) if late else u
            api.update_device(ids, *([t.data_ptr()] * 2 for t in u), [times[k]] * 2)
        assert api.error()[0] == 0, api.error()
        out = [api.flowmap(i, q) for i, q in zip(ids, h)]
        api.reset()
        return out

    torch.cuda.synchronize()
    ref = frame(False)
    with torch.cuda.stream(_streams()[stream]):
        for a, b in zip(ref, frame(True)):
            assert np.array_equal(a, b)
