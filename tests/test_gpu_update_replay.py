"""Calls captured in a CUDA graph see the parameters of the last
gal_potential_update where they read them from the handle's component table."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _changed(pot, rng, move):
    arr = pot.component_array().copy()
    arr["m"] *= rng.uniform(0.5, 2.0, len(arr))
    arr["l1"] *= rng.uniform(0.5, 2.0, len(arr))
    arr["origin"] += move * rng.normal(size=(len(arr), 3)) * np.any(arr["origin"] != 0.0, axis=1, keepdims=True)
    return arr


def _update(pot, arr):
    import torch

    from galax_gb300 import _lib

    torch.cuda.synchronize()
    a = np.ascontiguousarray(arr)
    _lib.check(_lib.load().gal_potential_update(pot.handle(), a.ctypes.data, len(a), None), "gal_potential_update")


@pytest.mark.parametrize("method", [5, 8])
@pytest.mark.parametrize("others", ["mw", "mw_moved", "table"])
def test_orbits_among_many_spheres(method, others):
    """Constant steps with the spheres in fixed point: centres (into another binade
    and out of range), scales, masses and the other components, all at once."""
    import torch

    import galax_gb300 as gx
    from galax_gb300.dynamics import Workspace, integrate
    from galax_gb300.potential import from_component_array

    rng = np.random.default_rng(2)
    spheres = [gx.PlummerPotential(m_tot=1e8, r_s=0.5, origin=tuple(c)) for c in rng.normal(size=(40, 3)) * 20.0]
    rest = gx.IsochronePotential(m_tot=4e11, r_s=8.0) if others == "table" else gx.MilkyWayPotential()
    pot = gx.CompositePotential(spheres[:7] + [rest] + spheres[7:])
    n = 70
    x = rng.normal(size=(3, n)) * 8.0
    y0 = torch.as_tensor(np.concatenate([x, rng.normal(size=(3, n)) * 0.1]), device="cuda")
    t0 = torch.zeros(n, dtype=torch.float64, device="cuda")
    t1 = torch.full((n,), 12.0, dtype=torch.float64, device="cuda")
    ts = torch.linspace(0.0, 12.0, 4, dtype=torch.float64, device="cuda")
    cfg = gx.Integrator(solver=gx.Dopri8() if method == 8 else gx.Dopri5(),
                        stepsize_controller=gx.ConstantStepSize(), dt0=1.0).config()
    ws = Workspace()

    def run(p):
        return integrate(p, y0, t0, t1, ts, cfg, soa=True, workspace=ws)[0]

    first = run(pot).clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = run(pot)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, first)
    for move in (0.0, 5.0, 400.0):
        arr = _changed(pot, rng, move)
        if move == 400.0:
            arr["m"][0] = 1e76  # beyond the fixed point's range: this sphere goes to FP64
            arr["origin"][0] = 1e70
        if others == "mw_moved" and move:
            arr["origin"][7:11] = [0.3, -0.1, 0.2]
        _update(pot, arr)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, run(from_component_array(arr, G=pot.G)))
        assert not torch.equal(out, first)


@pytest.mark.parametrize("what", ["potential", "hessian"])
@pytest.mark.parametrize("moved", [False, True])
def test_milky_way_evaluation(what, moved):
    import torch

    import galax_gb300 as gx
    from galax_gb300.potential import from_component_array

    rng = np.random.default_rng(4)
    pot = gx.MilkyWayPotential()
    x = torch.as_tensor(rng.normal(size=(1000, 3)) * 9.0, device="cuda")
    first = getattr(pot, what)(x).clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = getattr(pot, what)(x)
    arr = _changed(pot, rng, 0.0)
    if moved:
        arr["origin"][1] = [0.5, 0.0, -0.25]
    _update(pot, arr)
    g.replay()
    torch.cuda.synchronize()
    want = getattr(from_component_array(arr, G=pot.G), what)(x)
    if moved:  # the general code, compiled into another kernel: a few dozen roundings of 2^-53 at most
        assert torch.all((out - want).abs() <= 1e-13 * want.reshape(1000, -1).norm(dim=1).reshape(-1, *[1] * (out.dim() - 1)))
    else:
        assert torch.equal(out, want)
    assert not torch.equal(out, first)
