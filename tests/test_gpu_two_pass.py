"""The two-pass schedule above the size at which batches run on teams alone: parked
after a tenth of the span or 512 step attempts, resumed by the mixed kernel with the
number of team SMs fixed, chosen on the device, or none, against one pass with one
thread per orbit. The same operations in the same order throughout, so the same bits."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 12000  # above 64 orbits per SM


def _set_team(blocks):
    from galax_gb300 import _lib

    _lib.check(_lib.load().gal_set_team(int(blocks)), "gal_set_team")


def _cfg(method, schedule, case):
    import galax_gb300 as gx

    solver = gx.Dopri8() if method == 8 else gx.Dopri5()
    if case == "constant":
        return gx.Integrator(solver=solver, stepsize_controller=gx.ConstantStepSize(), dt0=2.0, schedule=schedule).config()
    return gx.Integrator(solver=solver, stepsize_controller=gx.PIDController(rtol=1e-8, atol=1e-10),
                         max_steps=150 if case == "max_steps" else 2**16, schedule=schedule).config()


def _batch(case):
    from galax_gb300 import workloads as W

    tmax = {"long": 1500.0, "max_steps": 500.0}.get(case, 250.0)
    b = W.uneven_ics(lambda x: O.gradient(O.milky_way(), x), N, seed=8, tmax=tmax, smax=20)
    if case == "long":  # close in: thousands of attempts in the first tenth of the span
        b.y0[:64, :3] *= 0.02 / np.linalg.norm(b.y0[:64, :3], axis=1, keepdims=True)
        b.y0[:64, 3:] *= 0.3
    return b


@pytest.mark.parametrize("method", [5, 8])
@pytest.mark.parametrize("case", ["csr", "backward", "constant", "max_steps", "long", "host_saves"])
def test_matches_one_pass_on_single_threads(method, case):
    import torch

    import galax_gb300 as gx
    from galax_gb300.dynamics import Workspace, integrate

    mw, b = gx.MilkyWayPotential(), _batch(case)

    def run(schedule, team):
        _set_team(team)
        kw = {}
        if case == "backward":
            args = (0.0, -200.0, np.linspace(0.0, -200.0, 9))
        else:
            args, kw = (b.t0, b.t1, b.save_ts), {"save_offsets": b.save_offsets}
            if case == "host_saves":  # Dopri8's saves inside the integration, across park and resume
                kw["out"] = torch.empty((6, len(b.save_ts)), dtype=torch.float64).pin_memory()
        res = integrate(mw, b.y0, *args, _cfg(method, schedule, case), workspace=Workspace(), **kw)
        torch.cuda.synchronize()
        return [v.cpu().numpy().copy() for v in res]

    alone = run(False, 0)
    for schedule, team in ((True, -1), (True, 0), (True, 8), (True, 1000)):
        for a, w in zip(run(schedule, team), alone):
            np.testing.assert_array_equal(a, w)
    assert (alone[1] == 0).any()
    if case == "max_steps":
        assert (alone[1] == 1).any()
    if case == "long":
        assert alone[2].max() > 5120  # some orbit takes more than 512 attempts in a tenth of its span


@pytest.mark.parametrize("method", [5, 8])
def test_replays_from_a_cuda_graph(method):
    """Two passes with the team count chosen on the device: on other orbits, the
    replay chooses anew."""
    import torch

    import galax_gb300 as gx
    from galax_gb300.dynamics import Workspace, integrate

    mw, b = gx.MilkyWayPotential(), _batch("csr")
    y0 = torch.as_tensor(b.y0, device="cuda").t().contiguous()
    t0 = torch.zeros(N, dtype=torch.float64, device="cuda")
    t1 = torch.as_tensor(b.t1 - b.t0, device="cuda").contiguous()
    ts = torch.linspace(0.0, 50.0, 5, dtype=torch.float64, device="cuda")
    cfg, ws = _cfg(method, True, "csr"), Workspace()

    def run():
        return integrate(mw, y0, t0, t1, ts, cfg, soa=True, workspace=ws)

    eager = [v.clone() for v in run()]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = run()
    g.replay()
    torch.cuda.synchronize()
    for a, w in zip(out, eager):
        assert torch.equal(torch.nan_to_num(a.double(), nan=-7.0), torch.nan_to_num(w.double(), nan=-7.0))
    y0.copy_(y0.roll(1777, dims=1) * 0.97)
    t1.copy_(t1.roll(311))
    g.replay()
    torch.cuda.synchronize()
    for a, w in zip(out, run()):
        assert torch.equal(torch.nan_to_num(a.double(), nan=-7.0), torch.nan_to_num(w.double(), nan=-7.0))


def test_automatic_teams_can_be_set_again():
    from galax_gb300 import _lib, autotune

    L = _lib.load()
    _set_team(8)
    autotune.set_automatic_teams()
    assert L.gal_set_team(-2) != 0 and L.gal_set_team(1025) != 0


@pytest.mark.parametrize("method", [5, 8])
def test_without_a_workspace(method):
    """gal_integrate_noalloc with two passes, call after call on other orbits and
    replayed from a graph: its array is reused by every call."""
    import ctypes as C

    import torch

    import galax_gb300 as gx
    from galax_gb300 import _lib
    from galax_gb300.dynamics import Workspace, integrate

    mw, L, cfg = gx.MilkyWayPotential(), _lib.load(), _cfg(method, True, "csr")
    b = _batch("csr")
    y0 = torch.as_tensor(b.y0, device="cuda").t().contiguous()
    t0, t1 = torch.as_tensor(b.t0, device="cuda"), torch.as_tensor(b.t1, device="cuda").contiguous()
    ts = torch.linspace(0.0, 50.0, 5, dtype=torch.float64, device="cuda")
    out = torch.empty((6, 5, N), dtype=torch.float64, device="cuda")
    status = torch.empty(N, dtype=torch.int32, device="cuda")
    steps = torch.empty(N, dtype=torch.int64, device="cuda")

    def call():
        _lib.check(L.gal_integrate_noalloc(
            mw.handle(), C.byref(cfg), y0.data_ptr(), t0.data_ptr(), t1.data_ptr(), None, ts.data_ptr(), 5,
            out.data_ptr(), status.data_ptr(), steps.data_ptr(), None, N, torch.cuda.current_stream().cuda_stream),
            "gal_integrate_noalloc")

    def check():
        torch.cuda.synchronize()
        want = integrate(mw, y0, t0, t1, ts, cfg, soa=True, workspace=Workspace())
        for a, w in zip((out, status, steps), want):
            assert torch.equal(a, w)

    for k in range(2):
        y0.copy_(y0.roll(1777 * k, dims=1))
        call()
        check()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    for k in range(2):
        y0.copy_(y0.roll(311, dims=1) * (1.0 - 0.01 * k))
        g.replay()
        check()
