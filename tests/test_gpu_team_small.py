"""Small batches on four-warp teams (two stages per round) against one thread
per orbit: the same operations in the same order, so the same bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [5, 8])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 2433, 9728])
@pytest.mark.parametrize("case", ["adaptive", "constant", "pid_dtmin", "host_saves", "order", "mw2022", "bovy", "linear",
                                  "sixteen"])
def test_small_batches_match_one_thread_per_orbit(method, n, case):
    import torch

    import galax_gb300 as gx
    from galax_gb300 import _lib
    from galax_gb300 import dynamics as D

    if n > 100 and case not in ("adaptive", "constant", "mw2022"):
        pytest.skip("the sizes that matter to these are the small ones")
    L = _lib.load()
    if case == "mw2022":
        mw = gx.MilkyWayPotential2022()
    elif case == "bovy":  # a disk, an incomplete gamma function, a halo
        mw = gx.BovyMWPotential2014()
    elif case == "linear":
        mw = gx.MilkyWayPotential(halo={"m": gx.LinearParameter(slope=6e8, point_time=10.0, point_value=5.4e11)})
    elif case == "sixteen":  # the largest table that teams take, components off the centre
        mw = gx.CompositePotential([gx.MilkyWayPotential()] + [
            gx.PlummerPotential(m_tot=1e9 * (k + 1), r_s=0.5, origin=(k, -k, 0.5 * k)) if k % 2 else
            gx.IsochronePotential(m_tot=1e9, r_s=1.0 + k, origin=(0.0, k, 1.0)) for k in range(12)])
    else:
        mw = gx.MilkyWayPotential()
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3)) * 6.0
    y0 = np.concatenate([x, rng.normal(size=(n, 3)) * 0.12], axis=1)
    t0 = np.zeros(n)
    t1 = rng.uniform(50.0, 250.0, n)
    if n > 3:
        t1[1] = 0.0       # nothing to integrate
        t1[2] = -80.0     # backwards
        y0[3, 1] = np.nan  # ends as non-finite
    lens = rng.integers(1, 6, n)
    offs = np.zeros(n + 1, np.int64)
    offs[1:] = np.cumsum(lens)
    ts = np.concatenate([np.linspace(t0[i], t1[i], lens[i]) if lens[i] > 1 else [t1[i]] for i in range(n)])
    solver = gx.Dopri8() if method == 8 else gx.Dopri5()
    dt0 = None
    if case == "constant":
        ctrl, dt0 = gx.ConstantStepSize(), 1.7
    elif case == "pid_dtmin":
        ctrl, dt0 = gx.PIDController(rtol=1e-8, atol=1e-10, pcoeff=0.3, icoeff=0.4, dcoeff=0.05, dtmin=0.4, dtmax=9.0), 2.0
    else:
        ctrl = gx.PIDController(rtol=1e-8, atol=1e-10)
    cfg = gx.Integrator(solver=solver, stepsize_controller=ctrl, dt0=dt0, max_steps=2**16).config()
    order = rng.permutation(n).astype(np.int32) if case == "order" else None

    def run():
        kw = {}
        if case == "host_saves":  # no save scratch: Dopri8's saves are sub-steps inside the integration
            kw["out"] = torch.empty((6, int(offs[-1])), dtype=torch.float64).pin_memory()
        out, status, steps = D.integrate(mw, y0, t0, t1, ts, cfg, save_offsets=offs, order=order,
                                         workspace=D.Workspace(), **kw)
        torch.cuda.synchronize()
        return [v.cpu().numpy().copy() for v in (out, status, steps)]

    try:
        team = run()
        _lib.check(L.gal_set_team(0), "gal_set_team")
        alone = run()
    finally:
        _lib.check(L.gal_set_team(32), "gal_set_team")
    for a, b in zip(team, alone):
        np.testing.assert_array_equal(a, b)
    assert (alone[1] == 0).any()
