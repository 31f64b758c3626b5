"""Dopri8 saves taken as one parallel pass after the integration against the
same saves taken inside it: the same arithmetic, so the same bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _potentials():
    import galax_gb300 as gx

    return {
        "mw": gx.MilkyWayPotential(),
        "table": gx.MilkyWayPotential2022(),
        "timed": gx.MilkyWayPotential(halo={"m": gx.LinearParameter(slope=6e7, point_time=0.0, point_value=5.4e11)}),
    }


@pytest.mark.parametrize("pot_name", ["mw", "table", "timed"])
@pytest.mark.parametrize("adaptive", [True, False])
@pytest.mark.parametrize("n,n_saves,csr,back", [(1, 1, False, False), (1, 257, False, False), (33, 7, False, True),
                                                (70, 19, True, False)])
def test_same_bits_as_inline_saves(monkeypatch, pot_name, adaptive, n, n_saves, csr, back):
    import torch

    import galax_gb300 as gx
    from galax_gb300 import dynamics as D

    pot = _potentials()[pot_name]
    rng = np.random.default_rng(7)
    x = rng.normal(size=(n, 3)) * 8.0
    y0 = np.concatenate([x, rng.normal(size=(n, 3)) * 0.12], axis=1)
    y0[0] = [8.0, 0.0, 0.0, 0.0, 0.22, 0.0]
    if n > 2:
        y0[2, 0] = np.inf  # ends as non-finite: NaN saves
    T = -300.0 if back else 300.0
    ctrl = gx.PIDController(rtol=1e-7, atol=1e-7) if adaptive else gx.ConstantStepSize()
    cfg = gx.Integrator(solver=gx.Dopri8(), stepsize_controller=ctrl, dt0=None if adaptive else 2.0).config()
    kw = {}
    if csr:
        lens = rng.integers(0, n_saves, n)
        offs = np.zeros(n + 1, np.int64)
        offs[1:] = np.cumsum(lens)
        ts = np.concatenate([np.sort(rng.uniform(0.0, T, k)) for k in lens])
        kw["save_offsets"] = offs
    else:
        ts = np.linspace(0.0, T, n_saves)  # the start, the end, and (constant steps) step ends among them

    def run():
        return D.integrate(pot, y0, 0.0, T, ts, cfg, workspace=D.Workspace(), **kw)

    deferred = run()
    monkeypatch.setattr(D, "SAVE_SCRATCH_MAX", -1)  # no scratch: saves inside the integration
    inline = run()
    for a, b in zip(deferred, inline):
        assert torch.equal(torch.nan_to_num(a.double(), nan=-7.0), torch.nan_to_num(b.double(), nan=-7.0))
    assert bool(torch.isfinite(deferred[0]).any())


def _saves_case():
    import galax_gb300 as gx

    rng = np.random.default_rng(7)
    y0 = np.concatenate([rng.normal(size=(40, 3)) * 8.0, rng.normal(size=(40, 3)) * 0.12], axis=1)
    return gx.MilkyWayPotential(), y0, np.linspace(0.0, 200.0, 50), gx.Integrator().config()


def test_no_memory_for_the_save_scratch(monkeypatch):
    """A workspace that cannot grow to the scratch: saves inside the integration, same results."""
    import torch

    from galax_gb300 import dynamics as D

    pot, y0, ts, cfg = _saves_case()
    want = D.integrate(pot, y0, 0.0, 200.0, ts, cfg, workspace=D.Workspace())

    class Small(D.Workspace):
        def get(self, nbytes):
            if nbytes > 40 * 50 * 8:
                raise torch.cuda.OutOfMemoryError("no room")
            sizes.append(nbytes)
            return super().get(nbytes)

    sizes = []
    got = D.integrate(pot, y0, 0.0, 200.0, ts, cfg, workspace=Small())
    monkeypatch.setattr(D, "_WS", Small())
    kept = D.integrate(pot, y0, 0.0, 200.0, ts, cfg)
    assert len(sizes) == 2
    for res in (got, kept):
        for a, b in zip(want, res):
            assert torch.equal(a, b)


@pytest.mark.parametrize("bound", ["SAVE_SCRATCH_KEPT", "SAVE_SCRATCH_MAX"])
def test_the_callers_workspace_is_used(monkeypatch, bound):
    import torch

    from galax_gb300 import dynamics as D

    pot, y0, ts, cfg = _saves_case()
    want = D.integrate(pot, y0, 0.0, 200.0, ts, cfg, workspace=D.Workspace())
    monkeypatch.setattr(D, bound, 100)

    class Own(D.Workspace):
        def get(self, nbytes):
            sizes.append(nbytes)
            return super().get(nbytes)

    sizes = []
    got = D.integrate(pot, y0, 0.0, 200.0, ts, cfg, workspace=Own())
    assert len(sizes) == 1 and (sizes[0] > 40 * 50 * 8) == (bound == "SAVE_SCRATCH_KEPT")
    for a, b in zip(want, got):
        assert torch.equal(a, b)
