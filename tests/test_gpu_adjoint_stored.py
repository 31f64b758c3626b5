"""The Milky Way adjoint with stored stages against the checkpointed one: the same
gradients to rounding, in one segment or several, at batch sizes with a partial
warp, forwards and backwards, for both methods and both kinds of loss."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [5, 8])
@pytest.mark.parametrize("n", [1, 33, 200])
@pytest.mark.parametrize("seg", [8, 31, 37, None])
@pytest.mark.parametrize("t1,given", [(36.6, "target"), (-36.6, "cotangent")])
def test_matches_checkpointed_adjoint(method, n, seg, t1, given, monkeypatch):
    import galax_gb300 as gx
    from galax_gb300 import adjoint as A

    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3))
    x *= rng.uniform(2.0, 20.0, (n, 1)) / np.linalg.norm(x, axis=1, keepdims=True)
    y0 = np.concatenate([x, rng.normal(size=(n, 3)) * 0.12], axis=1)
    kw = {given: y0 + 0.1 * rng.normal(size=y0.shape)}
    mw = gx.MilkyWayPotential()

    def run(extra):
        monkeypatch.setattr(A, "STORED_STAGES_MAX", extra)
        monkeypatch.setattr(A, "_WS", A.Workspace())
        return A.orbit_adjoint(mw, y0, 0.0, t1, dt=1.0, method=method, k_ckpt=5 if seg == 8 else 16, **kw)

    per_step = n * 80 * (13 if method == 8 else 7)  # 37 steps, the last one short
    stored, plain = run(1 << 30 if seg is None else seg * per_step), run(0)
    # 37 steps of a few hundred roundings of 2^-53 each, amplified by at most the
    # orbit map's derivative (about 10 over these spans): 1e-11 is an upper bound
    for a, b in ((stored.yT, plain.yT), (stored.grad_y0, plain.grad_y0)):
        scale = np.linalg.norm(b, axis=1, keepdims=True)
        assert np.max(np.abs(a - b) / scale) < 1e-11
    scale = np.abs(plain.grad_params)
    nz = scale > 0
    # sums of either sign over orbits and stages: relative to their largest per-row entry
    assert np.max(np.abs(stored.grad_params - plain.grad_params)[nz] / scale[nz]) < 1e-8
    assert np.array_equal(stored.grad_params[~nz], plain.grad_params[~nz])
