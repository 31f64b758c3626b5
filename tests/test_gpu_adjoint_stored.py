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


@pytest.mark.parametrize("method,per", [(5, 560), (8, 1040)])
def test_no_scratch_that_would_not_be_used(method, per):
    import ctypes as C

    import galax_gb300 as gx
    from galax_gb300 import _lib

    L, h = _lib.load(), gx.MilkyWayPotential().handle()
    cfg = _lib.solver_config(method, False, dt0=1.0)

    def extra(n, steps, k_ckpt, most):
        b, w = C.c_size_t(), C.c_size_t()
        _lib.check(L.gal_adjoint_workspace_size(h, C.byref(cfg), 0.0, float(steps), k_ckpt, n, C.byref(b)), "size")
        _lib.check(L.gal_adjoint_workspace_size_stored(h, C.byref(cfg), 0.0, float(steps), k_ckpt, n, most, C.byref(w)),
                   "size_stored")
        return w.value - b.value

    n = 1_000_000
    assert extra(n, 500, 256, 12 * n * per) == 12 * n * per
    assert extra(n, 500, 256, 8 * n * per) == 8 * n * per
    assert extra(n, 500, 256, 8 * n * per - 1) == 0           # seven steps: not worth it
    assert extra(n, 5, 256, 8 * n * per - 1) == 5 * n * per   # all there are
    assert extra(n, 5, 256, 5 * n * per - 1) == 0
    # 50 segments of eight steps, but 21 + 20 states in the checkpoints' area
    assert extra(n, 400, 20, 8 * n * per) == 0
    assert extra(n, 400, 20, 10 * n * per) == 10 * n * per


@pytest.mark.parametrize("free,stage_memory,stored", [(None, None, True), (None, 0, False), (10, None, False),
                                                      (None, 9 * 300 * 1040, True), (None, 7 * 300 * 1040, False)])
def test_memory_bounds(monkeypatch, free, stage_memory, stored):
    import galax_gb300 as gx
    from galax_gb300 import adjoint as A

    sizes = []
    scratch = A._scratch

    def record(nbytes):
        sizes.append(nbytes)
        return scratch(nbytes)

    monkeypatch.setattr(A, "_scratch", record)
    monkeypatch.setattr(A, "_KEPT_MAX", 0)
    if free is not None:
        monkeypatch.setattr(A, "_free_bytes", lambda: free)
    rng = np.random.default_rng(1)
    y0 = np.concatenate([rng.normal(size=(300, 3)) * 8.0, rng.normal(size=(300, 3)) * 0.12], axis=1)
    A.orbit_adjoint(gx.MilkyWayPotential(), y0, 0.0, 30.0, dt=1.0, cotangent=np.ones((300, 6)), k_ckpt=8,
                    stage_memory=stage_memory)
    assert (sizes[0] > 8 * 300 * 1040) == stored


def test_a_larger_kept_workspace_changes_nothing(monkeypatch):
    """stage_memory = 0 gives the checkpointed gradients also where an earlier call left room for stages."""
    import galax_gb300 as gx
    from galax_gb300 import adjoint as A

    rng = np.random.default_rng(1)
    y0 = np.concatenate([rng.normal(size=(30, 3)) * 8.0, rng.normal(size=(30, 3)) * 0.12], axis=1)

    def run(stage_memory):
        r = A.orbit_adjoint(gx.MilkyWayPotential(), y0, 0.0, 30.0, dt=1.0, cotangent=np.ones((30, 6)), k_ckpt=8,
                            stage_memory=stage_memory)
        return r.grad_y0, r.grad_params

    monkeypatch.setattr(A, "_WS", A.Workspace())
    fresh = run(0)
    stored = run(None)
    again = run(0)
    for f, s, a in zip(fresh, stored, again):
        np.testing.assert_array_equal(f, a)
        assert not np.array_equal(f, s)
