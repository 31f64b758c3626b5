"""Tables of many Plummer spheres with constant steps, whose spheres are
evaluated in fixed point, against the same orbits with every component in FP64
(one thread per orbit) and against the oracle."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _table(gx, k, others, rng):
    c = rng.normal(size=(k, 3))
    c *= rng.uniform(5.0, 50.0, (k, 1)) / np.linalg.norm(c, axis=1, keepdims=True)
    m, b = np.exp(rng.uniform(np.log(1e6), np.log(1e8), k)), rng.uniform(0.1, 1.0, k)
    m[0], b[0] = -3e7, 0.0        # a hole, and a point mass
    b[1], c[1] = 1e-9, [8.0, 0.0, 0.0]   # below the fixed-point unit's high word, on an orbit's start
    c[2], m[3] = 0.0, 0.0
    spheres = [gx.PlummerPotential(m_tot=m[i], r_s=b[i], origin=tuple(c[i])) for i in range(k)]
    if others == "mw":
        return gx.CompositePotential(spheres[:5] + [gx.MilkyWayPotential()] + spheres[5:])
    if others == "none":
        return gx.CompositePotential(spheres + [gx.PlummerPotential(m_tot=5e11, r_s=10.0)])
    return gx.CompositePotential([gx.IsochronePotential(m_tot=4e11, r_s=8.0), gx.KeplerPotential(m_tot=1e9)] + spheres)


@pytest.mark.parametrize("method", [5, 8])
@pytest.mark.parametrize("k,others", [(32, "mw"), (33, "table"), (45, "none"), (512, "mw")])
@pytest.mark.parametrize("n", [1, 37, 5000])
def test_fixed_point_spheres_match_fp64(method, k, others, n):
    import galax_gb300 as gx
    from galax_gb300 import _lib
    from galax_gb300.dynamics import integrate

    if n == 5000 and (method == 8 or k == 512):
        pytest.skip("covered by the smaller batches")
    L = _lib.load()
    rng = np.random.default_rng(k + n)
    pot = _table(gx, k, others, rng)
    x = rng.normal(size=(n, 3))
    x *= rng.uniform(4.0, 20.0, (n, 1)) / np.linalg.norm(x, axis=1, keepdims=True)
    y0 = np.concatenate([x, rng.normal(size=(n, 3)) * 0.1], axis=1)
    y0[0] = [9.0, 0.0, 0.0, 0.0, 0.2, 0.0]  # stays in the plane: exact zeros among the offsets
    if n > 4:
        y0[1, :3] = [900.0, 10.0, -3.0]     # beyond the range of the fixed-point positions
        y0[2, 3:] = [40.0, 1.0, 1.0]        # leaves it on the way
        y0[3] = np.nan
    cfg = gx.Integrator(solver=gx.Dopri8() if method == 8 else gx.Dopri5(),
                        stepsize_controller=gx.ConstantStepSize(), dt0=1.0).config()
    ts = np.linspace(0.0, 20.0, 7)
    try:
        fixed = [v.cpu().numpy() for v in integrate(pot, y0, 0.0, 20.0, ts, cfg)]
        _lib.check(L.gal_set_table_lanes(1), "gal_set_table_lanes")
        fp64 = [v.cpu().numpy() for v in integrate(pot, y0, 0.0, 20.0, ts, cfg)]
    finally:
        _lib.check(L.gal_set_table_lanes(0), "gal_set_table_lanes")
    for a, b in zip(fixed[1:], fp64[1:]):
        np.testing.assert_array_equal(a, b)
    a, b = fixed[0], fp64[0]
    assert np.array_equal(np.isnan(a), np.isnan(b))
    ok = ~np.isnan(b).any(axis=(0, 1))
    assert ok.any()
    # 20 steps of at most 13 gradients, each within a few dozen roundings of 2^-53 of
    # the other's, in orbits that amplify by less than 100 over 20 Myr: below 1e-11
    scale = np.linalg.norm(b.reshape(2, 3, *b.shape[1:]), axis=1, keepdims=True)
    assert np.max((np.abs(a - b).reshape(2, 3, *b.shape[1:]) / scale)[..., ok]) < 1e-11
    if n == 37:
        ref, st, _, _ = O.integrate(pot.component_array(), y0[4:], 0.0, 20.0, ts, O.solver_cfg(method, False, dt0=1.0))
        want = np.stack(ref).transpose(2, 1, 0)
        s = np.linalg.norm(want.reshape(2, 3, *want.shape[1:]), axis=1, keepdims=True)
        assert np.max(np.abs(a[:, :, 4:] - want).reshape(2, 3, *want.shape[1:]) / s) < 1e-9


@pytest.mark.parametrize("method", [5, 8])
@pytest.mark.parametrize("reach,b", [(50.0, 0.1), (50.0, 1e-3), (800.0, 0.01), (1e5, 0.01), (1e5, 1e-4)])
def test_near_a_sphere_of_a_wide_table(method, reach, b):
    """Orbits at rest within a few scales of one sphere, the others far away and as
    extended: the velocity after one short step is the gradient's error alone. FP64's
    own is some 10 roundings of 2^-53 per gradient, the fixed-point one's 5; the
    weights' sizes add up to 3.1 (Dopri8) with a rounding of each term: below 1e-14
    together."""
    import galax_gb300 as gx
    from galax_gb300 import _lib
    from galax_gb300.dynamics import integrate

    L = _lib.load()
    rng = np.random.default_rng(9)
    c0 = np.array([8.0, 1.0, -2.0])
    far = rng.normal(size=(40, 3))
    far *= reach / np.linalg.norm(far, axis=1, keepdims=True)
    pot = gx.CompositePotential([gx.PlummerPotential(m_tot=1e9, r_s=b, origin=tuple(c0))] + [
        gx.PlummerPotential(m_tot=1e6, r_s=0.1 * reach, origin=tuple(c)) for c in far])
    x = rng.normal(size=(200, 3))
    x *= b * rng.uniform(0.3, 3.0, (200, 1)) / np.linalg.norm(x, axis=1, keepdims=True)
    y0 = np.concatenate([c0 + x, np.zeros((200, 3))], axis=1)
    dt = 1e-3 * np.sqrt(b**3 / (4.5e-12 * 1e9))  # a thousandth of the sphere's own time
    cfg = gx.Integrator(solver=gx.Dopri8() if method == 8 else gx.Dopri5(),
                        stepsize_controller=gx.ConstantStepSize(), dt0=dt).config()
    try:
        fixed = integrate(pot, y0, 0.0, dt, np.array([dt]), cfg)[0].cpu().numpy()
        _lib.check(L.gal_set_table_lanes(1), "gal_set_table_lanes")
        fp64 = integrate(pot, y0, 0.0, dt, np.array([dt]), cfg)[0].cpu().numpy()
    finally:
        _lib.check(L.gal_set_table_lanes(0), "gal_set_table_lanes")
    v, w = fixed[3:, 0], fp64[3:, 0]
    assert np.all(np.abs(w).max(axis=0) > 0)
    assert np.max(np.linalg.norm(v - w, axis=0) / np.linalg.norm(w, axis=0)) < 1e-14
