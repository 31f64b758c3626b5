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
