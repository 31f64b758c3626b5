"""The surrogate's stages with a network (beside the analytic term where there is
no near field) against the stage kernel without one: a network of zeros adds
nothing. Batches with partial warps, points beyond the near field's cells,
captured and direct launches."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 300])
@pytest.mark.parametrize("with_near", [True, False])
@pytest.mark.parametrize("host", ["mw", "table"])
def test_zero_network_adds_nothing(n, with_near, host):
    import torch

    import galax_gb300 as gx
    from galax_gb300 import surrogate as S

    rng = np.random.default_rng(n)
    pot = gx.MilkyWayPotential() if host == "mw" else gx.MilkyWayPotential2022()
    c = rng.normal(size=(60, 3)) * 15.0
    spheres = gx.CompositePotential([gx.PlummerPotential(m_tot=1e8, r_s=0.3 + 0.01 * i, origin=tuple(c[i]))
                                     for i in range(60)])
    near = S.ShortRange(spheres, 8.0) if with_near else None
    mlp = S.MLPSurrogate(np.zeros(S.num_params(), np.float32), 50.0, 1e-3)
    x = rng.normal(size=(n, 3)) * 8.0
    y0 = np.concatenate([x, rng.normal(size=(n, 3)) * 0.12], axis=1)
    if n > 2:
        y0[1, :3] = [400.0, 0.0, 0.0]  # no cell there
    y0 = torch.as_tensor(y0, device="cuda")
    plain = S.integrate(pot, None, y0, 0.0, 10.0, 1.0, near=near)
    got = S.integrate(pot, mlp, y0, 0.0, 10.0, 1.0, near=near)
    direct = S.integrate(pot, mlp, y0, 0.0, 10.0, 1.0, near=near, use_graph=False)
    assert torch.equal(got, direct)
    assert torch.equal(got, plain)
