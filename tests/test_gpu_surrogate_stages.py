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


@pytest.mark.parametrize("use_graph", [0, 1])
def test_workspace_without_the_terms_apart(use_graph):
    """Seven slopes and the positions are enough; the analytic term then has no place
    of its own and is evaluated before the network's, with the same bits."""
    import ctypes as C

    import torch

    import galax_gb300 as gx
    from galax_gb300 import _lib
    from galax_gb300 import surrogate as S

    n = 300
    rng = np.random.default_rng(6)
    pot, mlp = gx.MilkyWayPotential(), S.MLPSurrogate(S.init_params(3), 50.0, 2e-4)
    y0 = torch.as_tensor(np.concatenate([rng.normal(size=(3, n)) * 8.0, rng.normal(size=(3, n)) * 0.12]), device="cuda")
    L = _lib.load()
    full = C.c_size_t()
    _lib.check(L.gal_surrogate_workspace_size(n, C.byref(full)), "gal_surrogate_workspace_size")

    def pad(b):
        return (b + 255) // 256 * 256

    least = pad(42 * 8 * n) + pad(3 * 8 * n)
    out = []
    for size in (full.value, least, least - 1):
        y, ws = y0.clone(), torch.empty(size, dtype=torch.uint8, device="cuda")
        out.append((L.gal_integrate_surrogate(pot.handle(), mlp.handle(), None, 1.0, 0.0, 10.0, y.data_ptr(), n, use_graph,
                                              ws.data_ptr(), size, torch.cuda.current_stream().cuda_stream), y))
        torch.cuda.synchronize()
    assert out[0][0] == out[1][0] == 0 and out[2][0] != 0
    assert torch.equal(out[0][1], out[1][1]) and not torch.equal(out[0][1], y0)
    assert torch.equal(out[2][1], y0)
