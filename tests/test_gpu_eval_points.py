"""Potential evaluation on points in any layout (slices, transposes, broadcasts
and other types), and the Milky Way's own Hessian kernel against the component
table's: rounding level, as the two order the same sums differently."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["potential", "gradient", "acceleration", "hessian"])
@pytest.mark.parametrize("n", [1, 127, 129, 5000])
def test_layouts(what, n):
    import torch

    import galax_gb300 as gx

    mw = gx.MilkyWayPotential()
    g = torch.Generator(device="cuda").manual_seed(n)
    base = torch.randn((n, 7), generator=g, device="cuda", dtype=torch.float64) * 9.0
    ref = getattr(mw, what)(base[:, 2:5].contiguous())
    for x in (base[:, 2:5], base[:, 2:5].t().contiguous().t()):
        assert torch.equal(getattr(mw, what)(x), ref)
    assert torch.equal(getattr(mw, what)(base[:, None, 2:5]), ref[:, None])
    assert torch.equal(getattr(mw, what)(base[:1, 2:5].expand(n, 3)), ref[:1].expand_as(ref))
    low = base[:, 2:5].float()
    assert torch.equal(getattr(mw, what)(low), getattr(mw, what)(low.double()))
    np.testing.assert_array_equal(getattr(mw, what)(base[:, 2:5].cpu().numpy()), ref.cpu().numpy())


def test_milky_way_hessian_over_the_radii():
    import galax_gb300 as gx

    rng = np.random.default_rng(4)
    d = rng.normal(size=(20000, 3))
    x = d / np.linalg.norm(d, axis=1, keepdims=True) * np.exp(rng.uniform(np.log(0.05), np.log(300.0), 20000))[:, None]
    x[:3] = [[8.0, 0.0, 0.0], [0.0, 0.0, 3.0], [0.0, 2.0, 0.0]]
    ref = O.hessian(O.milky_way(), x)
    H = gx.MilkyWayPotential().hessian(x)
    scale = np.abs(ref).max(axis=(1, 2), keepdims=True)
    # about 30 roundings of 2^-53 each in sums of like terms; the halo's cancel by (r_s / r)^2 / 6 < 2e4 at 0.05 kpc,
    # where it is below 1e-3 of the nucleus
    assert np.max(np.abs(H - ref) / scale) < 30 * 20 * 2.0**-53
    assert np.array_equal(H, np.swapaxes(H, 1, 2))


def test_lazily_negated_view():
    """The imaginary part of a conjugate is a view whose memory holds the negated values."""
    import torch

    import galax_gb300 as gx

    z = torch.complex(*torch.randn((2, 300, 3), device="cuda", dtype=torch.float64))
    x = z.conj().imag
    assert x.is_neg()
    mw = gx.MilkyWayPotential()
    for what in ("potential", "gradient", "hessian"):
        assert torch.equal(getattr(mw, what)(x), getattr(mw, what)(x.resolve_neg().contiguous()))
