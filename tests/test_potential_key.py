"""A potential's device handle is rebuilt when a value of its component table
changes, however its owner changes it."""

import numpy as np
import pytest

import galax_gb300 as gx


@pytest.mark.parametrize("change", [
    lambda p: setattr(p, "m_tot", 2e9),
    lambda p: p.m_tot.__setitem__(..., 2e9),
    lambda p: p.origin.__setitem__(1, 0.5),
    lambda p: setattr(p, "origin", np.array([1.0, 2.5, 3.0])),
    lambda p: p.constants.__setitem__("G", 1.0),
])
@pytest.mark.parametrize("composite", [False, True])
@pytest.mark.parametrize("step", [1, 2])  # an origin that is a strided view too
def test_key_follows_values(change, composite, step):
    inner = gx.PlummerPotential(m_tot=1e9, r_s=1.0)
    inner.m_tot, inner.origin = np.array(1e9), np.array([1.0, 9.0, 2.0, 9.0, 3.0, 9.0])[:3 * step:step]
    pot = gx.CompositePotential([inner, gx.KeplerPotential(m_tot=1e8)]) if composite else inner
    before, again = pot._table_key(), pot._table_key()
    assert before == again
    change(pot if composite and "constants" in change.__code__.co_names else inner)
    assert pot._table_key() != before
    assert pot._table_key() == pot._table_key()
