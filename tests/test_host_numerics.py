"""Kernel arithmetic that the host's compiler can run too, against exact values."""

from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from decimal import Decimal, getcontext
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "galax_gb300" / "csrc"
U = 2.0**-53


def _compile(tmp_path, source: str) -> C.CDLL:
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    src, lib = tmp_path / "host.cpp", tmp_path / "host.so"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-D__host__=", "-D__device__=",
                    "-D__forceinline__=inline", f"-I{CSRC}", "-o", str(lib), str(src)], check=True)
    return C.CDLL(str(lib))


FIXED = r"""
#include "fixed_plummer.cuh"
extern "C" int sphere(const double* c, double b, double Gm, const double* x, double* f, double* d) {
  const gal::FixedPlummer p = gal::fixed_record(c, b, Gm);
  return gal::fixed_plummer(p, x, f, d);
}
"""


@pytest.mark.parametrize("b,c,d", [
    (0.3, 15.0, 10.0), (0.1, 5.0, 0.1), (1e-3, 1.0, 1e-3), (0.01, 8.0, 0.01), (0.01, 800.0, 0.02), (0.01, 1e5, 1.0),
    (0.0, 8.0, 1e-8), (1e-9, 0.0, 1e-12), (5.0, 1e5, 1.0), (0.5, 20.0, 1e-9), (1e3, 5.0, 5.0), (0.0, 0.0, 3.0),
    (1e-60, 0.0, 1e-60), (1e60, 1.0, 1e61),
])
def test_fixed_point_sphere_terms(tmp_path, b, c, d):
    """A term's error relative to itself, component by component, at any scale of
    sphere and offset. The offset is rounded once (U); the norm takes its squares, so
    f has 3 U of that, its own truncations (U / 8) and its rounding (U); with the
    offset's again: 5.2 U. (FP64 as comp_grad has it: about 10 U.)"""
    getcontext().prec = 60
    L = _compile(tmp_path, FIXED)
    rng = np.random.default_rng(5)
    D = Decimal
    for i in range(300):
        centre, off = rng.normal(size=3), rng.normal(size=3)
        centre *= c / np.linalg.norm(centre)
        x = centre + off * d * rng.uniform(0.3, 3.0) / np.linalg.norm(off)
        if i % 5 == 0:
            x[2] = centre[2]
        if i % 7 == 0:
            x[1] = centre[1] + (x[1] - centre[1]) * 1e-9
        bi = b * rng.uniform(0.5, 1.5)
        Gm = float(np.exp(rng.uniform(-20.0, 20.0)) * rng.choice([-1.0, 1.0]))
        f, o = C.c_double(), (C.c_double * 3)()
        assert L.sphere((C.c_double * 3)(*centre), C.c_double(bi), C.c_double(Gm), (C.c_double * 3)(*x), C.byref(f), o)
        dx = [D(float(x[j])) - D(float(centre[j])) for j in range(3)]
        s = sum(v * v for v in dx) + D(bi) * D(bi)
        want = D(Gm) / (s * s.sqrt())
        for j in range(3):
            got = D(f.value) * D(o[j])
            assert abs(got - want * dx[j]) <= D(5.2 * U) * abs(want * dx[j])


def test_fixed_point_leaves_the_ends_of_the_range_to_fp64(tmp_path):
    L = _compile(tmp_path, FIXED)
    f, o = C.c_double(), (C.c_double * 3)()

    def fits(c, b, Gm, x):
        ok = L.sphere((C.c_double * 3)(*c), C.c_double(b), C.c_double(Gm), (C.c_double * 3)(*x), C.byref(f), o)
        assert ok or f.value == 0.0
        return bool(ok)

    nan, inf = float("nan"), float("inf")
    assert fits((1, 2, 3), 0.5, 1.0, (1, 2, 3)) and f.value != 0.0 and list(o) == [0.0] * 3
    assert fits((1, 2, 3), 0.5, 0.0, (3, 2, 1)) and f.value == 0.0
    assert not fits((1, 2, 3), 0.0, 1.0, (1, 2, 3))  # on a point mass
    assert not fits((0, 0, 0), 0.0, 1.0, (1e-80, 0, 0)) and not fits((0, 0, 0), 1.0, 1.0, (1e80, 0, 0))
    assert not fits((0, 0, 0), 1.0, 1e61, (1, 0, 0)) and not fits((0, 0, 0), 1.0, 1e-61, (1, 0, 0))
    for bad in (nan, inf, -inf):
        assert not fits((0, 0, 0), 1.0, 1.0, (0, bad, 0))


NYSTROM = r"""
#include <cmath>
using std::fma;
#include "nystrom.cuh"
using namespace gal;
template <class TB>
static void table(double* a, double* b, double* v) {
  for (int i = 0; i < TB::S; ++i) {
    for (int l = 0; l < TB::S; ++l) *a++ = kNystrom<TB>.a[i][l];
    *b++ = kNystrom<TB>.b[i];
    *v++ = kNystrom<TB>.v[i];
  }
}
extern "C" void nystrom(int method, double* a, double* b, double* v) {
  if (method == 8) table<Dopri8>(a, b, v);
  else table<Dopri5>(a, b, v);
}
"""


@pytest.mark.parametrize("method", [5, 8])
def test_nystrom_coefficients_are_rounded_once(tmp_path, method):
    """abar = A A and bbar = b A to one rounding (2^-53 relative) or exactly zero,
    and velocity weights next to b whose sum is 1 exactly."""
    from oracle import oracle as O

    S = 13 if method == 8 else 7
    a, b, v = np.empty((S, S)), np.empty(S), np.empty(S)
    _compile(tmp_path, NYSTROM).nystrom(method, *(w.ctypes.data_as(C.c_void_p) for w in (a, b, v)))
    _, A, B, _ = O.tableau(method)[-4:]
    exact = np.vectorize(Fraction)
    A, B = exact(A[:S, :S]), exact(B[:S])
    want_a, want_b = A @ A, B @ A
    for got, want in zip(np.append(a, b), np.append(want_a, want_b)):
        if got == 0.0:
            assert abs(want) < 1e-15
        else:
            assert abs(Fraction(float(got)) - want) <= abs(want) * Fraction(1, 2**53)
    assert sum(exact(v)) == 1
    assert np.all(np.abs(v - B.astype(float)) <= np.spacing(np.abs(v)))
