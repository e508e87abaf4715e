"""Quotients from a stored reciprocal (quotient.cuh) against exact ones.

The header's functions, compiled for the host (IEEE arithmetic there and on
the device), over random and extreme operands: within (1/2 + 2^-50) units in
the last place, and equal to the division where it is used instead.
"""
import ctypes as C
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "smili_b200", "csrc")


@pytest.fixture(scope="module")
def div(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotient")
    src, out = d / "q.cpp", d / "q.so"
    src.write_text('#include "quotient.cuh"\nextern "C" void quotients(int n, const double* b, const double* t, '
                   'double* q) { for (int i = 0; i < n; ++i) q[i] = div_by(b[i], t[i], rcp_of(t[i])); }\n')
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-o", str(out), str(src)],
                   check=True)
    lib = C.CDLL(str(out))

    def call(b, t):
        b, t = np.ascontiguousarray(b, dtype=np.float64), np.ascontiguousarray(t, dtype=np.float64)
        q = np.empty_like(b)
        p = C.POINTER(C.c_double)
        lib.quotients(b.size, b.ctypes.data_as(p), t.ctypes.data_as(p), q.ctypes.data_as(p))
        return q
    return call


def _operands(rng, n, spread):
    s = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    return s * rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-spread, spread + 1, n)


@pytest.mark.parametrize("spread", [0, 3, 100, 460])
def test_quotients_are_within_half_a_unit(div, spread):
    rng = np.random.default_rng(spread)
    n = 20000
    b, t = _operands(rng, n, spread), _operands(rng, n, spread)
    # significands at the ends of the binade, where q is furthest off
    ends = np.array([1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), np.nextafter(1.0, 2.0) + 2 ** -52, 1.5])
    b[:25], t[:25] = np.repeat(ends, 5), np.tile(ends, 5)
    q = div(b, t)
    limit = Fraction(1, 2) + Fraction(1, 2 ** 50)
    for bi, ti, qi in zip(b.tolist(), t.tolist(), q.tolist()):
        exact = Fraction(bi) / Fraction(ti)
        # the unit of the binade that holds the exact quotient
        k = math.frexp(abs(bi / ti))[1] - 53
        if abs(exact) < Fraction(2) ** (k + 52):
            k -= 1
        assert abs(Fraction(qi) - exact) <= limit * Fraction(2) ** k


def test_extreme_operands_take_the_division(div):
    v = [0.0, -0.0, 5e-324, 1e-310, 2.3e-308, 1e-290, 1e-141, 1e-139, 1.0, 3.0, 1e139, 1e141, 1e300, 1.7e308,
         np.inf, -np.inf, np.nan, -1e-300, -7.0]
    b, t = (a.ravel() for a in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        want = b / t
    got = div(b, t)
    same = (got == want) | (np.isnan(got) & np.isnan(want))
    with np.errstate(all="ignore"):
        near = np.abs(got - want) <= 2.0 ** -52 * np.abs(want)
    assert (same | (near & (np.abs(want) > 1e-140) & (np.abs(want) < 1e140))).all()
