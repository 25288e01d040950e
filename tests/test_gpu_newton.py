"""The reduction's 1 / sqrt(x) and 1 / x by Newton's iteration, against the exact values: within 1.5 and 1 units in
the last place (the last step rounds m r to half a unit, which enters the root with weight 1/2, and the result
once; two steps from 22 bits leave an error of 2^-87), over random mantissas and all exponents, powers of
two, the neighbours of 1, 2 and 4, both sides of the cut at 2^+-900 and subnormals.  And the reduction of
a Hamiltonian so small that squared norms are subnormal."""
import ctypes as C
from fractions import Fraction
from math import isqrt

import numpy as np
import pytest

from oracle import lm_oracle as o

pytestmark = pytest.mark.gpu


def _arguments():
    rng = np.random.default_rng(7)
    x = [np.ldexp(rng.uniform(1, 2, 4), e) for e in range(-1022, 1024)]
    p = np.ldexp(1.0, np.arange(-1074, 1024))
    near = [np.ldexp(v, e) for v in (1.0, 2.0, 4.0) for e in (-902, -901, -900, -899, -1, 0, 1, 898, 899, 900, 901)]
    near = np.array(near)
    mant = np.ldexp(1.0 + np.ldexp(rng.integers(0, 1 << 52, 20000).astype(float), -52), rng.integers(-3, 4, 20000))
    sub = np.ldexp(rng.uniform(1, 2, 50), rng.integers(-1073, -1022, 50))
    x = np.concatenate(x + [p, near, np.nextafter(near, 0), np.nextafter(near, np.inf), mant, sub])
    return np.ascontiguousarray(x[(x > 0) & np.isfinite(x)])


def _units(got, exact):
    """|got - exact| in units of got's last place."""
    return abs(Fraction(float(got)) - exact) / Fraction(float(np.spacing(got)))


def test_newton_reciprocals():
    import lmgpu as lm
    ctx = lm.default_context()
    x = _arguments()
    rs, rd = np.empty_like(x), np.empty_like(x)
    pd = C.POINTER(C.c_double)
    ctx.check(ctx.lib.lm_newton_reciprocals(ctx.handle, len(x), *(v.ctypes.data_as(pd) for v in (x, rs, rd))))
    worst = [Fraction(0), Fraction(0)]
    for v, r, d in zip(x, rs, rd):
        q = 1 / Fraction(float(v))
        n = (q * (1 << 2400))  # 1 / sqrt(v) to far beyond 53 bits
        root = Fraction(isqrt(n.numerator // n.denominator), 1 << 1200)
        worst[0] = max(worst[0], _units(r, root))
        if q < Fraction(float(np.finfo(float).max)):
            worst[1] = max(worst[1], _units(d, q))
        else:
            assert np.isinf(d) or float(d) == np.finfo(float).max
    print("largest errors in units of the last place:", [float(w) for w in worst])
    assert worst[0] <= Fraction(3, 2) + Fraction(1, 1000)
    assert worst[1] <= 1


@pytest.mark.parametrize("t1", [3e-155, 2.5e-155, 1e-140, 1e130])
def test_reduction_of_extreme_scale(t1):
    import lmgpu as lm
    lat = lm.SquareLattice(9, 8)
    f = lm.PointFlux(0.2, (4.5, 4.5))
    E = lm.diagonalize(lm.tightbinding_hamiltonian(lat, t1=t1, field=f)).values
    E1 = lm.diagonalize(lm.tightbinding_hamiltonian(lat, t1=1.0, field=f)).values
    assert np.all(np.isfinite(E))
    # squared norms near 1e-309 carry 48 bits
    assert np.abs(E / t1 - E1).max() <= (1e-12 if t1 < 1e-150 else 1e-13) * 4
