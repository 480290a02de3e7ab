"""The kernels divide by a level's h^2 with one product and fused corrections
(DivC in kernels.cuh).  CPU: the same steps in exact rational arithmetic give
the correctly rounded quotient for constants of both kinds (three and five
operations) and operands at and beside rounding boundaries.  GPU: solves on
grids whose h^2 is no power of two in one or both directions equal the
oracle, which divides, bit for bit."""
from fractions import Fraction
import math

import numpy as np
import pytest

from bsam import ebOptions, ebProblem
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend, OracleHier


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _ops(d):
    r = 1.0 / d
    return 1 if math.frexp(d)[0] == 0.5 else 3 if abs(_fma(r, d, -1.0)) < 2.0 ** -54 else 5


def _div(x, d):
    r, ops = 1.0 / d, _ops(d)
    q = x * r
    if ops == 1:
        return q
    for _ in range(1 if ops == 3 else 2):
        q = _fma(_fma(-q, d, x), r, q)
    return q


def test_quotients_are_correctly_rounded():
    rng = np.random.default_rng(3)
    seen = set()
    for lx, n in ((1.3, 120), (0.924, 44), (1.0, 15), (1.6, 13), (math.pi, 64), (0.7, 9), (1.0, 64)):
        d = (lx / n) * (lx / n)
        seen.add(_ops(d))
        xs = list(rng.normal(size=150)) + list(np.ldexp(rng.normal(size=50), rng.integers(-700, 700, 50)))
        for m in 1 + rng.random(150):       # quotients next to the midpoint of two doubles
            x = float(Fraction(d) * (Fraction(m) + Fraction(1, 2 ** 53)))
            xs += [x, np.nextafter(x, 0), np.nextafter(x, 10)]
        for x in xs:
            assert _div(float(x), d) == float(x) / d, (x, d)
    assert seen == {1, 3, 5}


@pytest.mark.gpu
@pytest.mark.parametrize('lx,base', [(1.3, [24, 16]), (1.0, [12, 20]), (0.924, [24, 32]), (1.6, [26, 18])])
def test_ragged_solves_match_the_oracle(lx, base):
    from bsam.device import DeviceBackend, DevHier
    D = lambda x, y: 1 + 0.5 * np.sin(3 * x) * np.cos(2 * y)
    prob = ebProblem([0, lx, 0, 1], D, 1.0, lambda x, y: np.cos(4 * x) * y,
                     {'west': ('dirichlet', 0.3), 'east': ('neumann', 0.1), 'south': ('neumann', 0),
                      'north': ('dirichlet', 0)})
    o = ebOptions('BaseCells', base, 'MaxLevels', 3, 'Indicator', 'fun', 'Verbose', 0, 'RelTol', 1e-10,
                  'TagFunction', lambda x, y, L: (x - 0.5 * lx) ** 2 + (y - 0.5) ** 2 < 0.09 / L ** 2)
    fl = flatten(build_hierarchy(prob, o, OracleBackend()))
    oh = OracleHier(fl, o)
    it, hist, rel, _ = oh.solve_cycles(o.MaxVCycles + 2)
    dh = DevHier(DeviceBackend.get(0).ctx, fl, o)
    itd, histd, reld, _ = dh.solve_cycles(o.MaxVCycles + 2)
    assert it == itd
    np.testing.assert_array_equal(hist, histd)
    np.testing.assert_array_equal(oh.Q, dh.get(0, fl.Q.size))
