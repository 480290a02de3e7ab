"""The smoother and the coarse load form the quotients of a cell together
(div_group in kernels.cuh), the FP32 cycle's from the FP32 reciprocal of h^2.
CPU: the FP32 steps in exact arithmetic give the correctly rounded quotient
for constants that take one and two steps.  GPU: the mixed solve with the
chained and the tile form equals the one whose smoother divides, bit for
bit, with sources large and small enough to leave the steps' range."""
from fractions import Fraction
import math

import numpy as np
import pytest

from bsam import ebOptions, ebProblem
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend

f32 = np.float32


def _rn(x):
    """correctly rounded FP32 value of an exact rational (normal range)"""
    if x == 0:
        return f32(0)
    m, e = math.frexp(float(x))              # float(): within half an FP64 ulp, only the exponent is used
    s = Fraction(2) ** (24 - e)
    n = round(x * s)                         # ties to even
    return f32(float(Fraction(n) / s))


def _steps(x, d):
    r = _rn(1 / Fraction(float(d)))
    fx, fd, fr = Fraction(float(x)), Fraction(float(d)), Fraction(float(r))
    rel = abs(fr * fd - 1)
    q = _rn(fx * fr)
    n = 1 if rel < Fraction(1, 2 ** 25) else 2
    for k in range(2):                       # a second step leaves a correct quotient as it is
        fq = Fraction(float(q))
        q = _rn(fq + Fraction(float(_rn(fx - fq * fd))) * fr)
        if k + 1 == n:
            first = q
    return first, q, n


def test_fp32_quotients_are_correctly_rounded():
    rng = np.random.default_rng(5)
    seen = set()
    for lx, n in ((1.3, 120), (0.924, 44), (1.0, 15), (1.6, 13), (math.pi, 64), (0.7, 9), (1.0, 11), (1.0, 23)):
        d = f32((lx / n) * (lx / n))
        xs = [f32(v) for v in rng.normal(size=120)]
        for m in 1 + rng.random(120):        # quotients next to the midpoint of two floats
            x = _rn(Fraction(float(d)) * (Fraction(float(f32(m))) + Fraction(1, 2 ** 24)))
            xs += [x, np.nextafter(x, f32(0)), np.nextafter(x, f32(10))]
        for x in xs:
            want = _rn(Fraction(float(x)) / Fraction(float(d)))
            a, b, k = _steps(x, d)
            seen.add(k)
            assert a == want and b == want, (x, d)
    assert seen == {1, 2}


@pytest.mark.gpu
@pytest.mark.parametrize('form', ['1', '6'])
@pytest.mark.parametrize('lx,base,scale', [(1.3, [24, 16], 1.0), (1.0, [12, 20], 1e-30), (0.924, [24, 32], 1e25),
                                           (1.0, [15, 11], 1.0)])
def test_mixed_solves_equal_the_dividing_form(monkeypatch, form, lx, base, scale):
    from bsam.device import DeviceBackend, DevHier
    D = lambda x, y: 1 + 0.5 * np.sin(3 * x) * np.cos(2 * y)
    prob = ebProblem([0, lx, 0, 1], D, 1.0, lambda x, y: scale * np.cos(4 * x) * y,
                     {'west': ('dirichlet', 0.3 * scale), 'east': ('neumann', 0.1 * scale), 'south': ('neumann', 0),
                      'north': ('dirichlet', 0)})
    o = ebOptions('BaseCells', base, 'MaxLevels', 3, 'Indicator', 'fun', 'Verbose', 0, 'RelTol', 1e-10,
                  'Precision', 'mixed',
                  'TagFunction', lambda x, y, L: (x - 0.5 * lx) ** 2 + (y - 0.5) ** 2 < 0.09 / L ** 2)
    fl = flatten(build_hierarchy(prob, o, OracleBackend()))
    out = []
    for kn in ('2', form):                   # 2: a launch form that keeps the divisions
        monkeypatch.setenv('BSAM_RELAX_N', kn)
        dh = DevHier(DeviceBackend.get(0).ctx, fl, o)
        it, hist, rel, _ = dh.solve_cycles(o.MaxVCycles + 2)
        out.append((it, hist, dh.get(0, fl.Q.size)))
    assert out[0][0] == out[1][0]
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][2], out[1][2])
