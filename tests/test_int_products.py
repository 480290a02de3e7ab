"""Products formed on the integer pipe (mul_int_pipe in kernels.cuh) on levels
of 16,384 cells and more: solves equal the oracle bit for bit on square and
ragged cells, one level and refined, with sources whose values are zero over
most of the domain, near the top of the exponent range, and whose products
fall into the denormal range.  The last on ragged cells only: on power-of-two
cells the coefficients are scaled by 1/h^2 beforehand, which rounds a
denormal product differently from the oracle's division after it."""
import numpy as np
import pytest

from bsam import ebOptions, ebProblem
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend, OracleHier

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('base,lx,levels', [([128, 128], 1.0, 1), ([160, 128], 1.25, 2), ([144, 120], 1.3, 2)])
@pytest.mark.parametrize('scale,source', [(1.0, 'smooth'), (1e-303, 'smooth'), (1e300, 'smooth'), (1.0, 'spot')])
def test_large_levels_match_the_oracle(base, lx, levels, scale, source):
    if scale < 1e-300 and lx != 1.3:
        pytest.skip('denormal products of scaled coefficients')
    from bsam.device import DeviceBackend, DevHier
    D = lambda x, y: 1 + 0.5 * np.sin(3 * x) * np.cos(2 * y)
    f = (lambda x, y: scale * (np.cos(4 * x) * y - 0.3)) if source == 'smooth' else \
        (lambda x, y: scale * np.where((x - 0.4) ** 2 + (y - 0.4) ** 2 < 0.001, 1.0, 0.0))
    prob = ebProblem([0, lx, 0, 1], D, 1.0, f, ('dirichlet', 0))
    o = ebOptions('BaseCells', base, 'MaxLevels', levels, 'Indicator', 'fun', 'Verbose', 0, 'RelTol', 0.0,
                  'MaxVCycles', 3, 'TagFunction', lambda x, y: np.abs(x / lx - y) < 0.3)
    fl = flatten(build_hierarchy(prob, o, OracleBackend()))
    oh = OracleHier(fl, o)
    it, hist, rel, _ = oh.solve_cycles(10)
    dh = DevHier(DeviceBackend.get(0).ctx, fl, o)
    itd, histd, reld, _ = dh.solve_cycles(10)
    assert it == itd
    np.testing.assert_array_equal(hist, histd)
    np.testing.assert_array_equal(oh.Q, dh.get(0, fl.Q.size))
    np.testing.assert_array_equal(oh.F, dh.get(1, fl.F.size))
