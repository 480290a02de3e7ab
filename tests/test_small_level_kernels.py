"""The coarse load with four lanes per footprint cell and the residual with one
cell per item (levels below 65,536 cells, hierarchies below 131,072): footprint
counts that leave partial warps and blocks, odd and one-cell-wide footprints,
several patches, both kinds of corrections.  FP64 equals the oracle bit for
bit."""
import numpy as np
import pytest

from bsam import ebOptions, ebProblem
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend, OracleHier


@pytest.mark.gpu
@pytest.mark.parametrize('ghost', ['qif', 'lif'])
@pytest.mark.parametrize('base,lx,levels', [([16, 16], 1.0, 4), ([12, 20], 1.3, 3), ([10, 6], 1.0, 3),
                                            ([50, 22], 1.0, 3)])
def test_small_levels_match_the_oracle(base, lx, levels, ghost):
    from bsam.device import DeviceBackend, DevHier
    D = lambda x, y: 1 + 0.5 * np.sin(3 * x) * np.cos(2 * y)
    prob = ebProblem([0, lx, 0, 1], D, 1.0, lambda x, y: np.cos(4 * x) * y,
                     {'west': ('dirichlet', 0.3), 'east': ('neumann', 0.1), 'south': ('neumann', 0),
                      'north': ('dirichlet', 0)})
    o = ebOptions('BaseCells', base, 'MaxLevels', levels, 'Indicator', 'fun', 'Verbose', 0, 'RelTol', 1e-10,
                  'GhostInterp', ghost,
                  'TagFunction', lambda x, y, L: ((x - 0.3 * lx) ** 2 + (y - 0.4) ** 2 < 0.03) | (x + y > 1.2 * lx))
    fl = flatten(build_hierarchy(prob, o, OracleBackend()))
    oh = OracleHier(fl, o)
    it, hist, rel, _ = oh.solve_cycles(o.MaxVCycles + 2)
    dh = DevHier(DeviceBackend.get(0).ctx, fl, o)
    itd, histd, reld, _ = dh.solve_cycles(o.MaxVCycles + 2)
    assert it == itd
    np.testing.assert_array_equal(hist, histd)
    np.testing.assert_array_equal(oh.Q, dh.get(0, fl.Q.size))
