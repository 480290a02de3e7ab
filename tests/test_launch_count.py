"""The count of launched kernels does not depend on how a solve ran: as one
graph (at once, or after others), or V-cycle by V-cycle with the stop test on
the host.  Hierarchies with and without levels whose coarse shadows the solve
refreshes at its end, corrections off, both precisions, a solve that has nothing
to do."""
import numpy as np
import pytest

from bsam import ebOptions
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend
from cases import vardc_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('levels,corrections,cycles', [(1, True, 100), (3, True, 100), (3, False, 100), (3, True, 1),
                                                       (3, True, 0)])
def test_every_way_counts_the_same(precision, levels, corrections, cycles, monkeypatch):
    from bsam.device import Context, DevHier
    o = ebOptions('BaseCells', 32, 'MaxLevels', levels, 'Indicator', 'fun', 'Verbose', 0, 'RelTol', 1e-8, 'Precision',
                  precision, 'MassCorrection', corrections, 'MaxVCycles', max(cycles, 1),
                  'TagFunction', lambda x, y: np.abs(x - y) < 0.15)
    if cycles == 0:
        o = ebOptions(dict(o, RelTol=1e30))
    fl = flatten(build_hierarchy(vardc_problem(), o, OracleBackend()))
    monkeypatch.setenv('BSAM_RELAX_N', '1')
    counts, its = set(), set()
    for loop in ('device', 'host'):
        monkeypatch.setenv('BSAM_SOLVE_LOOP', loop)
        dh = DevHier(Context(0), fl, o)
        for _ in range(3):
            dh.set(0, fl.Q)
            n = dh.launch_count()
            its.add(dh.solve_cycles(o.MaxVCycles + 2)[0])
            counts.add(dh.launch_count() - n)
    assert len(its) == 1 and (its.pop() == 0) == (cycles == 0)
    assert len(counts) == 1, counts
