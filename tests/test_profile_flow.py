"""A profile's V-cycles are the solve's: as many kernels as the V-cycle of the
solve's graph has, with the forms that the tuner chose or that are forced, and
the state after n of them is that of a solve stopped there."""
import numpy as np
import pytest

from bsam import ebOptions
from bsam.batch import merge_flats
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend
from cases import vardc_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('form', [None, '6', '1', '5'])
@pytest.mark.parametrize('count', [1, 3])
def test_profile_runs_the_solve_s_cycles(precision, form, count, monkeypatch):
    from bsam.device import DeviceBackend, DevHier
    if form:
        monkeypatch.setenv('BSAM_RELAX_N', form)
    else:
        monkeypatch.delenv('BSAM_RELAX_N', raising=False)
    flats = []
    for i in range(count):
        o = ebOptions('BaseCells', 32, 'MaxLevels', 3 - i % 2, 'Indicator', 'fun', 'Verbose', 0, 'RelTol', 1e-30,
                      'MaxVCycles', 3, 'Precision', precision, 'TagFunction', lambda x, y: np.abs(x - y) < 0.1 + 0.05 * i)
        flats.append(flatten(build_hierarchy(vardc_problem(), o, OracleBackend())))
    fl = merge_flats(flats) if count > 1 else flats[0]
    a, b = (DevHier(DeviceBackend.get(0).ctx, fl, o) for _ in range(2))
    a.solve_cycles(5)
    pr = b.profile(3)
    assert sum(r['launches'] for r in pr.values()) == 3 * a.kernels_per_vcycle()
    for which, n in ((0, fl.Q.size), (3, fl.QC.size)):
        np.testing.assert_array_equal(a.get(which, n), b.get(which, n))
    # and the handle solves on as any other
    for d in (a, b):
        d.set(0, fl.Q)
    (ia, ha, _, _), (ib, hb, _, _) = a.solve_cycles(5), b.solve_cycles(5)
    assert ia == ib
    np.testing.assert_array_equal(ha, hb)
