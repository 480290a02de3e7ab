"""The composite residual's report with the flux corrections off
(ebCompResidual.m:15-85 without its lines 40-65): every partial of the report
is written by the launch itself, whatever an earlier report left.  linf, fnorm
and rel are maxima and equal the oracle's; l2 is a sum of n squares in another
order, at most n rounding errors of eps / 2 on either side."""
import numpy as np
import pytest

from bsam import ebOptions
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend, OracleHier
from cases import vardc_problem

pytestmark = pytest.mark.gpu

BAND = lambda x, y, L: np.abs(x - y) < 0.3 / L


def _opts(corrections, base, levels):
    return ebOptions('BaseCells', base, 'MaxLevels', levels, 'Indicator', 'fun', 'TagFunction', BAND, 'Verbose', 0,
                     'MaxVCycles', 1, 'RelTol', 1e-15, 'MassCorrection', corrections)


@pytest.mark.parametrize('base,levels', [(16, 2), (32, 3), (144, 3)])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_report_without_corrections(base, levels, precision):
    from bsam.device import DeviceBackend, DevHier
    on, off = (_opts(c, base, levels) for c in (True, False))
    on, off = ebOptions(dict(on, Precision=precision)), ebOptions(dict(off, Precision=precision))
    fl = flatten(build_hierarchy(vardc_problem(), on, OracleBackend()))
    dh = DevHier(DeviceBackend.get(0).ctx, fl, on)
    dh.solve_cycles(3)
    fl.Q[:] = dh.get(0, fl.Q.size)
    ref = {c: OracleHier(fl, o).residual() for c, o in ((True, on), (False, off))}
    assert (ref[True]['l2'] != ref[False]['l2']) == (base > 16)   # 16: the fine level covers the domain
    fresh = DevHier(DeviceBackend.get(0).ctx, fl, off)     # its first report
    got = [(False, fresh.residual()), (False, fresh.residual())]
    dh.set(0, 50.0 * fl.Q)                                 # a report with the corrections on, of larger values
    dh.residual()
    dh.set(0, fl.Q)
    for c, o in ((False, off), (True, on), (False, off)):
        dh.set_opts(o)
        got.append((c, dh.residual()))
    for c, r in got:
        assert r['ncell'] == ref[c]['ncell']
        for key in ('linf', 'fnorm', 'rel'):
            assert r[key] == ref[c][key], (c, key, r, ref[c])
        assert abs(r['l2'] - ref[c]['l2']) <= r['ncell'] * np.finfo(float).eps * ref[c]['l2']
