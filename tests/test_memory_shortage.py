"""Calls that a shortage of device memory refuses: the same call afterwards
gives what it gives without one."""
import numpy as np
import pytest

from bsam import ebOptions
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend
from cases import vardc_problem
from shortage import no_device_memory

pytestmark = pytest.mark.gpu


def _flat(**kw):
    o = ebOptions('BaseCells', 32, 'MaxLevels', 3, 'Indicator', 'fun', 'Verbose', 0, 'RelTol', 1e-10, 'TagFunction',
                  lambda x, y: np.abs(x - y) < 0.15, *[v for kv in kw.items() for v in kv])
    return flatten(build_hierarchy(vardc_problem(), o, OracleBackend())), o


def test_mass_check_after_a_refused_one():
    from bsam.device import DeviceBackend, DeviceError, DevHier
    fl, o = _flat()
    ctx = DeviceBackend.get(0).ctx
    a, b = DevHier(ctx, fl, o), DevHier(ctx, fl, o)
    a.solve_cycles(o.MaxVCycles + 2)
    b.solve_cycles(o.MaxVCycles + 2)
    want = a.mass_check()
    for _ in range(2):
        with no_device_memory():
            with pytest.raises(DeviceError):
                b.mass_check()
    assert b.mass_check() == want
    assert want['flux'] != 0
