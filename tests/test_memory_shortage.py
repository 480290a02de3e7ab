"""Calls that a shortage of device memory refuses: the same call afterwards
gives what it gives without one."""
import numpy as np
import pytest

from bsam import ebOptions
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend, OracleHier
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


@pytest.mark.parametrize('form', ['6', None])
@pytest.mark.parametrize('tuned_before', [True, False])
def test_solve_whose_tile_tables_find_no_memory(form, tuned_before, monkeypatch):
    """The level runs its passes one by one (or, where the tuner's own copy is
    refused, the call fails), and the solves that follow are right."""
    from bsam.device import Context, DeviceError, DevHier
    if form:
        monkeypatch.setenv('BSAM_RELAX_N', form)
    else:
        monkeypatch.delenv('BSAM_RELAX_N', raising=False)
    fl, o = _flat()
    want = OracleHier(fl, o)
    it, hist, _, _ = want.solve_cycles(o.MaxVCycles + 2)
    ctx = Context(0)
    dh = DevHier(ctx, fl, o)
    if tuned_before:                       # the context knows the forms of these levels
        full = DevHier(ctx, fl, o)
        full.solve_cycles(o.MaxVCycles + 2)
    with no_device_memory():
        try:
            dh.solve_cycles(o.MaxVCycles + 2)
        except DeviceError:
            assert not form and not tuned_before
    for _ in range(2):
        dh.set(0, fl.Q)
        got = dh.solve_cycles(o.MaxVCycles + 2)
        assert got[0] == it
        np.testing.assert_array_equal(got[1], hist)
        np.testing.assert_array_equal(dh.get(0, fl.Q.size), want.Q)
    if form and tuned_before:
        assert dh.kernels_per_vcycle() > full.kernels_per_vcycle()
