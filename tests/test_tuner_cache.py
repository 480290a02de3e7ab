"""The smoother's tuner keeps its choices in the context for later hierarchies.
What came first there -- a profile, a solve without post-smoothing (where the
tile form cannot run) -- does not decide for later solves, which take the form
a fresh context gives them; nor do options that a hierarchy had before.  The
levels here are of 1,000 to 6,000 cells, where six passes on tiles take 0.7 of
the time of chained ones or less, so every timing finds the same."""
import numpy as np
import pytest

from bsam import ebOptions
from bsam.flat import flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend
from cases import vardc_problem

pytestmark = pytest.mark.gpu


def _opts(precision, **kw):
    return ebOptions('BaseCells', 32, 'MaxLevels', 3, 'Indicator', 'fun', 'Verbose', 0, 'RelTol', 1e-10, 'Precision',
                     precision, 'TagFunction', lambda x, y: np.abs(x - y) < 0.15, *[v for kv in kw.items() for v in kv])


def _kernels(ctx, fl, o, monkeypatch, form=None):
    from bsam.device import DevHier
    if form:
        monkeypatch.setenv('BSAM_RELAX_N', form)
    dh = DevHier(ctx, fl, o)
    dh.solve_cycles(o.MaxVCycles + 2)
    monkeypatch.delenv('BSAM_RELAX_N', raising=False)
    return dh.kernels_per_vcycle()


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('first', ['profile', 'vcycle', 'no post-smoothing', 'same handle'])
def test_what_came_first_does_not_decide(precision, first, monkeypatch):
    from bsam.device import Context, DevHier
    monkeypatch.delenv('BSAM_RELAX_N', raising=False)
    o, bare = _opts(precision), _opts(precision, NPost=0)
    fl = flatten(build_hierarchy(vardc_problem(), o, OracleBackend()))
    fresh = _kernels(Context(0), fl, o, monkeypatch)
    assert fresh < _kernels(Context(0), fl, o, monkeypatch, '1')
    ctx = Context(0)
    dh = DevHier(ctx, fl, bare if first in ('no post-smoothing', 'same handle') else o)
    if first == 'profile':
        dh.profile(1)
    elif first == 'vcycle':
        dh.vcycle()
    else:
        dh.solve_cycles(o.MaxVCycles + 2)
    if first == 'same handle':
        dh.set_opts(o)
        dh.time_relax(2, 1)
        dh.solve_cycles(o.MaxVCycles + 2)
        assert dh.kernels_per_vcycle() == fresh
        dh.set_opts(bare)
        dh.solve_cycles(o.MaxVCycles + 2)
        assert dh.kernels_per_vcycle() == _kernels(ctx, fl, bare, monkeypatch)
    assert _kernels(ctx, fl, o, monkeypatch) == fresh
