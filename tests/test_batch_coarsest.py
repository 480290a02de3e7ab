"""The batch's coarsest solve (16 rows per block, columns in runs of 256, packed
trees): coarsest grids whose cells leave a remainder of rows and columns and
one of more than 256 cells.  Every instance of a batch ends where the oracle
ends with it alone, bit for bit, and in the mixed form where its own solve
ends."""
import numpy as np
import pytest

from bsam import ebOptions, ebProblem
from bsam.batch import merge_flats, split_field
from bsam.flat import FIELD_Q, flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend, OracleHier


def _parts(base, **kw):
    out = []
    for i in range(3):
        prob = ebProblem([0, 1, 0, 1], lambda x, y, i=i: 1 + 0.4 * np.sin((3 + i) * x) * np.cos(2 * y), 1.0,
                         lambda x, y, i=i: np.cos((4 + i) * x) * y,
                         {'west': ('dirichlet', 0.3), 'east': ('neumann', 0.1), 'south': ('neumann', 0),
                          'north': ('dirichlet', 0.1 * i)})
        args = dict(BaseCells=base, MaxLevels=1 + i, Indicator='fun', Verbose=0, RelTol=1e-10,
                    TagFunction=lambda x, y, L: (x - 0.5) ** 2 + (y - 0.4) ** 2 < 0.05)
        args.update(kw)
        o = ebOptions(*[v for kv in args.items() for v in kv])
        out.append((flatten(build_hierarchy(prob, o, OracleBackend())), o))
    return out


@pytest.mark.parametrize('base,n', [([22, 18], 99), ([30, 30], 225), ([34, 34], 289)])
def test_coarsest_sizes(base, n):
    assert [int(f.ncoarse) if hasattr(f, 'ncoarse') else f.bcRhs.size for f, _ in _parts(base)] == [n] * 3


@pytest.mark.gpu
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('base', [[22, 18], [30, 30], [34, 34]])
def test_batch_equals_solo(base, precision):
    from bsam.device import DeviceBackend, DevHier
    ctx = DeviceBackend.get(0).ctx
    parts = _parts(base, Precision=precision)
    o = parts[0][1]
    cap = int(o.MaxVCycles) + 2
    b = merge_flats([f for f, _ in parts])
    dh = DevHier(ctx, b, o)
    dh.solve_cycles(cap)
    Q = dh.get(0, b.Q.size)
    for i, (f, oi) in enumerate(parts):
        if precision == 'fp64':
            oh = OracleHier(f, oi)
            it, hist = oh.solve_cycles(cap)[:2]
            q = oh.Q
        else:
            one = DevHier(ctx, f, oi)
            it, hist = one.solve_cycles(cap)[:2]
            q = one.get(0, f.Q.size)
        itb, histb = dh.batch_result(i, cap)[:2]
        assert it == itb
        np.testing.assert_array_equal(hist, histb)
        np.testing.assert_array_equal(q, split_field(b, FIELD_Q, Q, i))
