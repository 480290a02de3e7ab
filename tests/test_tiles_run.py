"""Forced on (BSAM_RELAX_N=6), the tile form runs: on every level of the
hierarchies whose results are compared elsewhere, in both precisions, in a
batch with frozen instances, with other sweeps; it steps aside, and says so,
without post-smoothing and on levels of 131,072 cells.  What it gives equals the
chained passes, and the tuned choice either, bit for bit."""
import numpy as np
import pytest

from bsam import ebOptions
from bsam.batch import merge_flats
from test_relax_tiles import BAND, CASES, DISC, DOTS, _build

pytestmark = pytest.mark.gpu


def _run(fl, o, stops=()):
    from bsam.device import Context, DevHier
    dh = DevHier(Context(0), fl, o)
    for s in stops:
        dh.set_stop(*s)
    dh.solve_cycles(o.MaxVCycles + 2)
    return dh, dh.get(0, fl.Q.size)


def _check(fl, o, expect, monkeypatch, stops=()):
    p = int(o.Precision == 'mixed')
    out = {}
    for form in ('1', '6', None):
        if form:
            monkeypatch.setenv('BSAM_RELAX_N', form)
        else:
            monkeypatch.delenv('BSAM_RELAX_N')
        dh, Q = _run(fl, o, stops)
        out[form] = Q
        tiles = dh.relax_tiles(p)
        assert np.all(dh.relax_tiles(1 - p) == -1)
        if form == '1':
            assert not tiles.any()
        elif form:
            assert tiles.tolist() == expect, (tiles, expect)
            assert np.all(dh.relax_tuning(p)[np.asarray(expect) == 1] == 1)
        else:
            assert np.all(tiles <= np.asarray(expect))
    np.testing.assert_array_equal(out['6'], out['1'])
    np.testing.assert_array_equal(out[None], out['1'])


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('case', CASES, ids=[str(i) for i in range(len(CASES))])
def test_one_hierarchy(case, precision, monkeypatch):
    fl, o = _build(Precision=precision, **case)
    cells = [int(L[5] - L[4]) for L in fl.levels]
    expect = [int(k > 0 and n < 131072 and o.NPost > 0) for k, n in enumerate(cells)]
    _check(fl, o, expect, monkeypatch)


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_batch(precision, monkeypatch):
    built = [_build([32, 32], lv, tag, Precision=precision) for lv, tag in ((3, DISC), (2, BAND), (1, DISC), (3, DOTS))]
    b = merge_flats([fl for fl, _ in built])
    _check(b, built[0][1], [0] + [1] * (b.nlev - 1), monkeypatch, ((1, 3, 1e-10), (3, 25, 1e-5)))
