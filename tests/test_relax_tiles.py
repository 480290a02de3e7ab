"""The smoother's tile form (tile.cuh): every colour pass of a relaxation in
one launch on tiles of the level, halo updates repeated, the level moving
between two copies of the solution.  Forced on every level that can take it
(BSAM_RELAX_N=6), a solve equals the oracle bit for bit (FP64) or the
chained passes (mixed): QC-ring and tree hierarchies, both ghost
interpolations, sides of every kind, patches narrower than a tile and no
multiple of one, one to four sweeps on either side (four: several launches a
relaxation; no post-smoothing: the form steps aside), over-relaxation, a
batch with frozen instances, and an eager V-cycle from ghosts that are out of
step with the cells."""
import numpy as np
import pytest

from bsam import ebOptions, ebProblem
from bsam.batch import merge_flats, split_field
from bsam.flat import FIELD_Q, flatten
from bsam.solve import build_hierarchy
from bsam_oracle import OracleBackend, OracleHier

pytestmark = pytest.mark.gpu

DISC = lambda x, y, L: (x - 0.45) ** 2 + (y - 0.55) ** 2 < 0.09 / L ** 2
BAND = lambda x, y, L: np.abs(x - y) < 0.2 / L
DOTS = lambda x, y, L: (np.abs(np.sin(11 * x)) > 0.9) & (np.abs(np.cos(9 * y)) > 0.85)
MIXED_BC = {'west': ('dirichlet', 0.3), 'east': ('neumann', 0.1), 'south': ('neumann', 0), 'north': ('dirichlet', 0)}


def _build(base, levels, tag, lx=1.0, tree=False, bc=('dirichlet', 0.2), **opts):
    D = lambda x, y: 1 + 0.5 * np.sin(3 * x) * np.cos(2 * y)
    prob = ebProblem([0, lx, 0, 1], D, 1.0, lambda x, y: np.cos(4 * x) * y + 3, bc)
    o = ebOptions('BaseCells', base, 'MaxLevels', levels, 'Indicator', 'fun', 'TagFunction', tag, 'Verbose', 0,
                  'RelTol', 1e-10, 'MaxVCycles', 25, *[v for kv in opts.items() for v in kv])
    return flatten(build_hierarchy(prob, o, OracleBackend(), tree=tree)), o


def _solve(fl, o, steps=2):
    from bsam.device import DeviceBackend, DevHier
    dh = DevHier(DeviceBackend.get(0).ctx, fl, o)
    out = []
    for _ in range(steps):       # the first solve runs step by step, later ones as one graph
        it, hist, rel, _ = dh.solve_cycles(o.MaxVCycles + 2)
        out.append((it, hist, dh.get(0, fl.Q.size), dh.get(3, fl.QC.size), dh.get(1, fl.F.size)))
    return dh, out


def _equal(a, b):
    for x, y in zip(a, b):
        assert x[0] == y[0]
        for u, v in zip(x[1:], y[1:]):
            np.testing.assert_array_equal(u, v)


CASES = [
    dict(base=[32, 32], levels=3, tag=DISC),
    dict(base=[44, 36], levels=3, tag=BAND, lx=1.3, bc=MIXED_BC),
    dict(base=[64, 48], levels=2, tag=DOTS, bc=('neumann', 0)),
    dict(base=[32, 32], levels=3, tag=DISC, GhostInterp='lif', NPre=2, NPost=1, bc=MIXED_BC),
    dict(base=[64, 64], levels=3, tag=BAND, tree=True, NPre=1, NPost=3),
    dict(base=[40, 24], levels=2, tag=DISC, NPre=4, NPost=4, Omega=1.1),
    dict(base=[32, 32], levels=2, tag=DISC, NPre=3, NPost=0),
    dict(base=[256, 200], levels=2, tag=BAND, lx=1.2),
]


@pytest.mark.parametrize('case', CASES, ids=[str(i) for i in range(len(CASES))])
def test_tiles_equal_the_oracle(case, monkeypatch):
    fl, o = _build(**case)
    oh = OracleHier(fl, o)
    it, hist, rel, _ = oh.solve_cycles(o.MaxVCycles + 2)
    monkeypatch.setenv('BSAM_RELAX_N', '1')
    chained, ref = _solve(fl, o)
    monkeypatch.setenv('BSAM_RELAX_N', '6')
    dh, got = _solve(fl, o)
    assert got[0][0] == it
    np.testing.assert_array_equal(got[0][1], hist)
    np.testing.assert_array_equal(got[0][2], oh.Q)
    _equal(got, ref)
    fewer = dh.kernels_per_vcycle() < chained.kernels_per_vcycle()
    assert fewer == (o.NPost > 0 and o.NPre + o.NPost > 2)


@pytest.mark.parametrize('case', CASES[:6], ids=[str(i) for i in range(6)])
def test_tiles_equal_chained_passes_in_the_mixed_form(case, monkeypatch):
    fl, o = _build(Precision='mixed', **case)
    monkeypatch.setenv('BSAM_RELAX_N', '1')
    _, ref = _solve(fl, o)
    monkeypatch.setenv('BSAM_RELAX_N', '6')
    _, got = _solve(fl, o)
    _equal(got, ref)


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_batch_with_frozen_instances(precision, monkeypatch):
    from bsam.device import DeviceBackend, DevHier
    built = [_build([32, 32], lv, tag, Precision=precision) for lv, tag in ((3, DISC), (2, BAND), (1, DISC), (3, DOTS))]
    o = built[0][1]
    b = merge_flats([fl for fl, _ in built])
    out = {}
    for form in ('1', '6'):
        monkeypatch.setenv('BSAM_RELAX_N', form)
        bh = DevHier(DeviceBackend.get(0).ctx, b, o)
        bh.set_stop(1, 3, 1e-10)
        bh.set_stop(3, 25, 1e-5)
        bh.solve_cycles(o.MaxVCycles + 2)
        out[form] = ([bh.batch_result(i, 30)[:2] for i in range(4)], bh.get(0, b.Q.size))
    for (ia, ha), (ib, hb) in zip(out['1'][0], out['6'][0]):
        assert ia == ib
        np.testing.assert_array_equal(ha, hb)
    np.testing.assert_array_equal(out['1'][1], out['6'][1])
    assert len({r[0] for r in out['6'][0]}) > 1


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_eager_vcycle_from_unfilled_ghosts(precision, monkeypatch):
    from bsam.device import DeviceBackend, DevHier
    fl, o = _build([32, 32], 3, DOTS, Precision=precision)
    q = np.random.default_rng(5).normal(size=fl.Q.size)      # ghosts and cells unrelated
    out = []
    for form in ('1', '6'):
        monkeypatch.setenv('BSAM_RELAX_N', form)
        dh = DevHier(DeviceBackend.get(0).ctx, fl, o)
        dh.solve_cycles(o.MaxVCycles + 2)                    # picks the form
        dh.set(0, q)
        dh.vcycle()
        out.append(dh.get(0, fl.Q.size))
    np.testing.assert_array_equal(out[0], out[1])
