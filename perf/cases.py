"""The measured cases: the work this framework's users have it do, through its public entry points.

Kinds:
  uniform   a solve on one grid without refinement (the plain multigrid solve)
  amr       a solve on a refined hierarchy, QC-ring or tree, either ghost interpolation, ragged grids too
  starfish  the diffuse-domain transmission problem refined around its interface (the benchmarked hierarchy)
  batch     many independent refined problems solved as one batch
  heat      a BDF2 run of the parabolic driver, regrids included
  check     what ebSolve and a regrid ask of a solved hierarchy: residual, mass balance, mean, refinement tags
  distance  the signed-distance minimum of the diffuse-domain sampling (points against a closed polygon)

A solve's pass is what a program with a resident hierarchy does for each new source: send the source and the
initial guess, run the solve, read the solution and the history.  The mesh and the coefficients stay; the source
comes from the seed.
"""
import functools
import os
import sys
import warnings

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, 'bsam-in-matlab_gb300'))

from bsam import ebOptions, ebProblem, build_hierarchy  # noqa: E402
from bsam.batch import merge_flats, split_field, join_field  # noqa: E402
from bsam.ddm import starfish_problem, starfish_tag  # noqa: E402
from bsam.device import (BSAM_FIELD_FTRUE, BSAM_FIELD_Q, DeferredBackend, DevHier, DeviceBackend,  # noqa: E402
                         polygon_dist2)
from bsam.flat import (LD_P0, PD_COFF, PD_ILO, PD_JLO, PD_LEVEL, PD_MX, PD_MY, PD_QOFF, FIELD_F,  # noqa: E402
                       flatten)
from bsam.instances import random_elliptic  # noqa: E402
from bsam.parabolic import ebpProblem, ebpSolve  # noqa: E402


def listed():
    return [
        # the smallest uniform solve of the test suite: two or three levels, all latency and launches
        {'name': 'uniform-32', 'kind': 'uniform', 'cx': 16, 'cy': 16, 'doublings': 1, 'lx': 1.0, 'neumann': False,
         'precision': 'fp64'},
        # the reference's recorded uniform 1024^2 solve: the largest single grid
        {'name': 'uniform-1024', 'kind': 'uniform', 'cx': 16, 'cy': 16, 'doublings': 6, 'lx': 1.0, 'neumann': False,
         'precision': 'fp64'},
        # the README example's shape: 64^2 base, three levels around a disc
        {'name': 'disc-64x3', 'kind': 'amr', 'cx': 16, 'cy': 16, 'doublings': 2, 'lx': 1.0, 'levels': 3,
         'shape': 'disc', 'tree': False, 'interp': 'qif', 'sweeps': 3, 'precision': 'fp64'},
        # tree hierarchy, linear ghost interpolation, two sweeps, non-square cells on a ragged grid
        {'name': 'tree-lif-ragged', 'kind': 'amr', 'cx': 15, 'cy': 11, 'doublings': 3, 'lx': 1.3, 'levels': 3,
         'shape': 'band', 'tree': True, 'interp': 'lif', 'sweeps': 2, 'precision': 'fp64'},
        # many small patches (the suite's scattered disks) on a ragged grid, in the mixed form
        {'name': 'scatter-ragged-mixed', 'kind': 'amr', 'cx': 13, 'cy': 9, 'doublings': 3, 'lx': 1.4, 'levels': 3,
         'shape': 'scatter', 'tree': False, 'interp': 'qif', 'sweeps': 3, 'precision': 'mixed'},
        # the benchmarked hierarchy: 543,384 stored cells on five refined levels
        {'name': 'starfish', 'kind': 'starfish', 'base': 64, 'levels': 5, 'precision': 'fp64'},
        {'name': 'starfish-mixed', 'kind': 'starfish', 'base': 64, 'levels': 5, 'precision': 'mixed'},
        # a batch of independent refined problems of mixed sizes, as the batched solver and the server run them
        {'name': 'batch-64', 'kind': 'batch', 'count': 64, 'first': 1000, 'precision': 'fp64'},
        {'name': 'batch-64-mixed', 'kind': 'batch', 'count': 64, 'first': 1000, 'precision': 'mixed'},
        # the README heat example's run: ten BDF2 steps, a regrid after five
        {'name': 'heat-64x3', 'kind': 'heat', 'base': 64, 'levels': 3, 'steps': 10, 'regrid': 5},
        # after a solve of the benchmarked hierarchy
        {'name': 'check-starfish', 'kind': 'check', 'base': 64, 'levels': 5},
        # one request's sample points (faces and centres of a refined level) against the 3000-point interface
        {'name': 'distance-300k', 'kind': 'distance', 'points': 300000, 'segments': 2999},
    ]


def draw(rng):
    kind = rng.choice(['uniform', 'uniform', 'amr', 'amr', 'amr', 'starfish', 'batch', 'heat', 'check', 'distance'])
    prec = rng.choice(['fp64', 'mixed'])
    if kind == 'uniform':
        return {'kind': kind, 'cx': rng.randint(9, 16), 'cy': rng.randint(9, 16), 'doublings': rng.randint(1, 6),
                'lx': round(rng.uniform(0.8, 1.6), 3), 'neumann': rng.random() < 0.4, 'precision': prec}
    if kind == 'amr':
        return {'kind': kind, 'cx': rng.randint(9, 16), 'cy': rng.randint(9, 16), 'doublings': rng.randint(1, 3),
                'lx': round(rng.uniform(0.8, 1.6), 3), 'levels': rng.randint(2, 4),
                'shape': rng.choice(['disc', 'band', 'scatter']), 'tree': rng.random() < 0.3,
                'interp': rng.choice(['qif', 'qif', 'lif']), 'sweeps': rng.choice([1, 2, 3, 3]), 'precision': prec}
    if kind == 'starfish':
        return {'kind': kind, 'base': rng.choice([24, 32, 40, 48, 56, 64]), 'levels': rng.randint(2, 4),
                'precision': prec}
    if kind == 'batch':
        return {'kind': kind, 'count': rng.randint(3, 32), 'first': rng.randint(2000, 9000), 'precision': prec}
    if kind == 'heat':
        return {'kind': kind, 'base': rng.choice([24, 32, 48, 64, 96]), 'levels': rng.randint(1, 3),
                'steps': rng.randint(4, 10), 'regrid': rng.randint(2, 5)}
    if kind == 'check':
        return {'kind': kind, 'base': rng.choice([24, 32, 40, 48, 56]), 'levels': rng.randint(2, 5)}
    return {'kind': kind, 'points': int(round(10 ** rng.uniform(2.5, 5.5))), 'segments': rng.randint(200, 2999)}


# ---- meshes and coefficients (built once per shape; the seed makes the sources) ----------------------------------

def _quiet(fn, *args, **kw):
    with warnings.catch_warnings():
        warnings.simplefilter('ignore')
        return fn(*args, **kw)


def _centres(fl, hs, dom):
    """x and y of every stored cell, in the order of the flat cell arrays."""
    x, y = np.empty(fl.F.size), np.empty(fl.F.size)
    for r in fl.patches:
        mx, my, o = int(r[PD_MX]), int(r[PD_MY]), int(r[PD_COFF])
        hx, hy = hs[int(r[PD_LEVEL]) - 1]
        xc = dom[0] + (np.arange(r[PD_ILO], r[PD_ILO] + mx) - 0.5) * hx
        yc = dom[2] + (np.arange(r[PD_JLO], r[PD_JLO] + my) - 0.5) * hy
        x[o:o + mx * my] = np.tile(xc, my)
        y[o:o + mx * my] = np.repeat(yc, mx)
    return x, y


def _tag(shape, lx):
    """Geometry-driven tags on [0, lx] x [0, 1]; L = 1 is the base level."""
    if shape == 'disc':
        return lambda X, Y, L: (X - 0.45 * lx) ** 2 + (Y - 0.55) ** 2 < (0.25 * 0.7 ** (L - 1)) ** 2
    if shape == 'band':
        return lambda X, Y, L: np.abs(X / lx - Y) < 0.16 * 0.5 ** (L - 1)
    r = np.random.RandomState(42).random_sample(48)
    px, py = lx * r[:24], r[24:]

    def scatter(X, Y, L):
        d = (np.asarray(X)[..., None] - px) ** 2 + (np.asarray(Y)[..., None] - py) ** 2
        return np.any(d < (0.035 * 0.6 ** (L - 1)) ** 2, axis=-1)
    return scatter


@functools.lru_cache(maxsize=3)
def _build(key):
    """(flat tables, options, cell centres) of one case's hierarchy, from the case's plain values."""
    c = dict(key)
    if c['kind'] in ('starfish', 'check'):
        prob, _, g = starfish_problem()
        o = ebOptions('BaseCells', c['base'], 'MaxLevels', c['levels'], 'Indicator', 'fun',
                      'TagFunction', starfish_tag(g, base=c['base']), 'TagBuffer', 2, 'RelTol', 1e-10, 'MaxVCycles', 100,
                      'Verbose', 0, 'Precision', c.get('precision', 'fp64'))
        H = _quiet(build_hierarchy, prob, o, DeferredBackend())
    elif c['kind'] == 'uniform':
        bc = ('neumann', 0.3) if c['neumann'] else ('dirichlet', 0.2)
        prob = ebProblem([0, c['lx'], 0, 1], 1.5, 2.0, lambda x, y: 10.0 + 0 * x, bc)
        o = ebOptions('BaseCells', [c['cx'] << c['doublings'], c['cy'] << c['doublings']], 'MaxLevels', 1,
                      'RelTol', 1e-10, 'Verbose', 0, 'Precision', c['precision'])
        H = build_hierarchy(prob, o, DeferredBackend())
    else:
        lx = c['lx']
        D = lambda x, y: 1 + 0.5 * np.sin(2 * np.pi * x / lx) * np.cos(np.pi * y)  # noqa: E731
        C = lambda x, y: 1 + x * y  # noqa: E731
        bc = {'west': ('dirichlet', 0.1), 'east': ('neumann', 0.2), 'south': ('dirichlet', lambda x, y: 0.3 * np.cos(x)),
              'north': ('neumann', 0)}
        prob = ebProblem([0, lx, 0, 1], D, C, lambda x, y: 30 * np.sin(3 * x + y), bc)
        o = ebOptions('BaseCells', [c['cx'] << c['doublings'], c['cy'] << c['doublings']], 'MaxLevels', c['levels'],
                      'Indicator', 'fun', 'TagFunction', _tag(c['shape'], lx), 'GhostInterp', c['interp'],
                      'NPre', c['sweeps'], 'NPost', c['sweeps'], 'RelTol', 1e-10, 'Verbose', 0,
                      'Precision', c['precision'])
        H = _quiet(build_hierarchy, prob, o, DeferredBackend(), tree=c['tree'])
    fl = flatten(H)
    return fl, o, _centres(fl, fl.hs, prob.domain)


@functools.lru_cache(maxsize=2)
def _build_batch(count, first):
    parts, xs, ys = [], [], []
    for i in range(count):
        prob, od = random_elliptic(first + i)
        r = np.random.RandomState(first + i).random_sample(4)
        ax, ay, rad = 0.25 + 0.5 * r[0], 0.25 + 0.5 * r[1], 0.1 + 0.15 * r[2]
        tag = lambda X, Y, L, ax=ax, ay=ay, rad=rad: (X - ax) ** 2 + (Y - ay) ** 2 < (rad * 0.6 ** (L - 1)) ** 2  # noqa: E731
        o = ebOptions(dict(od, Indicator='fun', TagFunction=tag))
        fl = flatten(_quiet(build_hierarchy, prob, o, DeferredBackend()))
        x, y = _centres(fl, fl.hs, prob.domain)
        parts.append(fl)
        xs.append(x)
        ys.append(y)
    bfl = merge_flats(parts)
    o = ebOptions('RelTol', 1e-10, 'Verbose', 0)
    return bfl, o, (join_field(bfl, FIELD_F, xs), join_field(bfl, FIELD_F, ys))


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != 'name'))


def _smooth(rng, x, y, modes=4):
    """A smooth random field: a few Fourier modes of wavelengths down to a quarter of the unit."""
    out = np.zeros(x.size)
    for _ in range(modes):
        kx, ky, ph, a = rng.uniform(-4, 4), rng.uniform(-4, 4), rng.uniform(0, 6.28), rng.normal()
        out += a * np.cos(2 * np.pi * (kx * x + ky * y) + ph)
    return out


def _polygon(segments):
    """Vertices of the closed five-armed star (the last repeats the first)."""
    t = 2 * np.pi * np.arange(segments + 1) / segments
    t[-1] = 0.0
    r = 0.9 * (1.2 + 0.7 * np.sin(5 * t))
    return np.ascontiguousarray(np.stack([r * np.cos(t), r * np.sin(t)], axis=1))


# ---- the interface ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case['kind']
    if kind == 'distance':
        # sample points as a level's patches give them: runs of a grid in a band around the interface
        verts = _polygon(case['segments'])
        n = case['points']
        h = 4.0 / 1024
        at = rng.integers(0, case['segments'], -(-n // 64))
        bx = np.round((verts[at, 0] + rng.normal(0, 0.1, at.size)) / h)
        by = np.round((verts[at, 1] + rng.normal(0, 0.1, at.size)) / h)
        x = ((bx[:, None] + np.arange(64) % 16 + 0.5) * h).ravel()[:n].copy()
        y = ((by[:, None] + np.arange(64) // 16 + 0.5) * h).ravel()[:n].copy()
        # the host's starting candidate: the vertex at the point's polar angle
        j = np.floor((np.arctan2(y, x) % (2 * np.pi)) / (2 * np.pi) * case['segments']).astype(np.int64)
        best = (x - verts[j, 0]) ** 2 + (y - verts[j, 1]) ** 2
        return {'kind': kind, 'ctx': DeviceBackend.get(0).ctx, 'verts': verts, 'x': x, 'y': y, 'best': best}
    if kind == 'heat':
        cx, cy, w = rng.uniform(0.3, 0.7), rng.uniform(0.3, 0.7), rng.uniform(0.05, 0.09)
        u0 = lambda x, y: (1 + 0.2 * np.cos(2 * np.pi * x) * np.cos(2 * np.pi * y)  # noqa: E731
                           + 0.8 * np.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * w ** 2)))
        prob = ebpProblem([0, 1, 0, 1], 0.05, 0, 0, ('neumann', 0), u0)
        args = ('Scheme', 'bdf2', 'Dt', 0.002, 'TFinal', 0.002 * case['steps'], 'BaseCells', case['base'],
                'MaxLevels', case['levels'], 'RegridEvery', case['regrid'], 'StepVerbose', 0,
                'Indicator', 'fun', 'TagFunction', _tag('disc', 1.0), 'RelTol', 1e-9)
        return {'kind': kind, 'prob': prob, 'args': args}
    if kind == 'batch':
        fl, o, (x, y) = _build_batch(case['count'], case['first'])
        o = ebOptions(dict(o, Precision=case['precision']))
    else:
        fl, o, (x, y) = _build(_key(case))
    dh = DevHier(DeviceBackend.get(0).ctx, fl, o)
    dh.setup_levels()
    f = fl.FTrue * (1 + 0.3 * _smooth(rng, x, y)) + _smooth(rng, x, y)
    state = {'kind': kind, 'dh': dh, 'fl': fl, 'cap': int(o.MaxVCycles) + 2, 'f': f,
             'q0': dh.get(BSAM_FIELD_Q, fl.Q.size)}
    if kind == 'check':
        L = fl.levels[fl.nlev - 1]
        state['n'] = (int(L[0]), int(L[1]))
        dh.set(BSAM_FIELD_FTRUE, f)
        q = state['q0'].copy()
        for r in fl.patches:
            mx, my, o_, c = int(r[PD_MX]), int(r[PD_MY]), int(r[PD_QOFF]), int(r[PD_COFF])
            v = q[o_:o_ + (mx + 2) * (my + 2)].reshape((mx + 2, my + 2), order='F')
            s = slice(c, c + mx * my)
            v[1:-1, 1:-1] = (np.cos(2 * x[s] + y[s]) * (1 + 0.2 * np.sin(rng.uniform(1, 9) * x[s]))).reshape((mx, my), order='F')
        dh.set(BSAM_FIELD_Q, q)
        for k in range(1, fl.nlev + 1):
            dh.fill(k)
        state['q0'] = dh.get(BSAM_FIELD_Q, fl.Q.size)
    return state


def run(state):
    kind = state['kind']
    if kind == 'distance':
        best = state['best'].copy()
        return {'dist2': polygon_dist2(state['ctx'], state['verts'], state['x'], state['y'], best)}
    if kind == 'heat':
        sol = _quiet(ebpSolve, state['prob'], *state['args'])
        return {'Q': flatten(sol['H']).Q, 'mass': sol['mass'], 'cycles': sol['cycles'], 'relres': sol['relres']}
    dh, fl = state['dh'], state['fl']
    if kind == 'check':
        dh.set(BSAM_FIELD_Q, state['q0'])
        r = dh.residual()
        m = dh.mass_check()
        mean, area = dh.composite_mean()
        tags = dh.tag_level(fl.nlev, 'ulap', 1e-3, 2, *state['n'])
        return {'residual': np.array([r['linf'], r['l2'], r['fnorm'], r['rel']]), 'cells': r['ncell'],
                'mass': np.array([m['lhs'], m['flux']]), 'mean': np.array([mean, area]), 'tags': tags}
    dh.set(BSAM_FIELD_FTRUE, state['f'])
    dh.set(BSAM_FIELD_Q, state['q0'])
    it, hist, rel, vis = dh.solve_cycles(state['cap'])
    Q = dh.get(BSAM_FIELD_Q, fl.Q.size)
    if kind == 'batch':
        its = [dh.batch_result(i, state['cap'])[0] for i in range(fl.ninst)]
        return {'Q': Q, 'vcycles': np.array(its), 'visible': vis}
    if kind == 'uniform':
        r = fl.patches[int(fl.levels[fl.nlev - 1][LD_P0])]
        mx, my, o = int(r[PD_MX]), int(r[PD_MY]), int(r[PD_QOFF])
        u = Q[o:o + (mx + 2) * (my + 2)].reshape((mx + 2, my + 2), order='F')[1:-1, 1:-1]
        return {'u': u, 'Q': Q, 'vcycles': it, 'visible': vis}
    return {'Q': Q, 'vcycles': it, 'visible': vis}


def work(case):
    kind = case['kind']
    if kind == 'distance':
        n = case['points']
        # at least the segments next to the nearest one have to be evaluated: a dozen operations each
        return {'bytes': 32.0 * n + 16.0 * case['segments'], 'flops': 16 * 12.0 * n}
    if kind == 'heat':
        # a step on the base grid at the least: source, coefficients and solution once, three V-cycles
        n = case['base'] ** 2 * (4 / 3)
        return {'bytes': 48.0 * n * case['steps'], 'flops': 3 * 100.0 * n * case['steps']}
    if kind == 'batch':
        n = float(_build_batch(case['count'], case['first'])[0].F.size)
    else:
        n = float(_build(_key(case))[0].F.size)
    if kind == 'check':
        return {'bytes': 41.0 * n, 'flops': 20.0 * n}
    sweeps = 2 * case.get('sweeps', 3)
    # source, three coefficients, guess and solution once; about ten V-cycles of `2 sweeps` relaxations
    # (9 operations a cell), the residual twice, restriction and prolongation
    return {'bytes': 48.0 * n, 'flops': 10 * (9.0 * sweeps + 50.0) * n}


def exact(case, seed):
    kind = case['kind']
    if kind == 'distance':
        s = prepare(dict(case), seed)
        dev = 'cuda' if torch.cuda.is_available() else 'cpu'
        v = torch.from_numpy(s['verts']).to(dev)
        a, e = v[:-1], v[1:] - v[:-1]
        l2 = (e * e).sum(1)
        out = torch.from_numpy(s['best']).to(dev)
        pts = torch.stack([torch.from_numpy(s['x']), torch.from_numpy(s['y'])], 1).to(dev)
        for i in range(0, pts.shape[0], 16384):
            d = pts[i:i + 16384, None, :] - a[None]
            t = ((d * e).sum(2) / l2).clamp(0, 1)
            q = ((d - t[..., None] * e) ** 2).sum(2).min(1).values
            out[i:i + 16384] = torch.minimum(out[i:i + 16384], q)
        return {'dist2': out.cpu().numpy()}
    if kind == 'uniform':
        # -div(D grad u) + C u = f with constant D and C: the one-dimensional operators, made symmetric by a
        # diagonal scaling of their end rows, diagonalise the whole one
        s = prepare(dict(case), seed)
        fl, D, C = s['fl'], 1.5, 2.0
        r = fl.patches[int(fl.levels[fl.nlev - 1][LD_P0])]
        mx, my, o = int(r[PD_MX]), int(r[PD_MY]), int(r[PD_COFF])
        f = s['f'][o:o + mx * my].reshape((mx, my), order='F').copy()
        parts = []
        for n, length in ((mx, case['lx']), (my, 1.0)):
            h = length / n
            A = 2 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1)
            b = np.zeros(n)
            if case['neumann']:      # ghost = u + h g
                A[0, 0] = A[-1, -1] = 1
                b[0] = b[-1] = 0.3 * h
                w = np.ones(n)
            else:                    # ghost = 8/3 g - 2 u1 + u2 / 3
                A[0, 0] = A[-1, -1] = 4
                A[0, 1] = A[-1, -2] = -4 / 3
                b[0] = b[-1] = 8 / 3 * 0.2
                w = np.ones(n)
                w[0] = w[-1] = np.sqrt(0.75)
            S = w[:, None] * (A * (D / h ** 2)) / w[None, :]
            lam, V = np.linalg.eigh((S + S.T) / 2)
            parts.append((lam, V, w, b * (D / h ** 2)))
        (lx, Vx, wx, bx), (ly, Vy, wy, by) = parts
        g = f + bx[:, None] + by[None, :]
        g = wx[:, None] * g * wy[None, :]
        u = Vx @ ((Vx.T @ g @ Vy) / (lx[:, None] + ly[None, :] + C)) @ Vy.T
        return {'u': u / wx[:, None] / wy[None, :], 'Q': None, 'vcycles': None, 'visible': None}
    if kind == 'check':
        s = prepare(dict(case), seed)
        fl, tot, area = s['fl'], [], 0.0
        for r in fl.patches:
            if int(r[PD_LEVEL]) < fl.rootIdx:
                continue
            mx, my, o, c = int(r[PD_MX]), int(r[PD_MY]), int(r[PD_QOFF]), int(r[PD_COFF])
            da = float(np.prod(fl.hs[int(r[PD_LEVEL]) - 1]))
            v = s['q0'][o:o + (mx + 2) * (my + 2)].reshape((mx + 2, my + 2), order='F')[1:-1, 1:-1].ravel(order='F')
            vis = fl.covered[c:c + mx * my] == 0
            tot.append(float(np.sum(v[vis].astype(np.longdouble))) * da)
            area += np.count_nonzero(vis) * da
        return {'residual': None, 'cells': None, 'mass': None, 'mean': np.array([sum(tot) / area, area]),
                'tags': None}
    return None
