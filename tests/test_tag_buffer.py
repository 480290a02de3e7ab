"""The tag buffer on the device, by words of four cells (rows of a multiple of
four, buffers up to four) and by cells, against the host's dilation and
erosion."""
import numpy as np
import pytest

from bsam import ebOptions, ebProblem
from bsam.flat import PD_MX, PD_MY, PD_QOFF, flatten
from bsam.solve import build_hierarchy
from bsam.tagcluster import _dilate, _erode8
from bsam_oracle import OracleBackend


@pytest.mark.gpu
@pytest.mark.parametrize('base,levels', [([32, 32], 2), ([18, 22], 1), ([18, 24], 1), ([10, 18], 3), ([8, 4], 1)])
@pytest.mark.parametrize('buffer', [0, 1, 2, 3, 4, 5])
def test_tag_mask_of_any_buffer(base, levels, buffer):
    from bsam.device import DeviceBackend, DevHier
    prob = ebProblem([0, 1, 0, 1], 1.0, 1.0, lambda x, y: np.cos(9 * x) * np.sin(7 * y) * (x > 0.4),
                     ('dirichlet', 0))
    o = ebOptions('BaseCells', base, 'MaxLevels', levels, 'Indicator', 'fun', 'Verbose', 0,
                  'TagFunction', lambda x, y, L: abs(x - y) < 0.25)
    H = build_hierarchy(prob, o, OracleBackend())
    fl = flatten(H)
    rng = np.random.default_rng(buffer)
    Q = rng.normal(size=fl.Q.size) * (rng.random(fl.Q.size) < 0.05)
    dh = DevHier(DeviceBackend.get(0).ctx, fl, o)
    dh.set(0, Q)
    lev = H.lev[H.nlev]
    n0, n1 = (int(v) for v in lev.n)
    T, C = np.zeros((n0, n1), bool), np.zeros((n0, n1), bool)
    thr = 0.5
    first = len(fl.patches) - lev.np
    for p in range(lev.np):
        r = fl.patches[first + p]
        mx, my, q0 = int(r[PD_MX]), int(r[PD_MY]), int(r[PD_QOFF])
        q = Q[q0:q0 + (mx + 2) * (my + 2)].reshape((mx + 2, my + 2), order='F')
        sx = (q[2:, 1:-1] - 2 * q[1:-1, 1:-1]) + q[:-2, 1:-1]
        sy = (q[1:-1, 2:] - 2 * q[1:-1, 1:-1]) + q[1:-1, :-2]
        b = [int(v) for v in lev.box[p]]
        T[b[0] - 1:b[1], b[2] - 1:b[3]] |= np.sqrt(sx ** 2 + sy ** 2) > thr
        C[b[0] - 1:b[1], b[2] - 1:b[3]] = True
    want = _dilate(T, buffer) & _erode8(C)
    np.testing.assert_array_equal(want, dh.tag_level(H.nlev, 'ulap', thr, buffer, n0, n1))
    assert T.any()
