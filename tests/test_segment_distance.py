"""bsam_polygon_dist2's search in FP32 with FP64 candidates gives the minimum
over every segment, bit for bit: polygons of one segment to several boxes,
remainders of the box sizes, points on vertices and edges, far away, at
scales FP32 holds and does not, not finite, with starting values above,
below and at the minimum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _brute(v, x, y, best):
    out = best.copy()
    with np.errstate(all='ignore'):
        for a, b in zip(v[:-1], v[1:]):
            e = b - a
            l2 = e[0] * e[0] + e[1] * e[1]
            rx, ry = x - a[0], y - a[1]
            t = (rx * e[0] + ry * e[1]) / l2
            t = np.fmax(0.0, np.fmin(1.0, t))
            qx, qy = rx - t * e[0], ry - t * e[1]
            out = np.fmin(out, qx * qx + qy * qy)
    return out


@pytest.mark.parametrize('segments', [1, 7, 8, 9, 63, 65, 517])
@pytest.mark.parametrize('scale', [1.0, 1e-14, 3e7, 1e16])
def test_minimum_over_all_segments(segments, scale):
    from bsam.device import DeviceBackend, polygon_dist2
    rng = np.random.default_rng(segments)
    t = 2 * np.pi * np.arange(segments + 1) / segments
    r = 1 + 0.4 * np.sin(5 * t) + 0.01 * rng.normal(size=t.size)
    v = np.stack([r * np.cos(t) + 0.3, r * np.sin(t)], axis=1)
    v[-1] = v[0] if segments > 1 else v[-1] + 0.5
    if segments > 20:
        v[5] = v[6]                                     # an empty segment
    v = np.ascontiguousarray(v * scale)
    x = np.concatenate([rng.normal(size=1500), np.repeat(np.linspace(-2, 2, 40), 40), v[:, 0] / scale,
                        0.5 * (v[1:, 0] + v[:-1, 0]) / scale, [1e6, -3e9, 0, 0, np.inf, np.nan]]) * scale
    y = np.concatenate([rng.normal(size=1500), np.tile(np.linspace(-2, 2, 40), 40), v[:, 1] / scale,
                        0.5 * (v[1:, 1] + v[:-1, 1]) / scale, [2e6, 1e9, 0, 1e-9, 1, 0]]) * scale
    exact = _brute(v, x, y, np.full(x.size, 1e300))
    for start in (np.full(x.size, 1e300), np.nextafter(exact, 0), exact * 1.0000001, exact + 0.1 * scale ** 2):
        want = _brute(v, x, y, start)
        got = polygon_dist2(DeviceBackend.get(0).ctx, v, x, y, start.copy())
        np.testing.assert_array_equal(got, want)
