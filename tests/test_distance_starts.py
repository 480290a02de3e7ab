"""Starting values of bsam_polygon_dist2 that are not distances: a NaN start is
kept whatever the other points of its warp hold (no comparison with it is
true), and so is a negative one, which is below every distance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('scale', [1.0, 1e16])            # the FP32 search, and the one in FP64
@pytest.mark.parametrize('every', [1, 2, 31, 40])
def test_starts_that_are_kept(scale, every):
    from bsam.device import DeviceBackend, polygon_dist2
    rng = np.random.default_rng(every)
    t = 2 * np.pi * np.arange(92) / 91
    v = np.ascontiguousarray(np.stack([np.cos(t), 0.7 * np.sin(t)], axis=1) * scale)
    x, y = rng.normal(size=(2, 333)) * scale
    ctx = DeviceBackend.get(0).ctx
    want = polygon_dist2(ctx, v, x, y, np.full(x.size, 1e300))
    for odd in (np.nan, -1.0, -np.inf):
        start = np.full(x.size, 1e300)
        start[::every] = odd
        got = polygon_dist2(ctx, v, x, y, start.copy())
        np.testing.assert_array_equal(got, np.where(start == 1e300, want, start))
