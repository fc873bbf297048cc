"""SSIM's score is the mean of the map over the pooled pixels, whatever the values' size.  Four rows of a column
are summed in FP32 (three roundings of 2^-24 of sums that the values' magnitudes bound) and held to 2^-38; the rest
is exact but for FP64's own rounding, which 2^-50 of the mean covers."""
import numpy as np
import pytest

import iqm_b200

pytestmark = pytest.mark.gpu


# SSIM near 1e-4 (a dark picture against black and white noise) and near 0.5
@pytest.mark.parametrize("level", [3, 200])
@pytest.mark.parametrize("h,w", [(13, 15), (16, 16), (40, 130), (140, 300), (700, 900)])
def test_score_is_the_mean_of_the_map(rt, h, w, level):
    rng = np.random.default_rng(h * w + level)
    noise = rng.integers(0, 2, (h, w, 1)) * 255
    other = rng.integers(0, level + 1, (h, w, 1))
    if level > 100:
        other = (noise + other) // 2
    a, b = (np.concatenate([p.repeat(3, 2), np.full((h, w, 1), 255)], 2).astype(np.uint8) for p in (other, noise))
    s = iqm_b200.SSIM(rt)
    r = s.compute_metric(a, b)
    R = s.kernel_size // 2
    v = r.image_data[R:h - R + 1, R:w - R + 1].astype(np.float64)
    assert v.size == (h - 2 * R + 1) * (w - 2 * R + 1)
    tol = 3 * 2.0 ** -24 * np.abs(v).mean() + 2.0 ** -38 + 2.0 ** -50
    assert abs(r.mssim - v.mean()) <= tol, (r.mssim, v.mean(), tol)
    assert s.compute_batch([(a, b)])[0] == r.mssim
