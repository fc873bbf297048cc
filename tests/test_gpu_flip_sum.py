"""FLIP's score is the mean of the FP32 values that the map holds: their sum loses nothing that FP64 would
keep.  A value is held to 2^-48, FP64 adds a rounding of 2^-53 of the sum for each of at most four steps
(and numpy's pairwise sum a few more), so the two agree to 2^-48 + 16 * 2^-53 of the mean; fixed point of
2^-28 missed that by up to 2^-29 a value."""
import numpy as np
import pytest

import iqm_b200
from iqm_b200 import synth

pytestmark = pytest.mark.gpu


def _compare(rt, a, b, ppd):
    args = iqm_b200.FLIPArguments(float(ppd * 180.0 / np.pi * 0.6 / 0.7), 0.7, 0.6)
    r = iqm_b200.FLIP(rt).compute_metric(a, b, args, want_map=True)
    mean = r.image_data.astype(np.float64).mean()
    assert mean > 0.0
    assert abs(r.mean_flip - mean) <= 2.0 ** -48 + 16 * 2.0 ** -53 * mean, (r.mean_flip, mean)


# radii (CSF) 4, 8, 10 and 12, the last at one CTA an SM
@pytest.mark.parametrize("ppd", [28, 52, 67, 87])
@pytest.mark.parametrize("step", [1, 6])
def test_one_changed_pixel(rt, ppd, step):
    _, b = synth.rgb_blockquant_pair(121, 203, config=2, pair=1)
    a = b.copy()
    a[60, 100, 1] += step if a[60, 100, 1] < 128 else -step
    _compare(rt, a, b, ppd)


@pytest.mark.parametrize("h,w", [(1, 1), (13, 63), (61, 129), (200, 300), (1080, 1920)])
def test_noisy_picture(rt, h, w):
    a, b = synth.rgb_blockquant_pair(h, w, config=2, pair=5)
    if h * w == 1:
        a, b = np.full((1, 1, 4), 255, np.uint8), np.full((1, 1, 4), 250, np.uint8)
    _compare(rt, a, b, 52)
