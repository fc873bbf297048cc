"""SSIM of identical images is 1 in every pixel and as a score, not 1 give or take a rounding."""
import numpy as np
import pytest

import iqm_b200
from iqm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ksize", [3, 11, 15])
@pytest.mark.parametrize("h,w", [(16, 16), (64, 64), (97, 211), (300, 500), (1080, 1920)])
def test_identical_images_score_one(rt, h, w, ksize):
    s = iqm_b200.SSIM(rt)
    s.kernel_size = ksize
    images = [synth.grey_pair(h, w, config=0, pair=1)[0], synth.rgb_gain_pair(h, w, config=1, pair=2)[1],
              np.random.default_rng(h).integers(0, 256, (h, w, 4), dtype=np.uint8), np.full((h, w, 4), 77, np.uint8)]
    for a in images:
        r = s.compute_metric(a, a.copy())
        assert r.mssim == 1.0 and np.all(r.image_data == 1.0)
    assert np.all(s.compute_batch([(a, a.copy()) for a in images]) == 1.0)
