"""SSIM at the edges of its tiles (128 columns, strips of 8 to 128 rows that a launch chooses by its number
of images), against the FP64 oracle within the 1e-5 of tests/test_gpu_ssim.py; an image's score and map do
not depend on the images it is launched with."""
import numpy as np
import pytest

import iqm_b200
from iqm_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("ksize", [3, 11, 15])
@pytest.mark.parametrize("h,w", [(15, 127), (16, 128), (17, 129), (127, 16), (128, 131), (129, 257), (64, 255), (131, 15)])
def test_tile_edges_match_oracle(rt, o64, h, w, ksize):
    s = iqm_b200.SSIM(rt)
    s.kernel_size = ksize
    a, b = synth.grey_pair(h, w, config=0, pair=(h + w) % 9)
    assert abs(s.compute_metric(a, b).mssim - o64.ssim(a, b, kernel_size=ksize)) <= TOL


@pytest.mark.parametrize("h,w", [(70, 200), (300, 310)])
def test_score_does_not_depend_on_the_batch(rt, h, w):
    s = iqm_b200.SSIM(rt)
    a, b = synth.grey_pair(h, w, config=0, pair=3)
    alone = s.compute_metric(a, b)
    big = synth.grey_pair(1500, 1700, config=0, pair=4)
    got = s.compute_batch([big, (a, b)] + [big] * 3 + [(a, b)])  # launches of more than 296 tiles: other strips
    assert got[1] == alone.mssim and got[5] == alone.mssim
    assert np.array_equal(alone.image_data, s.compute_metric(a, b).image_data)
