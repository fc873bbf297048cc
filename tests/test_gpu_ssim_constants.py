"""SSIM over the constants that it accepts, against the FP64 oracle within the 1e-5 of tests/test_gpu_ssim.py:
large ones, whose squares and their product have to stay in FP32's range (a product of k1 and k2 up to about
9e18), one large and one small, and none at all on pictures without flat areas."""
import numpy as np
import pytest

import iqm_b200
from iqm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k1,k2", [(2e4, 2e4), (1e6, 1e3), (3e8, 3e8), (1e15, 0.03), (0.01, 1e15), (3.0, 1e-6), (1e-8, 1e-8), (0.0, 0.0)])
@pytest.mark.parametrize("ksize", [3, 11])
def test_constants_match_oracle(rt, o64, k1, k2, ksize):
    s = iqm_b200.SSIM(rt)
    s.k_1, s.k_2, s.kernel_size = k1, k2, ksize
    a, b = synth.grey_pair(90, 140, config=0, pair=3)
    want, want_map = o64.ssim(a, b, kernel_size=ksize, k1=k1, k2=k2, want_map=True)
    r = s.compute_metric(a, b)
    assert np.isfinite(r.image_data).all()
    assert abs(r.mssim - want) <= 1e-5, (r.mssim, want)
    if k1 >= 1e3 and k2 >= 1e3:  # the constants swamp the pictures
        assert abs(want - 1.0) <= 1e-5
