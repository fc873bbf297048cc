"""FLIP's fused kernel over the filter radii it is compiled for and the first beyond them, at sizes around
its tiles (64 columns, strips of whole steps of 14 rows), against the FP64 oracle within the 1e-5 of
tests/test_gpu_flip.py; a picture's score and map do not depend on the pictures it is launched with."""
import numpy as np
import pytest

import iqm_b200
from iqm_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _args(ppd):
    return iqm_b200.FLIPArguments(float(ppd * 180.0 / np.pi * 0.6 / 0.7), 0.7, 0.6)


# radii (CSF) 1, 3, 4 .. 14, and 15 on the two-pass kernels
@pytest.mark.parametrize("ppd", [6, 20, 28, 36, 43, 50, 58, 65, 72, 80, 87, 95, 102, 107])
@pytest.mark.parametrize("h,w", [(13, 63), (61, 129)])
def test_radii_match_oracle(rt, o64, ppd, h, w):
    a, b = synth.rgb_blockquant_pair(h, w, config=2, pair=ppd % 7)
    f = iqm_b200.FLIP(rt)
    r = f.compute_metric(a, b, _args(ppd), want_map=True)
    assert abs(r.mean_flip - o64.flip(a, b, ppd=f.ppd(_args(ppd)))) <= TOL
    assert abs(r.image_data.astype(np.float64).mean() - r.mean_flip) <= 1e-6
    assert f.compute_metric(b, b, _args(ppd)).mean_flip == 0.0


@pytest.mark.parametrize("h,w", [(1, 1), (2, 130), (150, 3), (84, 64), (85, 65), (300, 200)])
def test_score_does_not_depend_on_the_batch(rt, o64, h, w):
    f = iqm_b200.FLIP(rt)
    a, b = synth.rgb_blockquant_pair(h, w, config=2, pair=3)
    alone = f.compute_metric(a, b, want_map=True)
    assert abs(alone.mean_flip - o64.flip(a, b, ppd=f.ppd())) <= TOL
    big = synth.rgb_blockquant_pair(1300, 1500, config=2, pair=4)
    got = f.compute_batch([big, (a, b)] + [big] * 3 + [(a, b)])
    assert got[1] == alone.mean_flip and got[5] == alone.mean_flip
