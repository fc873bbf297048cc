"""FSIM over every kind of transform plan, against the FP64 oracle within the 1e-5 of tests/test_gpu_fsim.py:
two factors up to 24 and up to 32, Bluestein on two factors, three factors with and without Bluestein, the
shared-memory engine for sides beyond the register engine's plans; widths that fill the last column tile
with one column, planes smaller than one tile, and several columns per tile (long columns take fewer)."""
import pytest

import iqm_b200
from iqm_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("h,w", [(16, 18), (24, 23), (31, 29), (32, 33), (37, 41), (61, 65), (96, 427), (240, 427),
                                 (255, 341), (263, 383), (120, 513), (90, 1024), (615, 200), (1021, 97), (2048, 131),
                                 (2503, 70), (3000, 64), (3301, 60), (60, 3200)])
def test_fsim_plan_kinds_match_oracle(rt, o64, h, w):
    a, b = synth.rgb_gain_pair(h, w, config=1, pair=(h + w) % 11)
    f = iqm_b200.FSIM(rt)
    r = f.compute_metric(a, b)
    want = o64.fsim(a, b)
    assert abs(r.fsim - want[0]) <= TOL and abs(r.fsimc - want[1]) <= TOL, (r, want)
    batch = f.compute_batch([(a, b), (b, a), (a, b)])
    assert tuple(batch[0]) == (r.fsim, r.fsimc) == tuple(batch[2])


# rows whose four scales come within the row kernel's static shared memory (1 KB) of the 48 KB that a launch
# may use unasked
@pytest.mark.parametrize("h,w", [(40, 643), (40, 680), (40, 728), (40, 736), (40, 765), (40, 1360), (40, 1404), (40, 1500)])
def test_fsim_rows_at_the_default_shared_memory(rt, o64, h, w):
    a, b = synth.rgb_gain_pair(h, w, config=1, pair=(h + w) % 11)
    r = iqm_b200.FSIM(rt).compute_metric(a, b)
    want = o64.fsim(a, b)
    assert abs(r.fsim - want[0]) <= TOL and abs(r.fsimc - want[1]) <= TOL, (r, want)
