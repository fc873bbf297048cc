"""FSIM batches whose chunks hold more pairs than a grid's z dimension takes images (two each, at most 65535)."""
import numpy as np
import pytest

import iqm_b200
from iqm_b200 import synth

pytestmark = pytest.mark.gpu


# 33000 pairs fit a chunk's budget in one piece; 40000 leave a second chunk
@pytest.mark.parametrize("n", [33000, 40000])
def test_more_pairs_than_a_grid_takes(rt, n):
    import torch
    a, b = synth.rgb_gain_pair(8, 8, config=1, pair=3)
    da, db = (torch.from_numpy(np.ascontiguousarray(i).reshape(-1)).cuda() for i in (a, b))
    items = [(da.data_ptr(), db.data_ptr(), 8, 8, 32), (db.data_ptr(), da.data_ptr(), 8, 8, 32)] * (n // 2)
    out = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    f = iqm_b200.FSIM(rt)
    f.compute_dev(items, out.data_ptr())
    rt.synchronize()
    got = out.cpu().numpy().reshape(-1, 2)
    want = [(r.fsim, r.fsimc) for r in (f.compute_metric(a, b), f.compute_metric(b, a))]
    assert np.array_equal(got, np.tile(want, (n // 2, 1)))
