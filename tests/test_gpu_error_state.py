"""A call that failed on the GPU's side leaves nothing behind that fails the next one."""
import numpy as np
import pytest

import iqm_b200
from iqm_b200 import synth

pytestmark = pytest.mark.gpu


def test_call_after_a_failed_allocation():
    import torch
    rt = iqm_b200.Runtime(0)
    f = iqm_b200.FSIM(rt)

    def dev(h, w):
        pair = synth.rgb_gain_pair(h, w, config=1, pair=2)
        bufs = [torch.from_numpy(np.ascontiguousarray(i).reshape(-1)).cuda() for i in pair]
        return pair, bufs, [(bufs[0].data_ptr(), bufs[1].data_ptr(), w, h, 4 * w)]

    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    for h, w in ((270, 300), (300, 270)):  # the lengths of the plane below, whose own tables are new
        keep = dev(h, w)
        f.compute_dev(keep[2], out.data_ptr())
    pair, bufs, items = dev(300, 300)
    rt.synchronize()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (4 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(iqm_b200.IQMError):
            f.compute_dev(items, out.data_ptr())
    finally:
        del filler
        torch.cuda.empty_cache()
    f.compute_dev(items, out.data_ptr())
    rt.synchronize()
    r = f.compute_metric(*pair)
    assert tuple(out.cpu().numpy()) == (r.fsim, r.fsimc)
    rt.close()
