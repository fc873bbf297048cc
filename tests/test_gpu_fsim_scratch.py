"""FSIM's transform scratch: one budget for all plane sizes in flight, smaller chunks where the GPU has little
memory left, and chunks whose images fit a grid's z dimension.  How a batch is cut changes no bit of a score."""
import numpy as np
import pytest

import iqm_b200
from iqm_b200 import synth

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _device_pairs(pairs, repeat):
    import torch
    keep = [tuple(torch.from_numpy(np.ascontiguousarray(i).reshape(-1)).cuda() for i in p) for p in pairs]
    items = [(a.data_ptr(), b.data_ptr(), p[0].shape[1], p[0].shape[0], p[0].shape[1] * 4) for (a, b), p in zip(keep, pairs)]
    return keep, items * repeat


def _scores(rt, items):
    import torch
    out = torch.zeros(2 * len(items), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    iqm_b200.FSIM(rt).compute_dev(items, out.data_ptr())
    rt.synchronize()
    return out.cpu().numpy().reshape(-1, 2)


def _fill_all_but(mb):
    """Memory that leaves `mb` MB of the GPU free."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - mb * MB, dtype=torch.uint8, device="cuda")


def _plane_bytes(n):  # what a pair takes apart from the chunks' planes: 144 bytes a point, with tiles' padding
    return 150 * n


@pytest.fixture
def fresh():
    import torch
    r = iqm_b200.Runtime(0)
    yield r
    r.close()
    torch.cuda.empty_cache()


def test_small_memory_takes_smaller_chunks(fresh):
    pairs = [synth.rgb_gain_pair(270, 480, config=1, pair=i) for i in range(4)]
    keep, items = _device_pairs(pairs, 8)
    want = [_scores(fresh, items[i:i + 1])[0] for i in range(4)]
    # 640 MB of chunks do not fit beside the planes, the 80 MB that two pairs take do
    filler = _fill_all_but(32 * _plane_bytes(270 * 480) // MB + 150)
    try:
        got = _scores(fresh, items)
        plan_scores = np.zeros(0)
        assert np.array_equal(got, np.tile(want, (8, 1)))
    finally:
        del filler


def test_small_memory_plan_is_built_and_replayed(fresh):
    import torch
    pairs = [synth.rgb_gain_pair(h, w, config=1, pair=i) for i, (w, h) in enumerate([(480, 270), (300, 256), (270, 270)])]
    keep, items = _device_pairs(pairs, 8)
    want = [_scores(fresh, items[i:i + 1])[0] for i in range(3)]
    out = torch.zeros(2 * len(items), dtype=torch.float64, device="cuda")
    # three sizes in turn: their planes together (they run side by side while memory lasts) and 150 MB
    filler = _fill_all_but(8 * _plane_bytes(270 * 480 + 300 * 256 + 270 * 270) // MB + 150)
    try:
        plan = iqm_b200.BatchPlan(fresh, iqm_b200.METRIC_FSIM, items, out.data_ptr(), autotune=True)
        try:
            plan.run()
            fresh.synchronize()
            got = out.cpu().numpy().reshape(-1, 2)
        finally:
            plan.close()
    finally:
        del filler
    assert np.array_equal(got, np.tile(want, (8, 1)))


@pytest.mark.parametrize("autotune", [False, True])
def test_many_sizes_share_the_budget(fresh, autotune):
    import torch
    sizes = [(256 + 4 * i, 256) for i in range(8)]
    pairs = [synth.rgb_gain_pair(h, w, config=1, pair=i) for i, (w, h) in enumerate(sizes)]
    keep, items = _device_pairs(pairs, 20)
    want = [_scores(fresh, items[i:i + 1])[0] for i in range(8)]
    out = torch.zeros(2 * len(items), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = iqm_b200.BatchPlan(fresh, iqm_b200.METRIC_FSIM, items, out.data_ptr(), autotune=autotune)
    try:
        took = before - torch.cuda.mem_get_info()[0]
        plan.run()
        fresh.synchronize()
        got = out.cpu().numpy().reshape(-1, 2)
    finally:
        plan.close()
    assert np.array_equal(got, np.tile(want, (20, 1)))
    # the planes, a budget of at most 1280 MB, and 100 MB for the graph
    assert took <= 20 * sum(_plane_bytes(w * h) for w, h in sizes) + (1280 if autotune else 640) * MB + 100 * MB, took


@pytest.mark.parametrize("mb", range(60, 400, 20))
def test_scratch_leaves_room_for_streams_and_graphs(fresh, mb):
    import torch
    pairs = [synth.rgb_gain_pair(h, w, config=1, pair=i) for i, (w, h) in enumerate([(480, 270), (300, 256), (270, 270)])]
    keep, items = _device_pairs(pairs, 8)
    want = [_scores(fresh, items[i:i + 1])[0] for i in range(3)]
    out = torch.zeros(2 * len(items), dtype=torch.float64, device="cuda")
    filler = _fill_all_but(8 * _plane_bytes(270 * 480 + 300 * 256 + 270 * 270) // MB + 100 + mb)
    try:
        plan = iqm_b200.BatchPlan(fresh, iqm_b200.METRIC_FSIM, items, out.data_ptr(), autotune=False)
        try:
            plan.run()
            fresh.synchronize()
            got = out.cpu().numpy().reshape(-1, 2)
        finally:
            plan.close()
    finally:
        del filler
    assert np.array_equal(got, np.tile(want, (8, 1)))


@pytest.mark.parametrize("w,h", [(300, 260), (20, 9), (7, 400), (2, 4096), (4096, 3)])
def test_planes_hold_the_spectra(fresh, w, h):
    """A pair takes 30 floats a point of its plane beside a chunk's, what the planes alone take, apart from planes
    narrower than a tile of 8 columns; and planes of any width hold them (the score is a lone pair's)."""
    import torch
    pairs = [synth.rgb_gain_pair(h, w, config=1, pair=i) for i in range(3)]
    count = max(3, int(3e9 / (120 * w * h)) // 3 * 3) if w >= 8 else 99
    keep, items = _device_pairs(pairs, min(count, 30000) // 3)
    want = [_scores(fresh, items[i:i + 1])[0] for i in range(3)]
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    got = _scores(fresh, items)
    took = before - torch.cuda.mem_get_info()[0]
    assert np.array_equal(got, np.tile(want, (len(items) // 3, 1)))
    if w >= 8:  # 4% for the pooling sums of a tile, the descriptors and what is left of a tile of 256 points
        assert took <= len(items) * (125 * w * h + 600) + 700 * MB, took
