"""M-SVD block distances on blocks whose singular values coincide or vanish: flat, rank one, rank two,
diagonal, a permutation, one pixel, checkerboards, and blocks of equal columns, next to noise.  Against
numpy's double-precision SVD of the grey blocks: an FP32 singular value of a block of norm s carries a few
units of 2^-24 s, at most 8 of them (backward error of the reflections and of the sweeps), and D adds up
16 of those in quadrature, so |D - D64| <= 8 * 2^-24 * 4 * max norm (2040) = 4e-3."""
import numpy as np
import pytest

import iqm_b200

pytestmark = pytest.mark.gpu


def _block(kind, rng):
    i, j = np.mgrid[0:8, 0:8]
    return {
        "zero": 0 * i, "flat": 0 * i + 200, "white": 0 * i + 255, "rows": 30 * i, "columns": 30 * j + 7,
        "rank two": 20 * i + 9 * j, "diagonal": 255 * (i == j), "scaled diagonal": (31 * i + 8) * (i == j),
        "antidiagonal": 90 * (i + j == 7), "permutation": 255 * (j == (3 * i + 1) % 8), "pixel": 255 * ((i == 5) & (j == 2)),
        "checker": 255 * ((i + j) % 2), "blocks": 100 * ((i // 4 + j // 4) % 2) + 20, "step": 255 * (j > i),
        "noise": rng.integers(0, 256, (8, 8)), "low noise": 128 + rng.integers(0, 2, (8, 8)),
        "flat plus pixel": 200 + 1 * ((i == 0) & (j == 7)), "two values": 3 + 250 * (i < 3),
    }[kind].astype(np.int64)


KINDS = ["zero", "flat", "white", "rows", "columns", "rank two", "diagonal", "scaled diagonal", "antidiagonal", "permutation",
         "pixel", "checker", "blocks", "step", "noise", "low noise", "flat plus pixel", "two values"]


@pytest.mark.parametrize("shift", [0, 1, 5, 11])
def test_degenerate_blocks_match_numpy(rt, shift):
    rng = np.random.default_rng(shift)
    bw, bh = len(KINDS), 4
    img = np.zeros((2, 8 * bh + 1, 8 * bw + 1), np.uint8)
    for y in range(bh):
        for x in range(bw):
            for k, s in ((0, 0), (1, shift * (y + 1))):
                img[k, 8 * y:8 * y + 8, 8 * x:8 * x + 8] = _block(KINDS[(x + s) % bw], rng)
    rgba = [np.dstack([g, g, g, np.full_like(g, 255)]) for g in img]  # grey: the weights sum to one
    r = iqm_b200.SVD(rt).compute_metric(rgba[0], rgba[1])
    blocks = [g[:8 * bh, :8 * bw].reshape(bh, 8, bw, 8).transpose(0, 2, 1, 3).astype(np.float64) for g in img]
    d = np.sqrt(((np.linalg.svd(blocks[0], compute_uv=False) - np.linalg.svd(blocks[1], compute_uv=False)) ** 2).sum(-1))
    tol = 8 * 2.0 ** -24 * 4 * 2040
    got = r.image_data.reshape(bh, bw).astype(np.float64) * (d.max() if d.max() else 1.0)
    if d.max() > 0:
        assert np.abs(got - d).max() <= 2 * tol, (np.abs(got - d).max(), tol)  # the map is D / max(D): twice
    want = np.abs(d - np.sort(d.reshape(-1))[d.size // 2]).mean()
    assert abs(r.msvd - want) <= 2 * tol
