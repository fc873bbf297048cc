"""M-SVD block distances on blocks whose bidiagonal form splits (an exact 0 on the diagonal and beside it:
a black first row and column, sparse pixels, block diagonal content) or has values close together (noisy
diagonals, some of which run out of sweeps and take the Jacobi path).  Against numpy's double-precision SVD
of the grey blocks: an FP32 singular value of a block of norm s carries at most 8 units of 2^-24 s, and D
adds up 16 of those in quadrature, so |D - D64| <= 8 * 2^-24 * 2040 * 4 = 3.9e-3; the map is D / max D in
FP32, two roundings of 2^-24 more."""
import numpy as np
import pytest

import iqm_b200

pytestmark = pytest.mark.gpu
TOL = 8 * 2.0 ** -24 * 2040 * 4
I, J = np.mgrid[0:8, 0:8]


def _sparse(rng, n):
    rank = rng.random((n, 64)).argsort(1).argsort(1).reshape(n, 8, 8)
    return rank < rng.integers(1, 65, (n, 1, 1))


def _blocks(kind, n, rng):
    noise, level = rng.integers(0, 256, (n, 8, 8)), rng.integers(1, 256, (n, 1, 1))
    if kind.startswith("border"):  # black border of k rows and l columns
        k, l = int(kind[-2]), int(kind[-1])
        return (noise if kind.startswith("border noise") else level) * ((I >= k) & (J >= l))
    if kind == "patch":
        y, x = rng.integers(0, 8, (2, n, 1, 1))
        return noise * ((I >= y) & (I < rng.integers(y + 1, 9)) & (J >= x) & (J < rng.integers(x + 1, 9)))
    if kind == "corner of four":
        return np.where((I >= 6) & (J >= 6), np.array([[200, 100], [50, 220]])[I % 2, J % 2], 0) + 0 * noise
    if kind == "sparse noise":
        return noise * _sparse(rng, n)
    if kind == "sparse level":
        return level * _sparse(rng, n)
    if kind == "sparse on white":
        return 255 - rng.integers(1, 30, (n, 1, 1)) * _sparse(rng, n)
    if kind == "two level":
        return np.where(rng.random((n, 8, 8)) < rng.random((n, 1, 1)), level, rng.integers(0, 256, (n, 1, 1)))
    if kind == "black and white":
        return 255 * (rng.random((n, 8, 8)) < rng.random((n, 1, 1)))
    if kind == "block diagonal":
        q = rng.integers(1, 8, (n, 1, 1))
        return np.where((I < q) & (J < q), np.where(rng.random((n, 1, 1)) < 0.5, level, noise), noise) * ((I < q) == (J < q))
    if kind == "bidiagonal":
        return noise * ((I == J) | (J == I + 1)) * (rng.random((n, 8, 8)) < 0.7)
    if kind == "permutation":
        return noise * np.eye(8, dtype=int)[rng.random((n, 8)).argsort(1)]
    if kind == "noisy diagonal":
        return np.clip(noise * (I == J) + rng.integers(0, 1 + rng.integers(1, 12, (n, 1, 1)), (n, 8, 8)), 0, 255)
    if kind == "rank two":
        f = [rng.integers(0, 12, s) for s in ((n, 8, 1), (n, 1, 8), (n, 8, 1), (n, 1, 8))]
        return np.clip(f[0] * f[1] + f[2] * f[3], 0, 255)
    t, p = 6.3 * rng.random((n, 1, 1)), 8 * (rng.random((n, 1, 1)) - 0.5)
    assert kind == "edge on black"
    return level * (np.cos(t) * (I - 3.5) + np.sin(t) * (J - 3.5) > p)


KINDS = (["border %s %d%d" % (c, k, l) for c in ("noise", "flat") for k, l in ((1, 1), (1, 2), (2, 1), (3, 3), (4, 6), (6, 4), (6, 6))]
         + ["patch", "corner of four", "sparse noise", "sparse level", "sparse on white", "two level", "black and white",
            "block diagonal", "bidiagonal", "permutation", "noisy diagonal", "rank two", "edge on black"])


def _check(rt, a, b, side):
    def picture(blocks):  # a last row and column of pixels, so that every block is computed
        g = np.zeros((8 * side + 1, 8 * side + 1), np.uint8)
        g[:-1, :-1] = blocks.reshape(side, side, 8, 8).transpose(0, 2, 1, 3).reshape(8 * side, 8 * side)
        return np.dstack([g, g, g, np.full_like(g, 255)])

    r = iqm_b200.SVD(rt).compute_metric(picture(a), picture(b))
    sa, sb = (np.linalg.svd(v.astype(np.float64), compute_uv=False) for v in (a, b))
    d = np.sqrt(((sa - sb) ** 2).sum(1))
    got = r.image_data.reshape(-1).astype(np.float64) * d.max()
    bad = np.abs(got - d) > 2 * TOL + 2.0 ** -23 * d.max()  # D and max D are both off by up to TOL
    assert not bad.any(), (bad.sum(), np.abs(got - d).max())
    want = np.abs(d - np.sort(d)[d.size // 2]).mean()
    assert abs(r.msvd - want) <= 2 * TOL, (r.msvd, want)


@pytest.mark.parametrize("kind", KINDS)
def test_block_distances_match_numpy(rt, kind):
    rng, side = np.random.default_rng(KINDS.index(kind)), 32
    n = side * side
    _check(rt, _blocks(kind, n, rng), _blocks("sparse noise", n, rng), side)


def test_blocks_that_run_out_of_sweeps(rt):
    rng, side = np.random.default_rng(1), 320
    n = side * side
    _check(rt, _blocks("noisy diagonal", n, rng), _blocks("noisy diagonal", n, rng), side)
