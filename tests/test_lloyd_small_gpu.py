"""Small Lloyd problems, a pass in one kernel (up to 2560 means) or assigned and
committed by one: one to 32 lanes per point, centre counts around them, up to 256
centres and 64 dimensions, sums in the block's shared memory and not, just below
and above the sizes from which the tiled scan takes over.  Bar: labels, centres and
iterations equal to the exact-mean oracle's."""
import numpy as np
import pytest

from fuel_gb300 import kmeans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [
    (1, 1, 1), (2, 3, 2), (31, 2, 3), (33, 7, 31), (255, 8, 4), (256, 9, 32), (257, 15, 33), (1000, 31, 64),
    (300, 64, 255), (700, 5, 256), (600, 4, 257), (9000, 3, 17), (40000, 4, 5), (25806, 31, 40), (25807, 31, 40),
    (300, 64, 40), (300, 64, 41), (6097, 41, 64), (6098, 41, 64), (30000, 2, 2), (5000, 20, 60),
])
@pytest.mark.parametrize("order", ["arm", "x86"])
def test_small_lloyd_matches_oracle(gpu, oracle, n, d, k, order):
    rng = np.random.default_rng(n + d + k)
    X = rng.normal(size=(n, d)) + 4 * rng.integers(0, 4, size=(n, 1))
    X = (np.round(X * 2) / 2 if n % 2 else X).astype(np.float32)  # ties
    init = X[rng.permutation(n)[:k]].copy()
    init[-1] = init[0]  # the first of two equal centres wins
    iters = 4 if n * k * d > 10**6 else 8
    got = kmeans(X, k=k, variant="lloyd", init=init, max_iter=iters, order=order, precision="fp32")
    c, lab, it, _ = oracle.lloyd_exact(X, k, init, max_iter=iters, order=order)
    np.testing.assert_array_equal(got.labels, lab)
    np.testing.assert_array_equal(got.centers.view(np.uint32), c.view(np.uint32))
    assert got.n_iter == it
