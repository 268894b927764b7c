"""Small Lloyd problems around the lines from which the tiled scan takes over, by the
rows' alignment: multiples of 128, 64 and 16 bytes, and rows past what L1 holds.  Bar:
labels, centres and iterations equal to the exact-mean oracle's."""
import numpy as np
import pytest

from fuel_gb300 import kmeans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [
    (1953, 64, 32), (1954, 64, 32), (4464, 32, 28), (4465, 32, 28), (325, 32, 192), (326, 32, 192), (318, 32, 196),
    (319, 32, 196), (10416, 16, 60), (10417, 16, 60), (6720, 48, 31), (6721, 48, 31), (20408, 56, 14), (20409, 56, 14),
    (100000, 36, 4), (100001, 36, 5), (100001, 36, 4),
])
@pytest.mark.parametrize("order", ["arm", "x86"])
def test_both_sides_of_the_lines(gpu, oracle, n, d, k, order):
    rng = np.random.default_rng(n + d + k)
    X = rng.normal(size=(n, d)) + 4 * rng.integers(0, 4, size=(n, 1))
    X = (np.round(X * 2) / 2 if n % 2 else X).astype(np.float32)  # ties
    init = X[rng.permutation(n)[:k]].copy()
    got = kmeans(X, k=k, variant="lloyd", init=init, max_iter=4, order=order, precision="fp32")
    c, lab, it, _ = oracle.lloyd_exact(X, k, init, max_iter=4, order=order)
    np.testing.assert_array_equal(got.labels, lab)
    np.testing.assert_array_equal(got.centers.view(np.uint32), c.view(np.uint32))
    assert got.n_iter == it
