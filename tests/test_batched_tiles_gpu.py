"""Batched k-means at the edges of its kernels: 128-row items (problems of one or
a few items, so nearly every item starts a problem), 16- and 32-column screens,
rows of 32 to 64 dimensions with and without whole 8-value chunks, and centres
taken two at a time (odd and even k) for 2 and 8 dimensions.  Bar: centres, labels
and iterations equal to each problem's own call, bit for bit."""
import numpy as np
import pytest

from fuel_gb300 import kmeans, kmeans_batched

pytestmark = pytest.mark.gpu


def problem(rng, n, d, k):
    X = rng.normal(size=(n, d)) + 4 * rng.integers(0, 3, size=(n, 1))
    X = np.round(X * 8) / 8 if n % 3 == 0 else X  # ties
    X = X.astype(np.float32)
    return X, X[rng.permutation(n)[:k]].copy()


def check(probs, order, max_iter):
    got = kmeans_batched(probs, max_iter=max_iter, order=order, fixed_iters=True)
    for (X, init), g in zip(probs, got):
        ref = kmeans(X, k=init.shape[0], variant="lloyd", init=init, max_iter=max_iter, order=order, fixed_iters=True)
        np.testing.assert_array_equal(g.centers.view(np.uint32), ref.centers.view(np.uint32))
        np.testing.assert_array_equal(g.labels, ref.labels)
        assert g.n_iter == ref.n_iter


@pytest.mark.parametrize("order", ["arm", "x86"])
@pytest.mark.parametrize("d", [2, 8, 32, 33, 36, 40, 63, 64])
def test_batched_tile_edges(gpu, order, d):
    rng = np.random.default_rng(d)
    sizes = [(1, 1), (127, 2), (128, 3), (129, 15), (255, 16), (257, 17), (300, 31), (500, 32), (700, 33), (300, 64),
             (300, 65), (400, 127), (600, 255), (600, 256), (3000, 5)]
    check([problem(rng, n, d, k) for n, k in sizes], order, 4)


def test_batched_many_small_problems(gpu):
    """Several hundred problems of one to four items: each CTA changes problem at nearly every item."""
    rng = np.random.default_rng(1)
    probs = [problem(rng, int(rng.integers(20, 450)), int(rng.choice([2, 8, 32, 64])), int(rng.integers(1, 20)))
             for _ in range(700)]
    check(probs, "arm", 5)
