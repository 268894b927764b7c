"""Pairwise distances in register tiles at the edges of a tile: 64 rows, 128
columns, strips of up to eight column tiles, one or two tile buffers (by d and
form), and the general kernel above 128 dimensions.  Bar: bit-exact with the
oracle."""
import numpy as np
import pytest

from conftest import threads
from fuel_gb300 import pairwise_distances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [
    (63, 8), (64, 16), (65, 15), (127, 31), (128, 32), (129, 33), (191, 60), (193, 64), (257, 87), (513, 88),
    (1025, 2), (700, 128), (3000, 9), (5200, 3), (140, 129),
])
@pytest.mark.parametrize("order,metric", [("arm", "sqeuclidean"), ("x86", "euclidean")])
@pytest.mark.parametrize("form", ["condensed", "square"])
def test_pairwise_tile_edges(gpu, oracle, n, d, order, metric, form):
    rng = np.random.default_rng(n + d)
    X = rng.normal(size=(n, d)).astype(np.float32)
    X[n // 2] = X[0]
    X[n // 3, 0] = np.inf
    g = pairwise_distances(X, distance=metric, form=form, order=order)
    c = oracle.pairwise_distances(X, metric, form, order=order, threads=threads())
    nan = np.isnan(c)
    assert np.array_equal(np.isnan(g), nan)
    np.testing.assert_array_equal(g[~nan].view(np.uint32), c[~nan].view(np.uint32))
