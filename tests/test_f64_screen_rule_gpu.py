"""float64 kNN on both sides of the line between the FP64 scan and its FP32 screen: up
to 32 candidates and more, few queries and many.  Bar: bit-exact with the oracle."""
import numpy as np
import pytest

from conftest import threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["normal", "integer", "offset", "ties"])
@pytest.mark.parametrize("n,d,k,ms", [
    (16500, 3, 29, (70, 71, 72, 73, 150)), (2500, 128, 200, (214, 215, 216, 217, 230)), (1200, 7, 28, (33, 60, 400)),
    (13000, 2, 1, (1, 2)), (9000, 33, 60, (69, 70, 71, 90)), (30000, 3, 40, (1, 4, 5)),
])
@pytest.mark.parametrize("order,metric", [("arm", "euclidean"), ("x86", "sqeuclidean")])
def test_both_sides_of_the_line(gpu, oracle, kind, n, d, k, ms, order, metric):
    rng = np.random.default_rng(n + d)
    X = rng.normal(size=(n, d))
    if kind == "integer":
        X = rng.integers(-2, 3, size=(n, d)).astype(np.float64)
    elif kind == "offset":
        X += 1e6
    elif kind == "ties":
        X = X[rng.integers(0, n // 50, n)]
    Q = X[rng.integers(0, n, max(ms))]
    ix = SearchIndex(X, distance=metric, tree="linear", order=order)
    ci, cd = oracle.knn(X, Q, k, metric=metric, order=order, threads=threads())
    for m in ms:
        gi, gd = ix.knn(Q[:m].copy(), k, exclude_self=False)
        assert np.array_equal(gi, ci[:m])
        assert np.array_equal(gd.view(np.uint64), cd[:m].view(np.uint64))
