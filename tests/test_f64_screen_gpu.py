"""float64 kNN through the FP32 screen (16 384 index rows and up, or enough
pairs): bit-exact with the oracle where the proof certifies a query, where the
screen is exact (integers), and where it cannot certify (ties, offsets that
f32 cannot hold, non-finite values)."""
import numpy as np
import pytest

from conftest import threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


def data(kind, n, d, rng):
    X = rng.normal(size=(n, d))
    if kind == "normal":
        return X
    if kind == "integer":
        return rng.integers(-3, 4, size=(n, d)).astype(np.float64)
    if kind == "clusters":  # nearest distances far below one f32 step of the coordinates
        return rng.normal(size=(20, d))[rng.integers(0, 20, n)] * 100.0 + 1e-7 * X
    if kind == "offset":
        return 1e9 + X
    X[n // 2] = 1e300  # outside the f32 range: no screen
    return X


@pytest.mark.parametrize("kind", ["normal", "integer", "clusters", "offset", "wide"])
@pytest.mark.parametrize("n,m,d,k,order,metric", [
    (16384, 9, 16, 28, "arm", "euclidean"), (16500, 70, 3, 29, "x86", "sqeuclidean"),
    (2000, 600, 9, 10, "arm", "sqeuclidean"), (1500, 64, 128, 200, "x86", "euclidean"),
])
def test_f64_screen_matches_oracle(gpu, oracle, kind, n, m, d, k, order, metric):
    rng = np.random.default_rng(n + m + d)
    X = data(kind, n, d, rng)
    Q = np.concatenate([X[:m // 2], data(kind, n, d, rng)[:m - m // 2]])
    ix = SearchIndex(X, distance=metric, tree="linear", order=order)
    gi, gd = ix.knn(Q, k, exclude_self=False)
    ci, cd = oracle.knn(X, Q, k, metric=metric, order=order, threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(gd.view(np.uint64), cd.view(np.uint64))


def test_f64_screen_self_join_excludes(gpu, oracle):
    X = np.random.default_rng(5).normal(size=(1700, 4))
    X[1000:1100] = X[:100]
    ix = SearchIndex(X, distance="euclidean", tree="linear", order="arm")
    gi, gd = ix.knn(X, 6)  # the index's own array: linear exclude rule
    ci, cd = oracle.knn(X, X, 6, metric="euclidean", order="arm", exclude="linear", threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(gd.view(np.uint64), cd.view(np.uint64))
