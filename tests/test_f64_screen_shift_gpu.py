"""float64 kNN through the FP32 screen on values that the shift by the index's first
row turns into integers although they are none: differences of the last bits, and
values far below the first row's, vanish in the shifted copies.  Such rows are not
integer data, and the screen's list is not final for them.  Bar: bit-exact with the
oracle."""
import numpy as np
import pytest

from conftest import threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu

SEVEN = 0.07 * 100  # 7.000000000000001: 100 - SEVEN rounds to 93, as 100 - 7 does


def rows(kind, n, d, rng):
    """(index, queries): the index's later rows are the nearest, its earlier ones tie with them after the shift."""
    half = n // 2
    if kind == "percent":
        X = np.full((n, d), 7.0)
        X[0], X[half:] = 100.0, SEVEN
        return X, np.array([SEVEN, 7.0, 100.0])[:, None] * np.ones(d)
    if kind == "tiny":
        X = np.full((n, d), 1e-20)
        X[0], X[half:] = 1.0, 0.0
        return X, np.array([0.0, 1e-20, 1.0, 2e-20])[:, None] * np.ones(d)
    # integers, their last bits changed at random
    X = rng.integers(1, 4, size=(n, d)).astype(np.float64)
    X[0] = 64.0
    Q = X[half:half + 40].copy()
    for a in (X[1:], Q):
        up = rng.integers(0, 3, size=a.shape)
        a[up == 1] = np.nextafter(a[up == 1], 100.0)
        a[up == 2] = np.nextafter(a[up == 2], -100.0)
    return X, Q


@pytest.mark.parametrize("kind", ["percent", "tiny", "noise"])
@pytest.mark.parametrize("d", [1, 3, 9])
@pytest.mark.parametrize("order,metric", [("arm", "sqeuclidean"), ("x86", "euclidean"), ("x86", "sqeuclidean"),
                                          ("arm", "euclidean")])
def test_shifted_values_that_round_to_integers(gpu, oracle, kind, d, order, metric):
    X, Q = rows(kind, 20000, d, np.random.default_rng(d))
    gi, gd = SearchIndex(X, distance=metric, tree="linear", order=order).knn(Q, 5, exclude_self=False)
    ci, cd = oracle.knn(X, Q, 5, metric=metric, order=order, threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(gd.view(np.uint64), cd.view(np.uint64))
