"""The register-tiled FP32 scan with few keys (up to 8, and just above), one key around
the index size from which it takes such calls, rows ever closer to the queries (every
tile has candidates for every row), many equal distances within a run and across the
runs that share a query's limit.  Bar: bit-exact with the oracle."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


def rows(kind, n, m, d, rng):
    if kind == "ray":
        X = np.linspace(1.0, 0.0, n)[:, None] + 0.01 * rng.normal(size=(n, d))
        return X, 0.02 * rng.normal(size=(m, d))
    if kind == "dup":  # each row some 50 times, all over the index
        X = rng.normal(size=(max(1, n // 50), d))[rng.integers(0, max(1, n // 50), n)]
    else:  # few distinct distances, none zero
        X = rng.integers(-2, 3, size=(n, d))
    Q = X[rng.integers(0, n, m)] + (0.0 if kind == "dup" else 0.5)
    return X, Q


@pytest.mark.parametrize("kind", ["ray", "dup", "lattice"])
@pytest.mark.parametrize("n,m,d,k", [(4095, 70, 3, 1), (4096, 70, 3, 1), (4097, 3, 2, 1), (30000, 9, 5, 1),
                                     (1000, 65, 2, 2), (5000, 300, 17, 7), (40000, 2, 4, 8), (40000, 2, 4, 9),
                                     (1025, 2000, 2, 8), (20000, 5, 3, 40)])
@pytest.mark.parametrize("order,metric", [("arm", "sqeuclidean"), ("x86", "euclidean")])
def test_few_keys(gpu, oracle, kind, n, m, d, k, order, metric):
    rng = np.random.default_rng(n + m + d + k)
    X, Q = (a.astype(np.float32) for a in rows(kind, n, m, d, rng))
    gi, gd = SearchIndex(X, distance=metric, tree="linear", order=order, precision="fp32").knn(
        Q, k, exclude_self=False)
    ci, cd = oracle.knn(X, Q, k, metric=metric, order=order, threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(f32_bits(gd), f32_bits(cd))
