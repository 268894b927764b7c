"""The register-tiled FP32 scan at the edges of its tiles: 128 index rows, 8
query rows per warp and 64 per block, 8-dimension groups, 32 keys per sorted
list and 256 per selection.  Bar: bit-exact with the oracle."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,d,k", [
    (1000, 1, 1, 1), (1023, 7, 7, 5), (1024, 8, 8, 32), (1025, 9, 9, 33), (1151, 63, 15, 31), (1152, 64, 16, 32),
    (1153, 65, 17, 100), (5000, 129, 24, 10), (5000, 3, 31, 256), (2049, 33, 33, 255), (1300, 70, 128, 64),
    (40000, 2, 16, 7), (3001, 300, 40, 3),
])
@pytest.mark.parametrize("order,metric", [("arm", "sqeuclidean"), ("x86", "euclidean")])
def test_tile_scan_edges(gpu, oracle, n, m, d, k, order, metric):
    rng = np.random.default_rng(n + m + d + k)
    X = rng.normal(size=(n, d)).astype(np.float32)
    X[n // 2:n // 2 + 40] = X[:40]  # duplicates: ties ordered by index
    Q = np.concatenate([X[:m // 2], rng.normal(size=(m - m // 2, d)).astype(np.float32)])
    index = SearchIndex(X, distance=metric, tree="linear", order=order, precision="fp32")
    gi, gd = index.knn(Q, k, exclude_self=False)
    ci, cd = oracle.knn(X, Q, k, metric=metric, order=order, threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(f32_bits(gd), f32_bits(cd))


def test_tile_scan_nonfinite(gpu, oracle):
    """NaN keys sort after +inf ones and fill rows that have too few others."""
    rng = np.random.default_rng(3)
    X = rng.normal(size=(1500, 5)).astype(np.float32)
    X[20:] = np.nan
    X[40:60] = np.inf
    gi, gd = SearchIndex(X, distance="sqeuclidean", tree="linear", order="arm", precision="fp32").knn(
        X[:10].copy(), 45, exclude_self=False)
    assert np.isfinite(gd[:, :20]).all() and np.isinf(gd[:, 20:40]).all() and np.isnan(gd[:, 40:]).all()
    assert (gi[:, 20:40] == np.arange(40, 60)).all()
    assert (gi[:, 40:] == np.arange(20, 25)).all()
