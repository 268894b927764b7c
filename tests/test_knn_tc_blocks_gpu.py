"""The tensor-core kNN screen at the edges of its blocks and tiles: 128 query rows
per half and 256 per block, 128 index rows per tile, 64-column chunks (the query
operand in shared memory up to two, in TMEM beyond), 32 keys per sorted list.
Bar: bit-exact with the oracle."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,d,k,precision", [
    (129, 1, 32, 1, "split_bf16"), (1000, 127, 64, 32, "bf16"), (2048, 128, 65, 10, "fp16"),
    (2049, 129, 128, 24, "split_bf16"), (5000, 256, 129, 100, "fp16"), (3000, 257, 256, 14, "bf16"),
    (20000, 300, 48, 200, "fp16"), (4100, 513, 96, 13, "fp16"), (40000, 20, 33, 64, "split_bf16"),
])
@pytest.mark.parametrize("data", ["normal", "integer", "ray"])
def test_knn_tc_blocks(gpu, oracle, n, m, d, k, precision, data):
    rng = np.random.default_rng(n + m + d + k)
    if data == "normal":
        X = rng.normal(size=(n, d))
    elif data == "integer":
        X = rng.integers(0, 4, size=(n, d))  # the exact screen: many ties
    else:
        # ever closer to the queries with the index: every tile has new neighbours
        X = np.linspace(1.0, 0.0, n)[:, None] * np.ones(d) + 0.01 * rng.normal(size=(n, d))
    X = X.astype(np.float32)
    X[n // 2:n // 2 + 20] = X[:20]
    Q = np.concatenate([X[-(m // 2):] if m > 1 else X[:0],
                        (rng.integers(0, 4, size=(m - m // 2, d)) if data == "integer"
                         else 0.1 * rng.normal(size=(m - m // 2, d))).astype(np.float32)])
    gi, gd = SearchIndex(X, distance="sqeuclidean", tree="linear", order="arm", precision=precision).knn(
        Q, k, exclude_self=False)
    ci, cd = oracle.knn(X, Q, k, metric="sqeuclidean", order="arm", threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(f32_bits(gd), f32_bits(cd))


def test_knn_tc_nan_rows(gpu, oracle):
    """Rows with a NaN come after every other one and fill lists that need them."""
    rng = np.random.default_rng(1)
    X = rng.normal(size=(400, 40)).astype(np.float32)
    X[30:, 3] = np.nan
    gi, gd = SearchIndex(X, distance="sqeuclidean", tree="linear", order="arm", precision="split_bf16").knn(
        X[:9].copy(), 35, exclude_self=False)
    assert np.isfinite(gd[:, :30]).all() and np.isnan(gd[:, 30:]).all()
    assert (gi[:, 30:] == np.arange(30, 35)).all()
