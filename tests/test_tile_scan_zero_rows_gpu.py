"""The register-tiled FP32 scan with index rows of zeros, which the padding rows of a
query block (zeros too) keep, several runs per block and query counts off the
blocks' 8 and 64 rows.  Bar: bit-exact with the oracle."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 65, 127, 129, 191])
@pytest.mark.parametrize("k", [1, 5, 40])
@pytest.mark.parametrize("d", [4, 32, 100])
def test_zero_rows(gpu, oracle, m, k, d):
    rng = np.random.default_rng(m + k + d)
    X = rng.normal(size=(40000, d)).astype(np.float32)
    X[rng.random(40000) < 0.1] = 0.0
    Q = rng.normal(size=(m, d)).astype(np.float32)
    Q[m // 2] = 0.0
    gi, gd = SearchIndex(X, distance="sqeuclidean", tree="linear", order="arm", precision="fp32").knn(
        Q, k, exclude_self=False)
    ci, cd = oracle.knn(X, Q, k, metric="sqeuclidean", order="arm", threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(f32_bits(gd), f32_bits(cd))


def test_zero_rows_f64(gpu, oracle):
    """The float64 screen's copies of the first row are zeros."""
    rng = np.random.default_rng(3)
    X = rng.normal(size=(30000, 5))
    X[rng.random(30000) < 0.1] = X[0]
    Q = np.concatenate([X[:3], rng.normal(size=(62, 5))])
    gi, gd = SearchIndex(X, distance="euclidean", tree="linear", order="arm").knn(Q, 6, exclude_self=False)
    ci, cd = oracle.knn(X, Q, 6, metric="euclidean", order="arm", threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(gd.view(np.uint64), cd.view(np.uint64))
