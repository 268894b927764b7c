"""Tensor-core kNN on small indexes cut into pieces of two and three tiles, sorted lists
and logs, up to and past the size from which pieces have sixteen.  Bar: bit-exact with
the oracle."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [129, 257, 400, 512, 513, 900, 1409, 3001, 8064, 8065, 8193])
@pytest.mark.parametrize("m,d,k,precision", [(3, 40, 5, "fp16"), (300, 64, 20, "bf16"), (300, 100, 100, "split_bf16"),
                                             (2500, 130, 60, "fp16"), (9000, 32, 10, "fp16")])
@pytest.mark.parametrize("data", ["normal", "ties"])
def test_small_index(gpu, oracle, n, m, d, k, precision, data):
    rng = np.random.default_rng(n + m)
    X = rng.normal(size=(n, d)).astype(np.float32)
    if data == "ties":
        X[n // 2:] = X[:n - n // 2]
    Q = rng.normal(size=(m, d)).astype(np.float32)
    Q[::3] = X[rng.integers(0, n, len(Q[::3]))]
    gi, gd = SearchIndex(X, distance="euclidean", tree="linear", order="arm", precision=precision).knn(
        Q, k, exclude_self=False)
    rows = rng.permutation(m)[:400]
    ci, cd = oracle.knn(X, Q[rows], k, metric="euclidean", order="arm", threads=threads())
    assert np.array_equal(gi[rows], ci)
    assert np.array_equal(f32_bits(gd[rows]), f32_bits(cd))
