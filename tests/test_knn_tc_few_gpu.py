"""Few queries through the tensor-core screen: one block's rows dealt to four or
eight warps, with and without a cut of the index into pieces, per tier, sorted
lists (up to 32 keys kept) and logs.  Bar: bit-exact with the oracle."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 15, 16, 17, 33, 63, 64, 65, 127, 129, 255, 256, 257])
@pytest.mark.parametrize("n,d,k,precision", [(700, 40, 3, "fp16"), (9000, 96, 10, "fp16"), (9000, 130, 40, "split_bf16"),
                                             (30000, 33, 100, "split_bf16"), (12000, 64, 5, "bf16")])
def test_few_queries(gpu, oracle, m, n, d, k, precision):
    rng = np.random.default_rng(m + n)
    X = rng.normal(size=(n, d)).astype(np.float32)
    X[n // 2:n // 2 + 30] = X[:30]  # ties
    Q = np.concatenate([X[:m // 2], rng.normal(size=(m - m // 2, d)).astype(np.float32)])
    gi, gd = SearchIndex(X, distance="euclidean", tree="linear", order="arm", precision=precision).knn(
        Q, k, exclude_self=False)
    ci, cd = oracle.knn(X, Q, k, metric="euclidean", order="arm", threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(f32_bits(gd), f32_bits(cd))
