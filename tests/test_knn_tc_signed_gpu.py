"""Tensor-core kNN on integers of both signs: squared distances reach four times
d V^2, so f32 sums may round (fuel's after every term, above 2^24) where those of
nonnegative integers are exact.  Index rows nearly opposite to the queries, with k
large enough that far rows are returned, around the sizes from which the screened
distances are final.  Bar: bit-exact with the oracle."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,vmax", [(32, 256), (64, 256), (65, 256), (100, 204), (100, 206), (128, 181), (128, 182),
                                    (128, 255), (200, 144), (200, 146), (256, 128), (256, 180)])
@pytest.mark.parametrize("precision", ["bf16", "split_bf16", "fp16"])
@pytest.mark.parametrize("metric,order", [("sqeuclidean", "arm"), ("euclidean", "x86")])
def test_signed_integers(gpu, oracle, d, vmax, precision, metric, order):
    rng = np.random.default_rng(d + vmax)
    n, m, k = 400, 70, 180
    sign = rng.choice([-1.0, 1.0], size=d)
    # sizes odd and even near the largest, one of each block at the largest itself
    Q = sign * rng.integers(vmax - 3, vmax + 1, size=(m, d))
    X = -sign * rng.integers(vmax - 3, vmax + 1, size=(n, d))
    X[rng.random((n, d)) < 0.03] *= -1
    X[0], Q[0] = -sign * vmax, sign * vmax
    X[200:240] = X[:40]
    X, Q = X.astype(np.float32), Q.astype(np.float32)
    if d > 128 and precision == "split_bf16":
        precision = "bf16"  # (the split operands of more than two chunks do not fit)
    ix = SearchIndex(X, distance=metric, tree="linear", order=order, precision=precision)
    gi, gd = ix.knn(Q, k, exclude_self=False)
    assert ix.last_stats["precision_used"] in (1, 2, 4), "a tensor-core tier serves the shape"
    ci, cd = oracle.knn(X, Q, k, metric=metric, order=order, threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(f32_bits(gd), f32_bits(cd))
