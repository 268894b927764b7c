"""The Lloyd tensor-core screen where its values are not finite (norms past the
float32 range, infinities in the data, NaN first centres), with centre counts that
leave padding columns and counts that do not: the exact re-score decides among the
real centres alone.  Bar: labels, centres and iterations equal to the plain FP32
tier's, bit for bit."""
import numpy as np
import pytest

from fuel_gb300 import kmeans

pytestmark = pytest.mark.gpu


def problem(kind, n, d, k, rng):
    X = rng.normal(size=(n, d)) + 3 * rng.integers(-2, 3, size=(n, 1))
    if kind == "large":
        X *= 1e20  # |x|^2 and the products overflow
    elif kind == "some_large":
        X[rng.random(n) < 0.3] *= 1e20
    X = X.astype(np.float32)
    init = X[rng.permutation(n)[:k]].copy()
    if kind == "inf":
        X[n // 2, 0] = np.inf
    elif kind == "nan_centres":
        init[rng.random(k) < 0.5] = np.nan
        init[0] = np.nan
    return X, init


@pytest.mark.parametrize("kind", ["large", "some_large", "inf", "nan_centres"])
@pytest.mark.parametrize("k", [1, 5, 15, 16, 17, 33, 40, 64, 65, 100, 250])
@pytest.mark.parametrize("d", [32, 65, 130])
@pytest.mark.parametrize("precision", ["bf16", "split_bf16"])
def test_screen_without_finite_values(gpu, kind, k, d, precision):
    X, init = problem(kind, 128 * 4 + 37, d, k, np.random.default_rng(k * 1000 + d))
    args = dict(k=k, variant="lloyd", init=init, max_iter=4, fixed_iters=True)
    got = kmeans(X, precision=precision, **args)
    ref = kmeans(X, precision="fp32", **args)
    assert got.stats["precision_used"] in (1, 2, 3), "the screen serves the shape"
    np.testing.assert_array_equal(got.labels, ref.labels)
    np.testing.assert_array_equal(got.centers.view(np.uint32), ref.centers.view(np.uint32))
    assert got.n_iter == ref.n_iter
