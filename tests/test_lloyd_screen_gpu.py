"""The Lloyd tensor-core screen at the edges of its column blocks (16 columns per
load, 32 per step, 64 per candidate word, up to 256 centres), with tied and
duplicate centres, signed and nonnegative data, against the plain FP32 tier.
Bar: labels, centres and iterations bit-identical."""
import numpy as np
import pytest

from fuel_gb300 import kmeans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 96, 127, 128, 129, 192, 193, 255, 256])
@pytest.mark.parametrize("d", [16, 33, 130])
@pytest.mark.parametrize("precision", ["bf16", "split_bf16"])
def test_screen_matches_fp32_tier(gpu, k, d, precision):
    rng = np.random.default_rng(k * 1000 + d)
    n = 128 * 5 + 37
    X = rng.normal(size=(n, d)) + 3 * rng.integers(-2, 3, size=(n, 1))
    if k % 2:
        X = np.abs(np.round(X * 4) / 4)  # nonnegative, with exact ties
    X = X.astype(np.float32)
    init = X[rng.permutation(n)[:k]].copy()
    init[k // 2] = init[0]  # duplicate centres: the first index wins
    got = kmeans(X, k=k, variant="lloyd", init=init, max_iter=5, fixed_iters=True, precision=precision)
    ref = kmeans(X, k=k, variant="lloyd", init=init, max_iter=5, fixed_iters=True, precision="fp32")
    np.testing.assert_array_equal(got.labels, ref.labels)
    np.testing.assert_array_equal(got.centers.view(np.uint32), ref.centers.view(np.uint32))
    assert got.n_iter == ref.n_iter


@pytest.mark.parametrize("n", [152 * 128, 152 * 128 + 1, 152 * 128 * 3 + 5])
@pytest.mark.parametrize("k,precision", [(65, "split_bf16"), (250, "split_bf16"), (200, "bf16"), (40, "split_bf16")])
def test_screen_several_tiles_per_block(gpu, n, k, precision):
    """One to four tiles per block, with one epilogue group (k = 40) and two."""
    rng = np.random.default_rng(n + k)
    X = (rng.normal(size=(n, 33)) + 3 * rng.integers(-2, 3, size=(n, 1))).astype(np.float32)
    init = X[rng.permutation(n)[:k]].copy()
    got = kmeans(X, k=k, variant="lloyd", init=init, max_iter=3, fixed_iters=True, precision=precision)
    ref = kmeans(X, k=k, variant="lloyd", init=init, max_iter=3, fixed_iters=True, precision="fp32")
    np.testing.assert_array_equal(got.labels, ref.labels)
    np.testing.assert_array_equal(got.centers.view(np.uint32), ref.centers.view(np.uint32))
