"""Batched k-means of 2 and 8 dimensions with more centres than a block stages (the
rows' coordinates in registers, centres from global memory) and the last counts that
it does.  Bar: equal to each problem's own call, bit for bit."""
import numpy as np
import pytest

from fuel_gb300 import kmeans, kmeans_batched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["arm", "x86"])
@pytest.mark.parametrize("d,k", [(2, 8191), (2, 8192), (2, 8193), (8, 2047), (8, 2048), (8, 2049)])
def test_batched_centres_around_the_stage(gpu, order, d, k):
    rng = np.random.default_rng(k)
    probs = []
    for kk in (k, 5):
        X = np.round(rng.normal(size=(k + 700, d)) * 64).astype(np.float32)  # ties
        probs.append((X, X[rng.permutation(len(X))[:kk]].copy()))
    got = kmeans_batched(probs, max_iter=3, order=order, fixed_iters=True)
    for (X, init), g in zip(probs, got):
        ref = kmeans(X, k=len(init), variant="lloyd", init=init, max_iter=3, order=order, fixed_iters=True,
                     precision="fp32")
        np.testing.assert_array_equal(g.labels, ref.labels)
        np.testing.assert_array_equal(g.centers.view(np.uint32), ref.centers.view(np.uint32))
