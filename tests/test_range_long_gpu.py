"""Range lists of more hits than a warp sorts, many to a call: 2 to 16 keys per thread
of the block that sorts one, and the lists that just fit each count.  Bar: bit-exact
with the oracle."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 512, 513, 1024, 1025, 2047, 2048, 2049, 4096])
@pytest.mark.parametrize("metric", ["sqeuclidean", "euclidean"])
@pytest.mark.parametrize("data", ["normal", "ties"])
def test_every_row_a_hit(gpu, oracle, n, metric, data):
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, 3)) if data == "normal" else rng.integers(0, 3, size=(n, 3))
    X = X.astype(np.float32)
    Q = X[:40].copy()
    Q[3:6] += 1000.0  # no hits
    gi, gd = SearchIndex(X, distance=metric, tree="linear", order="arm").radius_search(Q, 100.0)
    off, ci, cd = oracle.range_search(X, Q, 100.0, metric=metric, order="arm", threads=threads())
    for i in range(len(Q)):
        assert np.array_equal(gi[i], ci[off[i]:off[i + 1]]), i
        assert np.array_equal(f32_bits(gd[i]), f32_bits(cd[off[i]:off[i + 1]])), i
    assert len(gi[0]) == n
