"""Range search in register tiles at the edges of its tiles (64 queries, 128
index rows, strips of tiles, one or two buffers), of the sorts of a query's hits
(32, 64, 128 and 256 keys by a warp, up to 4096 by a block) and past them (second
pass and segmented sort).  Bar: bit-exact with the oracle."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


def check(oracle, X, Q, radius, metric, order, exclude=False):
    gi, gd = SearchIndex(X, distance=metric, tree="linear", order=order).radius_search(Q, radius, exclude_self=exclude)
    off, ci, cd = oracle.range_search(X, Q, radius, metric=metric, order=order, exclude_self=exclude,
                                      threads=threads())
    assert len(gi) == len(off) - 1
    for i in range(len(gi)):
        assert np.array_equal(gi[i], ci[off[i]:off[i + 1]]), i
        assert np.array_equal(f32_bits(gd[i]), f32_bits(cd[off[i]:off[i + 1]])), i
    return [len(g) for g in gi]


@pytest.mark.parametrize("n,m,d", [(1, 1, 1), (127, 63, 7), (128, 64, 8), (129, 65, 9), (3000, 130, 33),
                                   (50001, 257, 5), (700, 90, 86), (700, 90, 88), (640, 64, 128), (640, 64, 129)])
@pytest.mark.parametrize("order,metric", [("arm", "sqeuclidean"), ("x86", "euclidean")])
def test_range_tile_edges(gpu, oracle, n, m, d, order, metric):
    rng = np.random.default_rng(n + m + d)
    X = rng.normal(size=(n, d)).astype(np.float32)
    X[n // 2:] = X[:n - n // 2]  # ties
    r = float(np.sqrt(1.2 * d))
    r = r if metric == "euclidean" else r * r
    check(oracle, X, X[:m].copy(), r, metric, order)
    if n <= 1000:
        check(oracle, X, X, r, metric, order, exclude=True)


@pytest.mark.parametrize("hits", [31, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1024, 1025, 4095, 4096, 4097, 4700])
def test_range_sort_widths(gpu, oracle, hits):
    """Query 0 has exactly `hits` hits, the others far fewer or none."""
    rng = np.random.default_rng(hits)
    X = (100 + rng.normal(size=(5000, 6))).astype(np.float32)
    near = rng.permutation(5000)[:hits]
    X[near] = rng.integers(-3, 4, size=(hits, 6)).astype(np.float32) / 16
    Q = np.concatenate([np.zeros((1, 6)), X[:9]]).astype(np.float32)
    Q[1:][np.abs(Q[1:]).max(1) < 1] = -50
    for metric in ["euclidean", "sqeuclidean"]:
        assert check(oracle, X, Q, 2.0, metric, "arm")[0] == hits


@pytest.mark.parametrize("radius", [-0.0, 0.0, 1e-30, 3e38, np.inf, -1.0])
@pytest.mark.parametrize("metric", ["sqeuclidean", "euclidean"])
def test_range_special_radii_and_values(gpu, oracle, radius, metric):
    rng = np.random.default_rng(8)
    X = rng.integers(0, 2, size=(300, 3)).astype(np.float32)
    X[20:40] = np.inf
    X[40:60] = np.nan
    check(oracle, X, X[:64].copy(), radius, metric, "arm")
