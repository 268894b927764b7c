"""kNN with little device memory: calls whose tensor-core or register-tile lists do
not fit take the next scan, whose own do, and large calls keep their lists within
1 GiB by batches.  Bar: bit-exact with the oracle."""
import ctypes

import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex, _lib

pytestmark = pytest.mark.gpu

KB = 1 << 10


@pytest.fixture
def room(gpu):
    """Limits this thread's device scratch for the next calls."""
    fn = _lib.load().fuelg_test_scratch_room
    fn.argtypes, fn.restype = [ctypes.c_int64], None
    yield fn
    fn(-1)


# (the tiles' lists: 1.5 and 18 MB; the screen's, 12 MB or more)
@pytest.mark.parametrize("n,m,d,k,precision,limit", [
    (40000, 64, 8, 10, "fp32", 1000), (40000, 64, 8, 40, "fp32", 4000), (20000, 20, 64, 10, "bf16", 6000),
    (20000, 20, 64, 10, "split_bf16", 6000), (20000, 20, 64, 40, "fp16", 8000),
])
def test_knn_in_little_memory(room, oracle, n, m, d, k, precision, limit):
    rng = np.random.default_rng(n + k)
    X = rng.normal(size=(n, d)).astype(np.float32)
    Q = rng.normal(size=(m, d)).astype(np.float32)
    ix = SearchIndex(X, distance="sqeuclidean", tree="linear", order="arm", precision=precision)
    ix.knn(Q[:1], 1, exclude_self=False)  # the index's tensor-core form
    room(limit * KB)
    gi, gd = ix.knn(Q, k, exclude_self=False)
    assert ix.last_stats["precision_used"] == 0
    ci, cd = oracle.knn(X, Q, k, metric="sqeuclidean", order="arm", threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(f32_bits(gd), f32_bits(cd))
    room(10 * KB)
    with pytest.raises(MemoryError):
        ix.knn(Q, k, exclude_self=False)


def test_knn_f64_in_little_memory(room, oracle):
    """64 queries: 10 MB of distances, 20 MB of lists of the screen."""
    rng = np.random.default_rng(6)
    X, Q = rng.normal(size=(20000, 4)), rng.normal(size=(64, 4))
    ix = SearchIndex(X, distance="euclidean", tree="linear", order="arm")
    ix.knn(Q[:1], 1, exclude_self=False)
    room(14000 * KB)
    gi, gd = ix.knn(Q, 40, exclude_self=False)
    ci, cd = oracle.knn(X, Q, 40, metric="euclidean", order="arm", threads=threads())
    assert np.array_equal(gi, ci)
    assert np.array_equal(gd.view(np.uint64), cd.view(np.uint64))


def test_knn_lists_in_batches(room, oracle):
    """A million queries, 33 keys: 2312 bytes of lists a query, 464 384 queries a batch."""
    rng = np.random.default_rng(7)
    X = rng.normal(size=(1000, 2)).astype(np.float32)
    Q = rng.normal(size=(1_000_000, 2)).astype(np.float32)
    ix = SearchIndex(X, distance="sqeuclidean", tree="linear", order="arm", precision="fp32")
    # keys 264 MB, results 396, queries 8
    room(2_000_000 * KB)
    gi, gd = ix.knn(Q, 33, exclude_self=False)
    assert ix.last_stats["hot_kernel_launches"] == 3
    rows = np.r_[0:50, 464_300:464_450, 928_700:928_850, 999_900:1_000_000]
    ci, cd = oracle.knn(X, Q[rows], 33, metric="sqeuclidean", order="arm", threads=threads())
    assert np.array_equal(gi[rows], ci)
    assert np.array_equal(f32_bits(gd[rows]), f32_bits(cd))
