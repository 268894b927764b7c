"""Range search with little device memory: without room for the queries' slots the
two-pass scan answers, lists longer than the slots are made in the slots' place, and
a call that cannot be answered says so and leaves the index usable.  Bar: equal to
the call without a limit, which other tests hold against the oracle."""
import ctypes

import numpy as np
import pytest

from fuel_gb300 import SearchIndex, _lib

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture
def room(gpu):
    """Limits this thread's device scratch for the next calls."""
    fn = _lib.load().fuelg_test_scratch_room
    fn.argtypes, fn.restype = [ctypes.c_int64], None
    yield fn
    fn(-1)


def same(a, b):
    assert len(a[0]) == len(b[0])
    for x, y in zip(a[0] + a[1], b[0] + b[1]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("metric", ["sqeuclidean", "euclidean"])
@pytest.mark.parametrize("radius,limit,passes", [(1.0, 500, 1), (1.0, 8, 2), (100.0, 500, 2), (100.0, 270, 2)])
def test_range_in_little_memory(room, metric, radius, limit, passes):
    """2000 queries have 65 MB of slots; with every row a hit their lists are 80 MB, three times in the sort."""
    rng = np.random.default_rng(4)
    X = rng.normal(size=(5000, 6)).astype(np.float32)
    Q = X[:2000].copy()
    ix = SearchIndex(X, distance=metric, tree="linear", order="arm")
    ref = ix.radius_search(Q, radius)
    room(limit * MB)
    got = ix.radius_search(Q, radius)
    assert ix.last_stats["distance_evals"] == passes * 2000 * 5000
    same(got, ref)


def test_range_without_memory(room):
    rng = np.random.default_rng(5)
    X = rng.normal(size=(5000, 6)).astype(np.float32)
    ix = SearchIndex(X, distance="sqeuclidean", tree="linear", order="arm")
    ref = ix.radius_search(X[:2000].copy(), 100.0)
    for limit in (100, 1):
        room(limit * MB)
        with pytest.raises(MemoryError):
            ix.radius_search(X[:2000].copy(), 100.0)
    room(-1)
    same(ix.radius_search(X[:2000].copy(), 100.0), ref)
