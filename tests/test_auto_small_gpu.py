"""The automatic tier on small indexes of wide rows: the plain scan is timed beside the
tensor-core tiers, may be chosen, and is recorded for the bucket like them."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,m", [(1500, 83, 120, 300), (2500, 91, 8, 3), (300, 250, 100, 40)])
def test_auto_times_the_plain_scan(gpu, oracle, tmp_path, monkeypatch, n, d, k, m):
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("FUELG_TUNE_CACHE", str(cache))
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, d)).astype(np.float32)
    Q = rng.normal(size=(m, d)).astype(np.float32)
    ix = SearchIndex(X, distance="sqeuclidean", tree="linear", order="arm")
    ci, cd = oracle.knn(X, Q, k, metric="sqeuclidean", order="arm", threads=threads())
    for _ in range(2):  # timed, then by the bucket (which has the number of queries)
        gi, gd = ix.knn(Q, k, exclude_self=False)
        assert np.array_equal(gi, ci) and np.array_equal(f32_bits(gd), f32_bits(cd))
        tier = ix.last_stats["precision_used"]
        assert tier in (0, 1, 2, 4)
    lines = [ln.split() for ln in cache.read_text().splitlines()]
    assert [int(ln[5]) for ln in lines if ln[:2] == ["knn", str(d)]] == [tier]
    if n == 1500:
        assert tier == 0, "five times as fast as the screens here"
