"""The automatic tier on an index whose norms leave the tensor-core screen's range:
the plain scan answers, nothing is timed, and nothing is recorded for other indexes
of the same shape and value class."""
import numpy as np
import pytest

from conftest import f32_bits, threads
from fuel_gb300 import SearchIndex

pytestmark = pytest.mark.gpu


def test_auto_leaves_large_norms_to_the_plain_scan(gpu, oracle, tmp_path, monkeypatch):
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("FUELG_TUNE_CACHE", str(cache))
    rng = np.random.default_rng(7)
    X = (1e19 * rng.normal(size=(1531, 77))).astype(np.float32)
    ix = SearchIndex(X, distance="sqeuclidean", tree="linear", order="arm")
    gi, gd = ix.knn(X[:50].copy(), 9, exclude_self=False)
    ci, cd = oracle.knn(X, X[:50], 9, metric="sqeuclidean", order="arm", threads=threads())
    assert np.array_equal(gi, ci) and np.array_equal(f32_bits(gd), f32_bits(cd))
    assert ix.last_stats["precision_used"] == 0
    recorded = cache.read_text().splitlines() if cache.exists() else []
    assert not [ln for ln in recorded if ln.split()[:2] == ["knn", "77"]]
