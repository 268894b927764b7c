"""Batched k-means labels: widened on the host and on the device, at the sizes where
one gives way to the other, into arrays never written, one problem and several, and
without room for the device's.  Bar: equal to each problem's own call."""
import ctypes

import numpy as np
import pytest

from fuel_gb300 import _lib, kmeans, kmeans_batched

pytestmark = pytest.mark.gpu


def problems(sizes):
    rng = np.random.default_rng(len(sizes))
    out = []
    for n in sizes:
        X = (rng.normal(size=(n, 3)) + 4 * rng.integers(0, 3, size=(n, 1))).astype(np.float32)
        out.append((X, X[:6].copy()))
    return out


def check(probs):
    got = kmeans_batched(probs, max_iter=3, order="arm", fixed_iters=True)
    for (X, init), g in zip(probs, got):
        ref = kmeans(X, k=6, variant="lloyd", init=init, max_iter=3, order="arm", fixed_iters=True, precision="fp32")
        np.testing.assert_array_equal(g.labels, ref.labels)
        np.testing.assert_array_equal(g.centers.view(np.uint32), ref.centers.view(np.uint32))


@pytest.mark.parametrize("sizes", [(6,), (32768,), (32769,), (16384, 16384, 32768), (16385, 16384, 32768),
                                   (100003, 7, 513)])
def test_labels_of_few_and_many_rows(gpu, sizes):
    check(problems(sizes))


def test_labels_without_room(gpu):
    fn = _lib.load().fuelg_test_scratch_room
    fn.argtypes, fn.restype = [ctypes.c_int64], None
    probs = problems((100003, 50000))
    fn(1_000_000)  # (the wide labels alone are scratch of this kind: 1.2 MB)
    try:
        got = kmeans_batched(probs, max_iter=3, order="arm", fixed_iters=True)
    finally:
        fn(-1)
    ref = kmeans_batched(probs, max_iter=3, order="arm", fixed_iters=True)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a.labels, b.labels)
