"""Batched k-means with its arrays in different places: rows and first centres in
device memory (at 16-byte boundaries and one to three floats past them), in host
memory and pinned, centres out to host and device, sizes that are not multiples of
4 values, and labels into arrays never written.  Bar: bit-identical to the call
with everything in host memory."""
import ctypes

import numpy as np
import pytest

from fuel_gb300 import _lib

pytestmark = pytest.mark.gpu


def call(problems, order=0):
    arr = (_lib.KMeansProblem * len(problems))(*[
        _lib.KMeansProblem(x, n, d, k, c, oc, ol, 0, 0, 0.0) for x, n, d, k, c, oc, ol in problems])
    _lib.check(_lib.load().fuelg_kmeans_batched(ctypes.cast(arr, ctypes.c_void_p), len(arr), 5, order,
                                                _lib.PRECISION["auto"], _lib.LLOYD_FIXED_ITERS, None))
    return [(p.out_iters, p.status) for p in arr]


def test_batched_array_places(gpu):
    import torch
    rng = np.random.default_rng(2)
    shapes = [(n, d, k) for n in (1, 37, 130, 4001) for d in (1, 2, 3, 8, 31, 32, 37, 64, 70) for k in (1, 5)
              if k <= n] + [(70001, 3, 4)]
    data = [(rng.normal(size=(n, d)).astype(np.float32), n, d, k) for n, d, k in shapes]
    init = [x[rng.permutation(n)[:k]].copy() for x, n, d, k in data]
    ref_c = [np.empty((k, d), np.float32) for _, n, d, k in data]
    ref_l = [np.empty(n, np.int64) for _, n, d, k in data]
    ref = call([(x.ctypes.data, n, d, k, c.ctypes.data, oc.ctypes.data, ol.ctypes.data)
                for (x, n, d, k), c, oc, ol in zip(data, init, ref_c, ref_l)])

    keep = []  # owners of the memory

    def placed(a, where):
        if where == 5:
            return a.ctypes.data
        if where == 4:
            keep.append(torch.from_numpy(a).pin_memory())
            return keep[-1].data_ptr()
        t = torch.empty(a.size + 4, device="cuda")  # where: floats past the boundary
        t[where:where + a.size] = torch.from_numpy(a.ravel()).cuda()
        keep.append(t)
        return t.data_ptr() + 4 * where

    for shift in range(6):
        out_c = [np.empty((k, d), np.float32) if (i + shift) % 2 else torch.empty((k, d), device="cuda")
                 for i, (_, n, d, k) in enumerate(data)]
        out_l = [np.empty(n, np.int64) for _, n, d, k in data]
        problems = []
        for i, ((x, n, d, k), c, oc, ol) in enumerate(zip(data, init, out_c, out_l)):
            problems.append((placed(x, (i + shift) % 6), n, d, k, placed(c, (i // 2 + shift) % 6),
                             oc.ctypes.data if isinstance(oc, np.ndarray) else oc.data_ptr(), ol.ctypes.data))
        torch.cuda.synchronize()
        assert call(problems) == ref
        for oc, ol, rc, rl in zip(out_c, out_l, ref_c, ref_l):
            oc = oc if isinstance(oc, np.ndarray) else oc.cpu().numpy()
            np.testing.assert_array_equal(oc.view(np.uint32), rc.view(np.uint32))
            np.testing.assert_array_equal(ol, rl)
