"""Cancellation of a plain kNN scan over an index of few tiles: every block reads
the cancel word within its first 16 tiles of 128 rows."""
import threading
import time

import pytest

from fuel_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(2048, 4), (4500, 16), (4500, 20)])
def test_cancel_with_few_tiles(gpu, n, d):
    import ctypes

    import torch
    lib = _lib.load()
    m = 400_000_000 // (d * 4)
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn((n, d), device="cuda", generator=g)
    Q = torch.randn((m, d), device="cuda", generator=g)
    oi = torch.empty((m, 1), dtype=torch.int64, device="cuda")
    od = torch.empty((m, 1), device="cuda")
    torch.cuda.synchronize()
    h = ctypes.c_void_p()
    _lib.check(lib.fuelg_index_create(_lib.ptr(X), n, d, _lib.METRIC["sqeuclidean"], _lib.ORDER["arm"],
                                      ctypes.byref(h)))
    done = threading.Event()

    def cancel():
        while not done.is_set():  # (the call clears the word when it starts)
            lib.fuelg_cancel()
            time.sleep(2e-4)

    t = threading.Thread(target=cancel)
    try:
        t.start()
        rc = lib.fuelg_knn(h, _lib.ptr(Q), m, 1, _lib.EXCLUDE_NONE, _lib.PRECISION["fp32"], _lib.ptr(oi), _lib.ptr(od),
                           None)
    finally:
        done.set()
        t.join()
        lib.fuelg_index_destroy(h)
    assert rc == _lib.ECANCELLED
