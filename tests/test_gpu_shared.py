"""Launch rules of contexts that run side by side (a batch's shape groups, a
server's pools: micsa_create_shared) and of contexts of their own, seen from the
tuner's report and the number of launches; results as everywhere."""
import ctypes as C

import numpy as np
import pytest

import micsa
from test_gpu_parity import random_state

pytestmark = pytest.mark.gpu


class _Shared:
    """libmicsa with micsa_create standing for micsa_create_shared"""

    def __init__(self, lib):
        self._lib = lib
        lib.micsa_create_shared.argtypes = [C.c_void_p, C.c_void_p]
        lib.micsa_create_shared.restype = C.c_int

    def __getattr__(self, name):
        return getattr(self._lib, "micsa_create_shared" if name == "micsa_create" else name)


def _context(L, nr, ns, nc, shared):
    real = micsa.lib
    if shared:
        proxy = _Shared(real())
        micsa.lib = lambda: proxy
    try:
        return micsa.Context(L, nr, ns, nc)
    finally:
        micsa.lib = real


def test_side_by_side_no_chains_of_short_launches(monkeypatch):
    """60 samples of L = 24 take 55 to 75 us per iteration: two chains of 12
    launches would be shorter than 4 us each"""
    monkeypatch.setenv("MICSA_TUNE_CACHE", "0")
    st = random_state(np.random.default_rng(3), 24, 64, 6, 1)[0]
    with _context(24, 64, 60, 6, True) as a, _context(24, 64, 60, 6, False) as b:
        assert " chains=1/" in a.tuning(), a.tuning()
        for c in (a, b):
            c.set_active([1] + [0] * 59)
            c.upload_couplings(0, st[0])
            c.upload_spins(0, st[1], st[2])
            c.upload_demons(0, st[3], st[4])
            c.iterate(3)
        for x, y in zip(a.download_spins(0) + a.download_demons(0), b.download_spins(0) + b.download_demons(0)):
            assert np.array_equal(x, y)
