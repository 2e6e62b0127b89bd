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


@pytest.mark.parametrize("L,ns,shared,halves,resident", [
    (16, 100, False, 1, 2), (16, 300, False, 1, 2), (16, 300, True, 2, 3),  # two and four waves of clusters
    (32, 24, False, 4, 5), (32, 24, True, 11, 12), (24, 4, True, 0, 1)])
def test_calls_long_enough_to_run_in_shared_memory(monkeypatch, L, ns, shared, halves, resident):
    """calls of up to `halves` iterations run half-sweep by half-sweep, of `resident` and more in
    one or a few launches; the same state either way"""
    monkeypatch.setenv("MICSA_SWEEP_FLOW", "0")
    J, e, o, w0, w1, _ = random_state(np.random.default_rng(L), L, 64, 6, 1)[0]
    with _context(L, 64, ns, 6, shared) as a, _context(L, 64, ns, 6, not shared) as b:
        for c in (a, b):
            c.set_active([0] * (ns - 1) + [1])
            c.upload_couplings(ns - 1, J)
            c.upload_spins(ns - 1, e, o)
            c.upload_demons(ns - 1, w0, w1)
        for n, whole in ((halves, False), (resident, True)):
            before = a.kernel_launches()
            if n:
                a.iterate(n)
                assert (a.kernel_launches() - before < 12) == whole, (n, a.kernel_launches() - before)
                b.iterate(n)
        for x, y in zip(a.download_spins(ns - 1) + a.download_demons(ns - 1),
                        b.download_spins(ns - 1) + b.download_demons(ns - 1)):
            assert np.array_equal(x, y)


def test_resident_groups_beside_a_mixed_launch_run_in_one_launch_a_call():
    """20 clusters of L = 32 where about 15 run at once: in rounds when the context runs alone,
    in one launch (and the walk's) while the mixed launch of the other context has work"""
    shapes = [(32, 64, 10, 6), (48, 64, 1, 6)]
    ctxs = [micsa.Context(*s) for s in shapes]
    ref = micsa.Context(*shapes[0])
    st = [random_state(np.random.default_rng(L), L, nr, nc, 1)[0] for L, nr, _, nc in shapes]
    for c, (L, nr, ns, nc), (J, e, o, w0, w1, _) in zip(ctxs + [ref], shapes + shapes[:1], st + st[:1]):
        for s in range(ns):
            c.upload_couplings(s, J)
            c.upload_spins(s, e, o)
            c.upload_demons(s, w0, w1)
    before = ref.kernel_launches()
    ref.iterate(20)
    assert ref.kernel_launches() - before > 2
    with micsa.Multi(ctxs) as multi:
        before = ctxs[0].kernel_launches()
        multi.iterate(20)
        assert ctxs[0].kernel_launches() - before == 2
        multi.synchronize()
    for s in (0, 9):
        for x, y in zip(ctxs[0].download_spins(s) + ctxs[0].download_demons(s),
                        ref.download_spins(s) + ref.download_demons(s)):
            assert np.array_equal(x, y), s
    for c in ctxs + [ref]:
        c.close()
