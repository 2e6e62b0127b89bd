"""Uploads from page-locked, mapped host buffers (converted straight from them
by the device) equal uploads from ordinary ones (copied, then converted):
the states read back equal what went up, word for word."""
import ctypes as C

import numpy as np
import pytest

import micsa
from test_gpu_download import _pinned
from test_gpu_parity import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nr,nc,ns", [(8, 32, 1, 2), (16, 64, 6, 2), (24, 96, 3, 1), (40, 128, 2, 1)])
def test_upload_from_mapped_buffers_equals_staged(L, nr, nc, ns):
    st = random_state(np.random.default_rng(L + nr), L, nr, nc, ns)
    p64 = lambda v: v.ctypes.data_as(C.POINTER(C.c_uint64))
    keep = []

    def pinned(a):
        keep.append(_pinned(a.size))
        keep[-1][1][:] = a
        return p64(keep[-1][1])

    with micsa.Context(L, nr, ns, nc) as a, micsa.Context(L, nr, ns, nc) as b:
        lib = micsa.lib()
        for s, (J, e, o, w0, w1, _) in enumerate(st):
            a.upload_couplings(s, J)
            a.upload_spins(s, e, o)
            a.upload_demons(s, w0, w1)
            micsa.check(b.h, lib.micsa_upload_couplings(b.h, s, pinned(J)), "couplings")
            micsa.check(b.h, lib.micsa_upload_spins(b.h, s, pinned(e), pinned(o)), "spins")
            micsa.check(b.h, lib.micsa_upload_demons(b.h, s, pinned(w0), pinned(w1)), "demons")
            # one of the two page-locked only: staged
            micsa.check(b.h, lib.micsa_upload_demons(b.h, s, pinned(w0), p64(w1)), "demons")
            for c in (a, b):
                for got, want in zip(c.download_spins(s) + c.download_demons(s), (e, o, w0, w1)):
                    assert np.array_equal(got, want), s
        for c in (a, b):
            c.iterate(3)
        for s in range(ns):
            for x, y in zip(a.download_spins(s) + a.download_demons(s), b.download_spins(s) + b.download_demons(s)):
                assert np.array_equal(x, y), s
