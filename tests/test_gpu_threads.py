"""Contexts at work on host threads of their own, whose kernels ask for
different amounts of shared memory: no launch of one is refused because another
set a limit in between, and every result is the one of a context alone."""
import os
import threading

import numpy as np
import pytest

import micsa
from test_gpu_parity import random_state

pytestmark = pytest.mark.gpu

BETA = 0.9090909090909


def _together(works):
    """every work(k) on a thread of its own, started at once; the first error is raised"""
    gate, errs = threading.Barrier(len(works)), []

    def go(f):
        gate.wait()
        try:
            f()
        except Exception as e:  # noqa: BLE001
            errs.append(e)

    ts = [threading.Thread(target=go, args=(f,)) for f in works]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errs:
        raise errs[0]


@pytest.mark.parametrize("L,ncs", [(32, (6, 3, 6, 5)), (24, (6, 1, 5, 6)), (16, (6, 1, 3, 6))])
def test_small_lattices_of_several_demon_counts_side_by_side(L, ncs):
    nr, calls = 32, 1500
    states = [random_state(np.random.default_rng(L + k), L, nr, nc, 1)[0] for k, nc in enumerate(ncs)]
    ctxs = [micsa.Context(L, nr, 1, nc) for nc in ncs]
    for c, (J, e, o, w0, w1, _) in zip(ctxs, states):
        c.upload_couplings(0, J)
        c.upload_spins(0, e, o)
        c.upload_demons(0, w0, w1)

    def work(c):
        def f():
            for k in range(calls):
                c.iterate(2)
                if k % 50 == 49:
                    c.synchronize()
        return f

    _together([work(c) for c in ctxs])
    old = os.environ.get("MICSA_RESIDENT")
    os.environ["MICSA_RESIDENT"] = "0"
    try:
        for c, nc, (J, e, o, w0, w1, _) in zip(ctxs, ncs, states):
            with micsa.Context(L, nr, 1, nc) as ref:
                ref.upload_couplings(0, J)
                ref.upload_spins(0, e, o)
                ref.upload_demons(0, w0, w1)
                ref.iterate(2 * calls)
                for x, y in zip(c.download_spins(0) + c.download_demons(0),
                                ref.download_spins(0) + ref.download_demons(0)):
                    assert np.array_equal(x, y), nc
    finally:
        if old is None:
            os.environ.pop("MICSA_RESIDENT")
        else:
            os.environ["MICSA_RESIDENT"] = old
    for c in ctxs:
        c.close()


def test_overlaps_of_large_lattices_side_by_side(monkeypatch):
    monkeypatch.setenv("MICSA_SWEEP_ZC", "8")  # no launch shapes to time
    nr, Ls = 32, (256, 320, 256, 384)
    ctxs, first = [], []
    for k, L in enumerate(Ls):
        H = (L // 4) ** 3 // 2
        rng = np.random.default_rng(k)
        c = micsa.Context(L, nr, 1, 1)
        c.upload_couplings(0, np.zeros(12 * H, np.uint64))
        c.upload_spins(0, *(rng.integers(0, 2 ** 63, size=H * nr, dtype=np.uint64) for _ in range(2)))
        m = c.measure(spin=False, demon=False, overlap=True)
        ctxs.append(c)
        first.append(m)

    def work(c, m):
        def f():
            for _ in range(60):
                n = c.measure(spin=False, demon=False, overlap=True)
                assert np.array_equal(n["q"], m["q"]) and np.array_equal(n["c4"], m["c4"])
        return f

    _together([work(c, m) for c, m in zip(ctxs, first)])
    for c in ctxs:
        c.close()


def test_batches_of_small_lattices_with_several_demon_counts():
    jobs = [dict(L=32, nr=32, nc=nc, iterations=40 + nc, seed_J=7 + k, seed_u=9 + k, beta=BETA)
            for k, nc in enumerate((3, 5, 6, 3, 5, 6))]
    want = micsa.run_batch(jobs)
    for _ in range(10):
        es, ed, _ = micsa.run_batch(jobs)
        for a, b in zip(es + ed, want[0] + want[1]):
            assert np.array_equal(a, b)
