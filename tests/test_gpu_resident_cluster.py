"""The shared-memory-resident kernel over block clusters: every (lattice,
cluster size) it is built for, against the per-half-sweep kernels bit for bit
-- spins, demons in the frame of the walk, energies -- over calls of one, two
and more iterations than the walk's period, so that the demons moved between
the blocks along z come round, with few and many samples (several waves of
clusters) and with fewer demon planes (the last plane along z being the last
of the iteration, or none)."""
import os

import numpy as np
import pytest

import micsa
from test_gpu_parity import random_state

pytestmark = pytest.mark.gpu


def _ctx(L, nr, ns, nc, env, st):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        ctx = micsa.Context(L, nr, ns, nc)
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v
    for s, (J, e, o, w0, w1, _) in enumerate(st):
        ctx.upload_couplings(s, J)
        ctx.upload_spins(s, e, o)
        ctx.upload_demons(s, w0, w1)
    return ctx


def _same(a, b, ns, what):
    ma, mb = a.measure(), b.measure()
    assert np.array_equal(ma["e_spin"], mb["e_spin"]), what
    assert np.array_equal(ma["e_demon"], mb["e_demon"]), what
    for s in range(ns):
        for x, y in zip(a.download_spins(s) + a.download_demons(s),
                        b.download_spins(s) + b.download_demons(s)):
            assert np.array_equal(x, y), (what, s)


@pytest.mark.parametrize("L,C,nr,nc,ns", [
    (16, 1, 32, 6, 2), (16, 2, 64, 6, 1), (16, 2, 32, 3, 1), (16, 4, 32, 5, 2), (16, 4, 96, 6, 1),
    (16, 8, 64, 6, 2), (16, 8, 32, 2, 1), (24, 4, 32, 6, 1), (24, 4, 64, 3, 2), (24, 8, 32, 5, 2),
    (24, 8, 64, 6, 20), (32, 8, 64, 6, 1), (32, 8, 32, 3, 2), (32, 8, 32, 1, 1), (32, 8, 64, 6, 10)])
def test_cluster_sizes_equal_half_sweep_kernels(L, C, nr, nc, ns):
    rng = np.random.default_rng(L * 1000 + C * 100 + nr + nc)
    st = random_state(rng, L, nr, nc, ns)
    a = _ctx(L, nr, ns, nc, {"MICSA_RESIDENT_CTAS": str(C)}, st)
    b = _ctx(L, nr, ns, nc, {"MICSA_RESIDENT": "0"}, st)
    for n in (1, 2, L // 2 + 3, 1026 if ns <= 2 else 5):
        l0 = a.kernel_launches()
        a.iterate(n)
        assert a.kernel_launches() - l0 == 2 * (1 + (n - 1) // 1024)  # the kernel and the walk
        b.iterate(n)
        _same(a, b, ns, n)
    a.synchronize()  # no wait of the exchange ran out
    a.close()
    b.close()


def test_frozen_samples_and_refresh_between_cluster_launches():
    """A frozen sample keeps its state while the others advance; uploads,
    single iterations through the half-sweep kernels (micsa_monte_carlo) and
    cluster launches continue one another."""
    L, nr, nc, ns = 24, 64, 6, 3
    rng = np.random.default_rng(8)
    st = random_state(rng, L, nr, nc, ns)
    a = _ctx(L, nr, ns, nc, {}, st)
    b = _ctx(L, nr, ns, nc, {"MICSA_RESIDENT": "0"}, st)
    for flags in ([1, 0, 1], [0, 1, 1], None):
        for c in (a, b):
            c.set_active(flags)
            c.iterate(5)
            c.monte_carlo(1)
            c.iterate(2)
    _same(a, b, ns, "mixed")
    a.close()
    b.close()


@pytest.mark.parametrize("L,nr,nc,ns,n", [
    (32, 64, 6, 10, 20),   # 20 clusters where 15 run at once: two launches share units
    (32, 96, 6, 11, 40),   # 33 clusters; rounds of unequal length
    (32, 32, 6, 17, 33),   # more than one walk period
    (24, 64, 6, 20, 40)])  # more clusters than run at once with the smaller cluster too
def test_rounds_equal_half_sweep_kernels(L, nr, nc, ns, n):
    """Calls cut into rounds over several launches, each unit's walk going on
    from its round before, and the calls after them."""
    rng = np.random.default_rng(L + nr + ns)
    st = random_state(rng, L, nr, nc, ns)
    a = _ctx(L, nr, ns, nc, {}, st)
    b = _ctx(L, nr, ns, nc, {"MICSA_RESIDENT": "0"}, st)
    for k in (n, 1, n + 3):
        for c in (a, b):
            c.iterate(k)
        _same(a, b, ns, k)
    if L == 32: # the largest one: 15 clusters at once
        l0 = a.kernel_launches()
        a.iterate(n)
        assert a.kernel_launches() - l0 > 2  # several rounds
    a.synchronize()
    a.close()
    b.close()
