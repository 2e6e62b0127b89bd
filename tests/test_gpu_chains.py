"""An iteration's launches in chains of samples side by side, and several
iterations per graph replay, against one chain and one iteration: bit for bit,
with remainders of the replay's iterations, chains of unequal sample counts,
more chains asked for than samples, frozen samples, and the walk counters
continuing in single iterations."""
import os

import numpy as np
import pytest

import micsa
from test_gpu_parity import random_state

pytestmark = pytest.mark.gpu


def _ctx(L, nr, ns, nc, chains, st):
    env = {"MICSA_RESIDENT": "0", "MICSA_SWEEP_ZC": "2", "MICSA_SWEEP_CHAINS": chains}
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


@pytest.mark.parametrize("L,nr,nc,ns,chains,said", [
    (16, 32, 6, 2, "2/1", "2/1"), (16, 64, 3, 5, "2/4", "2/4"), (24, 96, 5, 7, "4/4", "4/4"),
    (16, 32, 6, 3, "4/2", "3/2"), (24, 64, 6, 1, "2/4", "1/4"), (8, 32, 1, 9, "4/16", "4/16")])
def test_chains_equal_one_chain(L, nr, nc, ns, chains, said):
    st = random_state(np.random.default_rng(L + ns), L, nr, nc, ns)
    a, b = _ctx(L, nr, ns, nc, chains, st), _ctx(L, nr, ns, nc, "1/1", st)
    assert "chains=%s " % said in a.tuning(), a.tuning()
    for n, frozen in ((1, None), (4, 0), (7, None), (L // 2 + 3, ns - 1), (33, None)):
        flags = None if frozen is None or ns == 1 else [int(s != frozen) for s in range(ns)]
        for c in (a, b):
            c.set_active(flags)
            c.iterate(n)
            c.monte_carlo(1)
    a.profile(3)
    b.iterate(3)
    ma, mb = a.measure(), b.measure()
    assert np.array_equal(ma["e_spin"], mb["e_spin"]) and np.array_equal(ma["e_demon"], mb["e_demon"])
    for s in range(ns):
        for x, y in zip(a.download_spins(s) + a.download_demons(s), b.download_spins(s) + b.download_demons(s)):
            assert np.array_equal(x, y), s
    a.close()
    b.close()
