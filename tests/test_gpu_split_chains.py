"""A pinned sample order (MICSA_SWEEP_SPLIT) together with pinned chains and
iterations per replay (MICSA_SWEEP_CHAINS): the order holds, one chain and one
iteration per replay, and calls of any length equal the oracle."""
import numpy as np
import pytest

import micsa
import oracle
from test_gpu_parity import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split,chains,ns", [("1", "2/4", 3), ("2", "4/16", 5), ("1", "1/4", 1)])
def test_sample_order_with_chains_and_iterations_per_replay(monkeypatch, split, chains, ns):
    L, nr, nc = 24, 64, 3
    for k, v in (("ZC", "2"), ("SPLIT", split), ("CHAINS", chains)):
        monkeypatch.setenv("MICSA_SWEEP_" + k, v)
    st = random_state(np.random.default_rng(ns), L, nr, nc, ns)
    with micsa.Context(L, nr, ns, nc) as ctx:
        # one sample has no order of its own to hold
        assert "chains=%s " % ("1/1" if ns > 1 else chains) in ctx.tuning(), ctx.tuning()
        for s, (J, e, o, w0, w1, _) in enumerate(st):
            ctx.upload_couplings(s, J)
            ctx.upload_spins(s, e, o)
            ctx.upload_demons(s, w0, w1)
        for n in (1, 4, 9):
            ctx.iterate(n)
        ctx.monte_carlo(1)
        for s, (J, e, o, w0, w1, _) in enumerate(st):
            for _ in range(15):
                oracle.micsa_iteration(L, nr, nc, J, e, o, w0, w1, 16)
            for got, want in zip(ctx.download_spins(s) + ctx.download_demons(s), (e, o, w0, w1)):
                assert np.array_equal(got, want), s
