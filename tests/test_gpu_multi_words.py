"""The mixed-lattice launch where a site has several word groups: odd numbers
of 32-replica words (96 and 160 replicas: three and five one-word groups), and
six words (three groups of two), every group in the launch, against the oracle
bit for bit -- more iterations than half the smallest side, several samples per
tile, several iterations per launch, a frozen sample, and the tuned shape."""
import os

import pytest

import micsa
from test_gpu_multi import _check, _groups, _upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes,iters,pin", [
    ([(8, 96, 6, 3), (16, 96, 3, 2), (24, 96, 6, 1)], 9, {"MICSA_MULTI_ZC": "4", "MICSA_MULTI_ITERS": "4"}),
    ([(8, 160, 2, 2), (16, 160, 6, 1)], 6, {"MICSA_MULTI_ZC": "2"}),
    ([(16, 192, 6, 2), (24, 192, 1, 1)], 9, {"MICSA_MULTI_ZC": "8"}),
    ([(16, 96, 6, 2), (40, 96, 6, 1)], 9, {}),  # the tuned shape
])
def test_mixed_launch_of_several_word_groups(shapes, iters, pin):
    pin = dict(pin, MICSA_MULTI_RESIDENT="0")
    old = {k: os.environ.get(k) for k in pin}
    os.environ.update(pin)
    try:
        ctxs, states = _groups(shapes, seed=iters + shapes[0][1])
        multi = micsa.Multi(ctxs)
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v
    with multi:
        assert "resident" not in multi.report(), multi.report()
        for ctx, st in zip(ctxs, states):
            _upload(ctx, st)
        multi.iterate(iters - 2)
        ctxs[0].set_active([1] * (shapes[0][3] - 1) + [0])
        multi.iterate(2)
        multi.synchronize()
        for k, (ctx, st, (L, nr, nc, ns)) in enumerate(zip(ctxs, states, shapes)):
            last = ns - 1 if k == 0 else ns
            _check(ctx, st[:last], L, nr, nc, iters)
            if k == 0:  # the sample frozen after iters - 2
                J, e, o, w0, w1, _ = st[last]
                _check_one(ctx, last, (L, nr, nc), (J, e, o, w0, w1), iters - 2)
    for c in ctxs:
        c.close()


def _check_one(ctx, s, shape, state, iters):
    import numpy as np
    import oracle
    J, e, o, w0, w1 = state
    for _ in range(iters):
        oracle.micsa_iteration(*shape, J, e, o, w0, w1, 16)
    for got, want in zip(ctx.download_spins(s) + ctx.download_demons(s), (e, o, w0, w1)):
        assert np.array_equal(got, want), (shape, s)
