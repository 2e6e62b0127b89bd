"""Overlaps and C4(r) where the kernel's tiling has edges: lattices whose L/2
is below, at and above a chunk of 32 distances, sides that are odd multiples
of 8, one replica word, odd and even word counts, several samples with one
frozen -- against the scalar oracle, and against plain torch at a side whose
lines need more than 48 KB of shared memory.  All counts are exact."""
import os

import numpy as np
import pytest

import micsa
import oracle
from test_gpu_parity import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nr,ns", [(8, 32, 3), (8, 96, 1), (24, 64, 2), (40, 160, 1), (64, 32, 1),
                                     (72, 32, 1), (32, 128, 2)])
def test_overlap_counts_at_tile_edges(L, nr, ns):
    rng = np.random.default_rng(L + nr)
    st = random_state(rng, L, nr, 1, ns)
    with micsa.Context(L, nr, ns, 1) as ctx:
        for s, (J, e, o, *_r) in enumerate(st):
            ctx.upload_couplings(s, J)
            ctx.upload_spins(s, e, o)
        if ns > 2:
            ctx.set_active([1] * (ns - 2) + [0, 1])
        m = ctx.measure(spin=False, demon=False, overlap=True)
        for s, (J, e, o, *_r) in enumerate(st):
            if ns > 2 and s == ns - 2:
                assert not m["q"][s].any() and not m["c4"][s].any()
                continue
            q, c4 = oracle.overlap_c4(L, nr, micsa.unpack_spins(L, nr, e, o))
            assert np.array_equal(m["q"][s], q)
            assert np.array_equal(m["c4"][s], c4)


def test_overlap_counts_of_a_long_line():
    import torch
    L, nr = 248, 32
    rng = np.random.default_rng(3)
    H = (L // 4) ** 3 // 2
    e, o = (rng.integers(0, 1 << 64, size=H * nr, dtype=np.uint64) for _ in range(2))
    J = np.zeros(12 * H, np.uint64)
    old = os.environ.get("MICSA_SWEEP_ZC")
    os.environ["MICSA_SWEEP_ZC"] = "8"  # no launch-shape timing
    try:
        ctx = micsa.Context(L, nr, 1, 1)
    finally:
        if old is None:
            del os.environ["MICSA_SWEEP_ZC"]
        else:
            os.environ["MICSA_SWEEP_ZC"] = old
    with ctx:
        ctx.upload_couplings(0, J)
        ctx.upload_spins(0, e, o)
        m = ctx.measure(spin=False, demon=False, overlap=True)
    u = torch.from_numpy(micsa.unpack_spins(L, nr, e, o)).cuda().reshape(nr, L, L, L)
    d = u[0::2] ^ u[1::2]
    V = L ** 3
    assert np.array_equal(m["q"][0], (V - 2 * d.sum((1, 2, 3))).cpu().numpy())
    for axis in range(3):
        for r in (0, 1, 4, 5, 31, 32, 33, 36, 64, 95, 96, 97, 121, 123, 124):
            c = V - 2 * (d ^ d.roll(-r, 3 - axis)).sum((1, 2, 3))
            assert np.array_equal(m["c4"][0][:, axis, r], c.cpu().numpy()), (axis, r)
