"""Heat-bath bits where the threshold search has edges: LUTs of hot and cold
temperatures, thresholds that fill every bin of the prebisection table (every
draw bisected, the waiting draws of a warp at their most), equal thresholds,
thresholds on bin borders, and replica counts whose counters travel with the
launch (192) or through device arrays (224) -- Metropolis steps against the
oracle, bit for bit."""
import struct

import numpy as np
import pytest

import micsa
import oracle
import runs
from test_gpu_parity import random_state

pytestmark = pytest.mark.gpu


def _lut(thr, pre=None):
    """4096 bytes: 256 thresholds as (high, low), 1024 x (min | max << 8)."""
    thr = [int(t) for t in thr]
    if pre is None:  # first threshold above the bin's first and last value
        pre = []
        for b in range(1024):
            lo, hi = b << 54, ((b + 1) << 54) - 1
            pre.append(tuple(min(255, sum(t <= u for t in thr)) for u in (lo, hi)))
    w = b"".join(struct.pack("<II", t >> 32, t & 0xFFFFFFFF) for t in thr)
    return w + b"".join(struct.pack("<H", a | (b << 8)) for a, b in pre)


M = 1 << 64
LUTS = {
    "beta 0.1": runs.lut_bytes(0.1)[8:], "beta 1.5": runs.lut_bytes(1.5)[8:],
    "uniform": _lut([(i + 1) * (M // 256) - 1 for i in range(256)]),
    "one bin": _lut([(5 << 54) + (i << 40) for i in range(255)] + [M - 1]),
    "borders": _lut([(4 * i + 1) << 54 for i in range(255)] + [M - 1]),
    "equal": _lut([1 << 63] * 255 + [M - 1]),
    "whole range": _lut([(i + 1) * (M // 256) - 1 for i in range(256)], [(0, 255)] * 1024),
}


@pytest.mark.parametrize("name", list(LUTS))
def test_metropolis_with_any_lut(name):
    L, nr = 16, 32
    rng = np.random.default_rng(9)
    (J, e, o, *_r), = random_state(rng, L, nr, 1, 1)
    keys = rng.integers(0, 1 << 32, size=nr, dtype=np.uint32)
    with micsa.Context(L, nr, 1, 1) as ctx:
        ctx.set_lut(LUTS[name])
        ctx.upload_couplings(0, J)
        ctx.upload_spins(0, e, o)
        for _ in range(2):
            te = rng.integers(0, 1 << 32, size=8 * nr, dtype=np.uint32)
            ctx.monte_carlo(0, te, keys)
            oracle.metropolis_iteration(L, nr, J, e, o, te[:4 * nr].copy(), te[4 * nr:].copy(), keys,
                                        LUTS[name])
        ge, go = ctx.download_spins(0)
        assert np.array_equal(ge, e) and np.array_equal(go, o)


@pytest.mark.parametrize("L,nr", [(8, 192), (8, 224), (40, 96), (32, 64)])
def test_metropolis_replica_counts(L, nr):
    rng = np.random.default_rng(L + nr)
    lut = runs.lut_bytes()[8:]
    (J, e, o, *_r), = random_state(rng, L, nr, 1, 1)
    keys = rng.integers(0, 1 << 32, size=nr, dtype=np.uint32)
    with micsa.Context(L, nr, 1, 1) as ctx:
        ctx.set_lut(lut)
        ctx.upload_couplings(0, J)
        ctx.upload_spins(0, e, o)
        for _ in range(2):
            te = rng.integers(0, 1 << 32, size=8 * nr, dtype=np.uint32)
            ctx.monte_carlo(0, te, keys)
            te[:] = 0  # the call has taken its counters
        rng = np.random.default_rng(L + nr)
        random_state(rng, L, nr, 1, 1)
        rng.integers(0, 1 << 32, size=nr, dtype=np.uint32)
        for _ in range(2):
            te = rng.integers(0, 1 << 32, size=8 * nr, dtype=np.uint32)
            oracle.metropolis_iteration(L, nr, J, e, o, te[:4 * nr].copy(), te[4 * nr:].copy(), keys, lut)
        ge, go = ctx.download_spins(0)
        assert np.array_equal(ge, e) and np.array_equal(go, o)


@pytest.mark.parametrize("L,nr", [(8, 32), (40, 64), (48, 64), (16, 224)])  # 1, 125, 216 and 28 blocks
def test_steps_back_to_back(L, nr):
    """Steps queued one behind another, the bits of one colour drawn while the
    sweep of the other still runs, by blocks of one word each (up to one block
    per SM) or of all three."""
    rng = np.random.default_rng(L * nr)
    lut = runs.lut_bytes()[8:]
    (J, e, o, *_r), = random_state(rng, L, nr, 1, 1)
    keys = rng.integers(0, 1 << 32, size=nr, dtype=np.uint32)
    te = rng.integers(0, 1 << 32, size=(6, 8 * nr), dtype=np.uint32)
    with micsa.Context(L, nr, 1, 1) as ctx:
        ctx.set_lut(lut)
        ctx.upload_couplings(0, J)
        ctx.upload_spins(0, e, o)
        for t in te:
            ctx.monte_carlo(0, t, keys)
        for t in te:
            oracle.metropolis_iteration(L, nr, J, e, o, t[:4 * nr].copy(), t[4 * nr:].copy(), keys, lut)
        ge, go = ctx.download_spins(0)
        assert np.array_equal(ge, e) and np.array_equal(go, o)
