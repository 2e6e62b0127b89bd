"""Demon draws at the edge of a comparison.  The GPU decides a draw from the
high halves of its terms and draws a word again in full where those leave it
open; random streams meet that once in 10^8 draws.  Here the first draw of
every stream is put where it matters -- the draw is linear in the
congruential state, so any 64-bit value can be had -- next to each threshold,
next to 0 and next to 2^64, with thresholds of ordinary and extreme values,
and every word and stream byte must equal the host's."""
import ctypes as C

import numpy as np
import pytest

import micsa
from test_gpu_refresh import _copy, _host_draw, _streams

pytestmark = pytest.mark.gpu

A = 3202034522624059733  # random_generator.h:66
M64 = 1 << 64


def _first_draw(prc, xo):
    """The 64-bit value of a stream's next draw (the stream is left as it is)."""
    p, x = _copy((micsa.PRC * 1).from_buffer_copy(prc), micsa.PRC), micsa.Xoshiro.from_buffer_copy(xo)
    ira, ip = list(p[0].ira), p[0].ip
    at = lambda k: ira[(ip - k) & 255]
    xn = (at(24) + at(55)) % M64
    pr = xn ^ at(61)
    z = (p[0].zseed * A + 1) % M64
    s = list(x.s)
    v = (s[0] + s[3]) % M64
    return (z + pr + (((v << 23) | (v >> 41)) % M64 + s[0])) % M64


@pytest.mark.parametrize("thr", [
    None, (3 << 62, 1 << 63, 1 << 62), (0, 0, 0), (M64 - 1, M64 - 1, M64 - 1), (M64 - 1, 1, 0),
    (0xFFFFFFFF << 32, (1 << 32) + 5, 1 << 32), (5, 0xFFFFFFFE00000007, 0x7FFFFFFF80000000),
    ((1 << 32) - 1, 0x80000000FFFFFFFF, 2 << 32)])
def test_draws_next_to_a_threshold_and_to_the_wrap(thr):
    L, nr, nc, ns = 8, 64, 2, 2
    thr = micsa.thresholds(0.9090909090909) if thr is None else np.array(thr, np.uint64)
    prc, xo = _streams(ns * nr, 77)
    rng = np.random.default_rng(5)
    # high halves around every threshold's and around 0 = 2^32; low halves at the
    # threshold's, around it, at the ends and random
    want = []
    for t in list(map(int, thr)) + [0]:
        for dh in range(-5, 3):
            lo = [t & 0xFFFFFFFF, (t - 1) & 0xFFFFFFFF, (t + 1) & 0xFFFFFFFF, int(rng.integers(1 << 32))]
            want += [((((t >> 32) + dh) % (1 << 32)) << 32) | v for v in lo]
    assert len(want) == ns * nr
    inv = pow(A, -1, M64)
    for i, e in enumerate(want):
        now = _first_draw(prc[i], xo[i])
        prc[i].zseed = (prc[i].zseed + (e - now) * inv) % M64
        assert _first_draw(prc[i], xo[i]) == e
    hp, hx = _copy(prc, micsa.PRC), _copy(xo, micsa.Xoshiro)
    with micsa.Context(L, nr, ns, nc) as ctx:
        ctx.refresh_demons(0, prc, xo, thr)
        for s in range(ns):
            w0, w1 = _host_draw(L, nr, nc, hp, hx, s, thr)
            # the first draw is bit 0 of word 0: D = number of thresholds above it
            d = [(int(w0[r]) & 1) + 2 * (int(w1[r]) & 1) for r in range(nr)]
            assert d == [sum(e < int(t) for t in thr) for e in want[s * nr:(s + 1) * nr]]
            g0, g1 = ctx.download_demons(s)
            assert np.array_equal(g0, w0) and np.array_equal(g1, w1)
        assert bytes(prc) == bytes(hp) and bytes(xo) == bytes(hx)
