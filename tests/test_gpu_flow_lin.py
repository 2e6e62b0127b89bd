"""The dataflow sweep on tiles of consecutive (row, x/2) units -- pairs, and
four one-word sites -- against the oracle: slabs smaller than a block, tiles
that end inside a row, slab depths that are not powers of two, one, three and
several word groups, several iterations per launch; and the division by a
multiplication that decodes its tickets."""
import ctypes as C

import numpy as np
import pytest

import micsa
from test_gpu_flow import _check, _upload
from test_gpu_parity import random_state


@pytest.mark.parametrize("d", [1, 2, 3, 5, 25, 40, 800, 9600, 65537, 2**30 + 1, 2**31 - 1])
def test_division_by_multiplication(d):
    sh = 0
    while (1 << sh) < d:
        sh += 1
    m = ((1 << (31 + sh)) + d - 1) // d
    assert m < 2**32
    top = 2**31 - 1
    ns = {0, 1, top, top // d * d, max(top // d * d - 1, 0)}
    ns |= {k * d + e for k in (1, 2, 3, 1000, top // d) for e in (-1, 0, 1) if 0 <= k * d + e <= top}
    for n in ns:
        assert (n * m) >> (31 + sh) == n // d, (n, d)


@pytest.mark.gpu
@pytest.mark.parametrize("L,nr,nc,ns,zc,pd,occ,quad,split,fit", [
    (8, 32, 6, 3, 2, 0, 4, 1, 0, 4),     # 8 units of four sites a plane
    (8, 64, 6, 2, 4, 2, 3, 0, 1, 1),     # two slabs
    (24, 64, 2, 1, 3, 2, 4, 0, 0, 8),
    (40, 32, 3, 2, 5, 2, 3, 1, 1, 2),    # 200 units
    (48, 96, 2, 2, 6, 0, 3, 0, 0, 1),    # three word groups; 2.25 tiles
    (48, 32, 3, 2, 12, 4, 4, 0, 0, 16),
    (40, 128, 3, 1, 10, 2, 3, 0, 0, 3),  # four-word vectors
    (72, 64, 1, 2, 9, 0, 4, 0, 1, 2),    # tiles that end inside a row
    (72, 32, 2, 1, 3, 0, 4, 1, 0, 5),
])
def test_consecutive_units_match_oracle(L, nr, nc, ns, zc, pd, occ, quad, split, fit, monkeypatch):
    for k, v in dict(ZC=zc, PD=pd, OCC=occ, QUAD=quad, SPLIT=split, FLOW=1, TILE="lin").items():
        monkeypatch.setenv("MICSA_SWEEP_" + k, str(v))
    monkeypatch.setenv("MICSA_FLOW_ITERS", str(fit))
    monkeypatch.setenv("MICSA_RESIDENT", "0")
    st = random_state(np.random.default_rng(L + nr + zc), L, nr, nc, ns)
    iters = L // 2 + 3 # every walk shift
    with micsa.Context(L, nr, ns, nc) as ctx:
        assert "load=flow tile=%s " % ("lin4" if quad else "lin") in ctx.tuning(), ctx.tuning()
        _upload(ctx, st)
        ctx.iterate(iters)
        ctx.synchronize()
        _check(ctx, st, L, nr, nc, iters)


@pytest.mark.gpu
def test_contexts_side_by_side_leave_the_dataflow_sweep_to_large_lattices(monkeypatch):
    monkeypatch.setenv("MICSA_TUNE_CACHE", "0")
    cfg = micsa.Config(0, 64, 64, 8, 2)
    h = C.c_void_p()
    assert micsa.lib().micsa_create_shared(C.byref(cfg), C.byref(h)) == micsa.MICSA_OK
    try:
        buf = C.create_string_buffer(1 << 16)
        assert micsa.lib().micsa_tuning_report(h, buf, C.c_size_t(len(buf))) == micsa.MICSA_OK
        head, _, rest = buf.value.decode().partition("|")
        assert "flow" not in head, head
        assert rest.split() and all(c.split("/")[4] not in ("4", "7") for c in rest.split())
    finally:
        micsa.lib().micsa_destroy(h)
