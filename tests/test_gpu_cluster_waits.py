"""The bounded waits of the cluster exchange (resident kernel, L = 16 to 32).
With the waits' barriers held open and a 1 ms limit every wait runs out; the
launch ends, and the next call of that context that waits for its stream --
synchronize, measure, a download, the mixed launch's synchronize -- reports it,
once; other contexts neither report it nor lose their results.  With the waits
restored the same context runs bit-exact again.  Nothing faults or hangs."""
import numpy as np
import pytest

import micsa
from test_gpu_parity import random_state
from test_gpu_resident_cluster import _ctx, _same

pytestmark = pytest.mark.gpu


def _upload(c, st):
    for s, (J, e, o, w0, w1, _) in enumerate(st):
        c.upload_spins(s, e, o)
        c.upload_demons(s, w0, w1)


@pytest.mark.parametrize("L,C,nr,nc,ns", [(16, 2, 64, 6, 2), (16, 8, 32, 3, 1), (24, 4, 32, 6, 2), (24, 8, 64, 5, 1),
                                          (32, 8, 64, 6, 2)])
def test_exchange_that_runs_out_is_reported_once_and_by_its_own_context(L, C, nr, nc, ns):
    st = random_state(np.random.default_rng(L + C), L, nr, nc, ns)
    a = _ctx(L, nr, ns, nc, {"MICSA_RESIDENT_CTAS": str(C)}, st)
    b = _ctx(L, nr, ns, nc, {"MICSA_RESIDENT_CTAS": str(C)}, st)
    ref = _ctx(L, nr, ns, nc, {"MICSA_RESIDENT": "0"}, st)
    lib = micsa.lib()
    calls = [lambda: micsa.check(a.h, lib.micsa_synchronize(a.h), "synchronize"), lambda: a.measure(),
             lambda: a.download_spins(0), lambda: a.download_demons(ns - 1)]
    for call in calls:
        assert lib.micsa_debug_flow_waits(a.h, 1000000, 1) == micsa.MICSA_OK
        try:
            a.iterate(3)
            b.iterate(2)
            b.synchronize()  # not b's to report, and b's own waits go on
            with pytest.raises(micsa.MicsaError, match="timed out"):
                call()
            a.synchronize()  # reported once
        finally:
            assert lib.micsa_debug_flow_waits(a.h, 0, 0) == micsa.MICSA_OK
    ref.iterate(2 * len(calls))
    _same(b, ref, ns, "beside")
    _upload(a, st)
    a.iterate(2 * len(calls))
    a.synchronize()
    _same(a, ref, ns, "restored")
    for c in (a, b, ref):
        c.close()


def test_mixed_launch_reports_its_resident_groups():
    st = [random_state(np.random.default_rng(k), L, 64, 6, 1) for k, L in enumerate((32, 48))]
    a, b = (_ctx(L, 64, 1, 6, {}, s) for L, s in zip((32, 48), st))
    lib = micsa.lib()
    with micsa.Multi([a, b]) as multi:
        assert "L32:resident" in multi.report()
        assert lib.micsa_debug_flow_waits(a.h, 1000000, 1) == micsa.MICSA_OK
        try:
            # the mixed launch's own waits, on the device-wide setting, as they were
            assert lib.micsa_debug_flow_waits(b.h, 0, 0) == micsa.MICSA_OK
            multi.iterate(4)
            with pytest.raises(micsa.MicsaError, match="group 0: .*timed out"):
                multi.synchronize()
            multi.synchronize()  # once
        finally:
            assert lib.micsa_debug_flow_waits(a.h, 0, 0) == micsa.MICSA_OK
    for c in (a, b):
        c.close()
