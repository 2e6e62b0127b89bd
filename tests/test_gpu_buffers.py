"""Page-locked host buffers that a kernel cannot address as they are -- off
their 8-byte alignment, or page-locked in part -- take the staged path: the
states that go up and come back are those of ordinary buffers, and a buffer
that a copy refuses leaves the context usable."""
import ctypes as C

import numpy as np
import pytest

import micsa
from test_gpu_parity import random_state

pytestmark = pytest.mark.gpu


def _addr(a):
    return C.cast(C.c_void_p(a), C.POINTER(C.c_uint64))


def _unaligned_pinned(n, keep):
    """n words of page-locked memory 4 bytes off their alignment: (address, bytes)"""
    import torch
    t = torch.zeros(8 * n + 8, dtype=torch.uint8, pin_memory=True)
    keep.append(t)
    return t.data_ptr() + 4, t.numpy()[4:8 * n + 4]


@pytest.mark.parametrize("L,nr,nc", [(8, 32, 1), (16, 96, 6), (24, 64, 3)])
def test_unaligned_page_locked_buffers_are_staged(L, nr, nc):
    J, e, o, w0, w1, _ = random_state(np.random.default_rng(L + nr), L, nr, nc, 1)[0]
    keep, lib = [], micsa.lib()

    def up(a):
        at, v = _unaligned_pinned(a.size, keep)
        v[:] = a.view(np.uint8)
        return _addr(at)

    with micsa.Context(L, nr, 1, nc) as ctx:
        micsa.check(ctx.h, lib.micsa_upload_couplings(ctx.h, 0, up(J)), "couplings")
        micsa.check(ctx.h, lib.micsa_upload_spins(ctx.h, 0, up(e), up(o)), "spins")
        micsa.check(ctx.h, lib.micsa_upload_demons(ctx.h, 0, up(w0), up(w1)), "demons")
        for got, want in zip(ctx.download_spins(0) + ctx.download_demons(0), (e, o, w0, w1)):
            assert np.array_equal(got, want)
        for call, pair in ((lib.micsa_download_spins, (e, o)), (lib.micsa_download_demons, (w0, w1))):
            (a0, v0), (a1, v1) = (_unaligned_pinned(x.size, keep) for x in pair)
            micsa.check(ctx.h, call(ctx.h, 0, _addr(a0), _addr(a1)), "download")
            for v, want in zip((v0, v1), pair):
                assert np.array_equal(np.frombuffer(v.tobytes(), np.uint64), want)


def test_buffer_page_locked_in_part_is_not_read_in_place():
    """Only the first page of each array is registered: a copy from it is right
    or refused (copies may not cross a registration's end), never a kernel's
    read past the registered part."""
    import torch
    L, nr, nc = 24, 64, 3
    J, e, o, w0, w1, _ = random_state(np.random.default_rng(5), L, nr, nc, 1)[0]
    rt, page, keep, lib = torch.cuda.cudart(), 65536, [], micsa.lib()

    def part(a):
        raw = np.zeros(a.nbytes + 2 * page, np.uint8)
        off = -raw.ctypes.data % page
        v = raw[off:off + a.nbytes]
        v[:] = a.view(np.uint8)
        assert a.nbytes > page and int(rt.cudaHostRegister(raw.ctypes.data + off, page, 2)) == 0
        keep.append((raw, raw.ctypes.data + off))
        return _addr(raw.ctypes.data + off)

    with micsa.Context(L, nr, 1, nc) as ctx:
        ctx.upload_couplings(0, J)
        ctx.upload_spins(0, e, o)
        ctx.upload_demons(0, w1, w0)
        rc = lib.micsa_upload_demons(ctx.h, 0, part(w0), part(w1))
        assert rc in (micsa.MICSA_OK, micsa.MICSA_ERR_CUDA)
        if rc == micsa.MICSA_OK:
            for got, want in zip(ctx.download_demons(0), (w0, w1)):
                assert np.array_equal(got, want)
        ctx.upload_demons(0, w0, w1)
        for got, want in zip(ctx.download_spins(0) + ctx.download_demons(0), (e, o, w0, w1)):
            assert np.array_equal(got, want)
    for _, at in keep:
        rt.cudaHostUnregister(at)
