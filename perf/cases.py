"""Workloads that time this library through its public entry points.

A case is one leg of what a spin-glass run asks for: uploading a state, drawing
its demons, iterating it, measuring it and reading it back, at lattices from
L = 8 to the headline L = 160.  Everything goes through the C ABI and its
Python binding (`micsa-ea-mc_gb300/micsa.py`), with reference-layout host
buffers, as `micsa_run` and `bench.py` use it.  Every output is a whole number.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs, context and page-locked buffers of a caller
    run(state)           one pass and its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the measured values from plain torch, where they are
                         a closed function of the inputs
"""
import ctypes as C
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "micsa-ea-mc_gb300"))
import micsa  # noqa: E402

BETA = 0.9090909090909  # the reference's input/BETAS/beta.in
L2_BYTES = 129e6  # a sample below this can stay on the chip between iterations
MOST_ATTEMPTS = 160 ** 3 * 64 * 2 * 6 * 32  # spin-flip attempts of the largest listed leg


def listed():
    return [
        # the smallest call: one iteration of one small lattice, read back
        {"name": "run_L8_one_step", "op": "run", "L": 8, "nr": 32, "ns": 1, "nc": 6, "n": 1},
        # one small job alone (the bench's L = 16 configuration), 2^10 sweeps
        {"name": "run_L16_one_job", "op": "run", "L": 16, "nr": 64, "ns": 1, "nc": 6, "n": 1024},
        # two samples at the size and replica count of the L = 24 golden run, 5 demons per site
        {"name": "run_L24_2s_nc5", "op": "run", "L": 24, "nr": 32, "ns": 2, "nc": 5, "n": 256},
        # one shape group of a batch or a server: many small samples in one context
        {"name": "run_L32_group", "op": "run", "L": 32, "nr": 64, "ns": 24, "nc": 6, "n": 256},
        # the bench's second configuration, 8 samples x 64 replicas
        {"name": "run_L64_8s", "op": "run", "L": 64, "nr": 64, "ns": 8, "nc": 6, "n": 64},
        # a server pool of its largest lattice with 32 replicas
        {"name": "run_L96_nr32", "op": "run", "L": 96, "nr": 32, "ns": 8, "nc": 6, "n": 32},
        # the headline: L = 160, 2 samples x 64 replicas
        {"name": "run_L160", "op": "run", "L": 160, "nr": 64, "ns": 2, "nc": 6, "n": 32},
        # the Metropolis branch a run starts with (nterm steps)
        {"name": "thermalise_L64", "op": "thermalise", "L": 64, "nr": 64, "ns": 2, "nc": 6, "n": 8},
        # one demon refresh of the headline state
        {"name": "refresh_L160", "op": "refresh", "L": 160, "nr": 64, "ns": 2, "nc": 6, "n": 1},
        # a measurement point with overlaps and C4(r) (MICSA_OBSERVABLES=1)
        {"name": "observables_L64", "op": "observables", "L": 64, "nr": 64, "ns": 2, "nc": 6, "n": 1},
        # resume and checkpoint: a sample's whole state up and down again
        {"name": "checkpoint_L96", "op": "checkpoint", "L": 96, "nr": 64, "ns": 1, "nc": 6, "n": 1},
        # a whole job on the reference's schedule: upload, refresh at 0 and powers of two,
        # iterate, measure, read the state back
        {"name": "job_L48", "op": "job", "L": 48, "nr": 64, "ns": 4, "nc": 6, "n": 64},
    ]


def _log_int(rng, a, b):
    return int(round(a * (b / a) ** rng.random()))


def draw(rng):
    while True:
        op = rng.choice(["run"] * 6 + ["thermalise", "refresh", "observables", "checkpoint", "job"])
        c = {"op": op, "L": 8 * _log_int(rng, 1, 20), "nr": rng.choice([32, 32, 64, 64, 64, 96, 128]),
             "ns": _log_int(rng, 1, 24), "nc": rng.choice([1, 3, 5, 6, 6, 6]), "n": 1}
        if op in ("run", "job"):
            c["n"] = _log_int(rng, 1, 1024 if op == "run" else 64)
        elif op == "thermalise":
            c["n"] = _log_int(rng, 1, 16)
        elif op == "checkpoint":
            c["ns"] = 1 + c["ns"] // 12
        V, nr, ns, nc, n = c["L"] ** 3, c["nr"], c["ns"], c["nc"], c["n"]
        dem = V * nr * ns * nc / 4
        if V * nr * ns * nc * n > MOST_ATTEMPTS or dem > 8e8:
            continue
        if op in ("checkpoint", "job") and dem > 1.6e8:
            continue
        if op == "observables" and c["L"] * V * nr * ns > 64 ** 4 * 128 * 4:
            continue
        if op == "thermalise" and V * nr * n * (2 + ns / 4) > 64 ** 3 * 64 * 8 * 10:
            continue
        if op != "refresh" and nr * ns > 3072:
            continue
        if any(all(c[k] == v for k, v in x.items() if k != "name") for x in listed()):
            continue
        return c


def _streams(rng, n):
    """n replica generator streams: one seeded stream's ring pointers, with
    random words in every ring and state."""
    p, x, _ = micsa.init_cpu_generators(int(rng.integers(1, 1 << 62)))
    prc, xo = (micsa.PRC * n).from_buffer_copy(bytes(p) * n), (micsa.Xoshiro * n).from_buffer_copy(bytes(x) * n)
    w = np.frombuffer(prc, dtype=np.uint64).reshape(n, -1)
    w[:, :256] = _words(rng, 256 * n).reshape(n, 256)
    w[:, 257] = _words(rng, n)  # zseed
    np.frombuffer(xo, dtype=np.uint64).reshape(n, -1)[:, :4] = _words(rng, 4 * n).reshape(n, 4)
    return prc, xo


def _words(rng, n):
    return rng.integers(0, 1 << 64, size=n, dtype=np.uint64)


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.int64, pin_memory=True)


def _u64(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_uint64))


def _inputs(case, seed):
    """Couplings (site bits), spins (reference words) of every sample."""
    rng = np.random.default_rng(seed)
    L, H, nr = case["L"], (case["L"] // 4) ** 3 // 2, case["nr"]
    bonds = [rng.integers(0, 2, size=(3, L ** 3), dtype=np.uint8) for _ in range(case["ns"])]
    spins = [_words(rng, 2 * H * nr).reshape(2, H * nr) for _ in range(case["ns"])]
    return rng, bonds, spins


def prepare(case, seed):
    op, L, nr, ns, nc = (case[k] for k in ("op", "L", "nr", "ns", "nc"))
    H = (L // 4) ** 3 // 2
    rng, bonds, spins = _inputs(case, seed)
    s = dict(case, ctx=micsa.Context(L, nr, ns, nc))
    ctx = s["ctx"]
    s["J"] = [micsa.pack_couplings(L, *b) for b in bonds]
    s["thr"] = micsa.thresholds(BETA)
    s["spins"] = _pinned(ns, 2, H * nr)
    s["spins"].numpy().view(np.uint64)[...] = np.stack(spins)
    for b in range(ns):
        ctx.upload_couplings(b, s["J"][b])
        micsa.check(ctx.h, micsa.lib().micsa_upload_spins(ctx.h, b, _u64(s["spins"][b, 0]), _u64(s["spins"][b, 1])), "spins")
    if op in ("checkpoint", "job"):
        s["J_host"] = _pinned(ns, 12 * H)
        s["J_host"].numpy().view(np.uint64)[...] = np.stack(s["J"])
        s["demons"] = _pinned(ns, 2, 2 * H * nc * nr)
    if op == "checkpoint":
        for b in range(ns):
            w = _words(rng, 2 * H * nc * nr)
            s["demons"][b].numpy().view(np.uint64)[...] = np.stack([w, w & _words(rng, w.size)])
    elif op == "thermalise":
        lut = np.zeros(4096, np.uint8)
        build = micsa.lib().micsa_build_lut
        build.argtypes, build.restype = [C.c_double, C.c_void_p], None
        build(BETA, lut.ctypes.data)
        ctx.set_lut(lut)
        s["te"] = rng.integers(0, 1 << 32, size=(case["n"], 8 * nr), dtype=np.uint32)
        s["keys"] = rng.integers(0, 1 << 32, size=nr, dtype=np.uint32)
    else:
        s["prc"], s["xo"] = _streams(rng, nr * ns)
        s["start"] = bytes(s["prc"]), bytes(s["xo"])
        if op != "refresh":
            ctx.refresh_demons(0, s["prc"], s["xo"], s["thr"])
    ctx.synchronize()
    return s


def _read_spins(s):
    h, lib = s["ctx"].h, micsa.lib()
    for b in range(s["ns"]):
        micsa.check(h, lib.micsa_download_spins(h, b, _u64(s["spins"][b, 0]), _u64(s["spins"][b, 1])), "download_spins")


def _read_demons(s):
    h, lib = s["ctx"].h, micsa.lib()
    for b in range(s["ns"]):
        micsa.check(h, lib.micsa_download_demons(h, b, _u64(s["demons"][b, 0]), _u64(s["demons"][b, 1])), "download_demons")


def _upload(s, demons):
    h, lib = s["ctx"].h, micsa.lib()
    for b in range(s["ns"]):
        micsa.check(h, lib.micsa_upload_couplings(h, b, _u64(s["J_host"][b])), "upload_couplings")
        micsa.check(h, lib.micsa_upload_spins(h, b, _u64(s["spins"][b, 0]), _u64(s["spins"][b, 1])), "upload_spins")
        if demons:
            micsa.check(h, lib.micsa_upload_demons(h, b, _u64(s["demons"][b, 0]), _u64(s["demons"][b, 1])), "upload_demons")


def _stream_bytes(s):
    return [np.frombuffer(x, dtype=np.uint8) for x in (s["prc"], s["xo"])]


def run(s):
    op, ctx = s["op"], s["ctx"]
    if op == "run":
        ctx.iterate(s["n"])
        out = ctx.measure()
        _read_spins(s)
        return dict(out, e_demon=out["e_demon"].view(np.int64), spins=s["spins"])
    if op == "thermalise":
        for te in s["te"]:
            ctx.monte_carlo(0, te, s["keys"])
        out = ctx.measure(demon=False)
        _read_spins(s)
        return dict(out, spins=s["spins"])
    if op == "refresh":
        ctx.refresh_demons(0, s["prc"], s["xo"], s["thr"])
        out = ctx.measure(spin=False)
        return [out["e_demon"].view(np.int64)] + _stream_bytes(s)
    if op == "observables":
        out = ctx.measure(overlap=True)
        return dict(out, e_demon=out["e_demon"].view(np.int64))
    if op == "checkpoint":
        _upload(s, True)
        _read_spins(s)
        _read_demons(s)
        return [s["spins"], s["demons"]]
    # job: the schedule of the reference's main loop, the next refresh asked for ahead
    _upload(s, False)
    C.memmove(s["prc"], s["start"][0], len(s["start"][0]))
    C.memmove(s["xo"], s["start"][1], len(s["start"][1]))
    t, n, out = 0, s["n"], []
    while t < n:
        if t & (t - 1) == 0:
            if t == 0:
                ctx.refresh_demons_async(0, s["prc"], s["xo"], s["thr"])
            else:
                ctx.refresh_commit()
            if (2 * t if t else 1) < n:
                ctx.refresh_demons_ahead(0, s["prc"], s["xo"], s["thr"])
        nxt = min(n, 2 * t if t else 1)
        ctx.iterate(nxt - t)
        t = nxt
        m = ctx.measure()
        out += [m["e_spin"], m["e_demon"].view(np.int64)]
    ctx.refresh_wait()
    _read_spins(s)
    _read_demons(s)
    return [s["spins"], s["demons"]] + _stream_bytes(s) + out


def work(case):
    """Bytes: the state in and out once per pass (samples are independent, one
    can stay on the chip for a whole leg), or once per iteration where one
    sample alone exceeds the L2; host transfers count once as device bytes.
    Operations: 32-bit logic and integer operations."""
    op, L, nr, ns, nc, n = (case[k] for k in ("op", "L", "nr", "ns", "nc", "n"))
    V = L ** 3
    spin, dem, jb = V * nr * ns / 8, V * nr * ns * nc / 4, V * ns
    update = 30 * V * nr * ns / 32  # about 30 operations per 32 replicas of a site

    def leg(n):
        times = n if (spin + dem + jb) / ns > L2_BYTES else 1
        return times * (2 * spin + 2 * dem + jb), n * nc * update

    draws = V * nr * ns * nc * 30  # 64-bit generator steps of one refresh, per demon
    if op == "run":
        b, f = leg(n)
        return {"bytes": b + 2 * spin + dem, "flops": f}
    if op == "thermalise":
        # three random words per site and replica word, shared by all samples
        return {"bytes": n * (2 * spin + jb) + 2 * spin, "flops": n * (update + V * nr * 6)}
    if op == "refresh":
        return {"bytes": dem, "flops": draws}
    if op == "observables":
        return {"bytes": spin + dem + jb, "flops": V * nr * ns / 64 * 3 * (L // 2 + 1) * 3}
    if op == "checkpoint":
        return {"bytes": 4 * spin + 4 * dem + 2 * jb, "flops": V * nr * ns * (nc + 1) / 8}
    k = n.bit_length()
    k += n & (n - 1) != 0
    b, f = leg(n)
    return {"bytes": b + k * dem + 3 * spin + dem, "flops": f + draws * k}


def _sites(L, nr, even, odd):
    """Spins (0/1, int64) as [nr, z, y, x] from the reference words: bit b of
    word h holds one site of each of the 4 x 4 x 4 blocks."""
    m = L // 4
    out = np.zeros((nr, L, L, L), np.uint8)
    h = np.arange(m ** 3 // 2)
    a2, bb, c = h % (m // 2), h // (m // 2) % m, h // (m // 2 * m)
    for p, words in ((0, even), (1, odd)):
        w = words.reshape(-1, nr)
        a = 2 * a2 + ((bb + c + p) & 1)
        for b in range(64):
            bit = ((w >> np.uint64(b)) & np.uint64(1)).astype(np.uint8)
            out[:, (b >> 4) * m + c, ((b >> 2) & 3) * m + bb, (b & 3) * m + a] = bit.T
    return out


def exact(case, seed):
    """The measured spin energies, overlaps and C4(r) of given spins, counted
    site by site in 64-bit integers.  What updates and draws leave has no
    closed form: those outputs are words and counts that stay the same."""
    L, nr, ns = case["L"], case["nr"], case["ns"]
    if case["op"] != "observables" or L * L ** 3 * nr * ns > 64 ** 4 * 128 * 2:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    _, bonds, spins = _inputs(case, seed)
    out = {"e_spin": [], "e_demon": None, "q": [], "c4": []}
    for b in range(ns):
        u = torch.from_numpy(_sites(L, nr, *spins[b])).to(dev)
        J = torch.from_numpy(bonds[b].reshape(3, L, L, L)).to(dev)
        unsat = sum((u ^ u.roll(-1, 3 - k) ^ J[k]).sum((1, 2, 3)) for k in range(3))
        out["e_spin"].append(3 * L ** 3 - 2 * unsat)
        d = u[0::2] ^ u[1::2]
        out["q"].append(L ** 3 - 2 * d.sum((1, 2, 3)))
        out["c4"].append(torch.stack([torch.stack([L ** 3 - 2 * (d ^ d.roll(-r, 3 - k)).sum((1, 2, 3)) for r in range(L // 2 + 1)], 1)
                                      for k in range(3)], 1))
    return dict({k: torch.stack(v).cpu() for k, v in out.items() if v is not None}, e_demon=None,
                e_spin=torch.stack(out["e_spin"]).cpu().to(torch.int32))
