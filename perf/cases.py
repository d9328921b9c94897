"""Performance cases: the work that users of this library have it do.

Each case is one call (or, for the server, one burst of requests) through the
public entry points of cuda-pi-chudnovsky-bbp_b200/b200mul.py on operands that
are already where such a caller has them: on the GPU for the *_device calls,
batches and the server, in host memory for the host-buffer calls. Operands are
uniform random limbs with a non-zero top limb, which is what products, trees
and Newton steps in the middle of a computation look like.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) operands, output buffers, plans and handles
    run(state)          one pass, returning its whole outputs
    work(case)          bytes (and floating-point operations: none) of one pass
    exact(case, seed)   what run returns, from numpy and Python integers alone

Every value is an integer, so results are compared bit for bit.
"""
import math
import os
import sys
import weakref

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-pi-chudnovsky-bbp_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)


def _lib():
    import b200mul

    b200mul.init(0)
    return b200mul


# ---- cases -----------------------------------------------------------------------


def listed():
    return [
        # One product of small device-resident operands: the leaves of a
        # caller's own product tree, where the call itself is the cost.
        {"name": "mul_200x150", "kind": "mul", "na": 200, "nb": 150},
        # A product that still fits one CTA (the size of the smoke check).
        {"name": "mul_3000x1234", "kind": "mul", "na": 3000, "nb": 1234},
        # The reference self-test's large product, 60,000 x 60,000 limbs.
        {"name": "mul_60000", "kind": "mul", "na": 60000, "nb": 60000},
        # Unbalanced and odd: a long number times a shorter one, as in the
        # upper levels of uneven trees and in number-times-reciprocal steps.
        {"name": "mul_1000003x131071", "kind": "mul", "na": 1000003, "nb": 131071},
        # A square (the same operand twice) of a few million limbs, as in
        # Newton steps and powers; its length is not a power of two.
        {"name": "square_3000001", "kind": "square", "na": 3000001},
        # The benchmark's product: 2^24 x 2^24 limbs on the device.
        {"name": "mul_16777216", "kind": "mul", "na": 1 << 24, "nb": 1 << 24},
        # The reference's own call shape: host arrays in, host array out.
        {"name": "host_700001x600000", "kind": "host", "na": 700001, "nb": 600000},
        # The benchmark's batch: 4,096 independent products, both lengths
        # log-uniform in 64..65,536 limbs, planned once and replayed.
        {"name": "batch_4096", "kind": "batch", "jobs": 4096, "lo": 64, "hi": 65536},
        # Floor division with remainder, a two-to-one division of the length
        # that a few million decimal digits need.
        {"name": "divmod_400003x200001", "kind": "divmod", "na": 400003, "nb": 200001},
        # Decimal conversion of a one-million-digit integer.
        {"name": "decimal_103810", "kind": "decimal", "na": 103810},
        # One million digits of pi: tree, square root, division, decimal.
        {"name": "pi_1000000", "kind": "pi", "digits": 1000000},
        # The server under a burst: 128 requests of mixed sizes submitted at
        # once and waited for (eight to a dispatch, as the benchmark runs it).
        {"name": "serve_128", "kind": "serve", "requests": 128, "lo": 1024, "hi": 1 << 20},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["mul", "mul", "mul", "mul", "square", "host", "batch", "divmod", "isqrt", "decimal", "pi",
                       "serve"])
    if kind == "mul":
        return {"kind": kind, "na": _log_uniform(rng, 16, 1 << 24), "nb": _log_uniform(rng, 16, 1 << 24)}
    if kind == "square":
        return {"kind": kind, "na": _log_uniform(rng, 16, 1 << 24)}
    if kind == "host":
        return {"kind": kind, "na": _log_uniform(rng, 64, 1 << 20), "nb": _log_uniform(rng, 64, 1 << 20)}
    if kind == "batch":
        return {"kind": kind, "jobs": _log_uniform(rng, 64, 4096), "lo": 64, "hi": _log_uniform(rng, 2048, 65536)}
    if kind == "divmod":
        nb = _log_uniform(rng, 256, 250000)
        return {"kind": kind, "na": nb + _log_uniform(rng, 128, 250000), "nb": nb}
    if kind == "isqrt":
        return {"kind": kind, "na": _log_uniform(rng, 256, 500000)}
    if kind == "decimal":
        return {"kind": kind, "na": _log_uniform(rng, 256, 150000)}
    if kind == "pi":
        return {"kind": kind, "digits": _log_uniform(rng, 10000, 1000000)}
    return {"kind": kind, "requests": _log_uniform(rng, 16, 128), "lo": 1024, "hi": _log_uniform(rng, 1 << 14, 1 << 20)}


# ---- inputs ----------------------------------------------------------------------


def _operand(rng, n):
    a = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    a[-1] |= 1
    return a


def _pairs(case):
    """Sizes of a batch's or burst's products: fixed by the case, so that
    every seed runs the same work on other operands."""
    n = case.get("jobs") or case["requests"]
    rng = np.random.default_rng(n * 1000003 + case["hi"])
    lens = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), (n, 2)))
    return [(int(x), int(y)) for x, y in np.clip(lens, case["lo"], case["hi"])]


def _operands(case, seed):
    """Host operands of a case, from the seed alone."""
    rng = np.random.default_rng([seed, 7])
    kind = case["kind"]
    if kind in ("mul", "host", "divmod"):
        return [_operand(rng, case["na"]), _operand(rng, case["nb"])]
    if kind in ("square", "isqrt", "decimal"):
        return [_operand(rng, case["na"])]
    if kind in ("batch", "serve"):
        out = []
        for na, nb in _pairs(case):
            out += [_operand(rng, na), _operand(rng, nb)]
        return out
    return []


def _digits(case, seed):
    """Digits of a pi case: the seed takes less than 0.1 percent off the count
    (the unused end of the output buffer stays zero)."""
    return case["digits"] - seed % max(1, case["digits"] // 1000)


def _decimal_room(case):
    """Bytes that hold the decimal digits of any integer of the case's length."""
    return int(case["na"] * 32 * math.log10(2)) + 2


def _dev(a):
    return torch.from_numpy(a.view(np.int32)).cuda()


def _offsets(lens):
    """Start of each buffer, every one 256-byte aligned, and the total."""
    offs, tot = [], 0
    for n in lens:
        offs.append(tot)
        tot += (n + 63) // 64 * 64
    return offs, tot


class _Server:
    """A running server that stops when the state that holds it goes away."""

    def __init__(self, lib):
        self.server = lib.Server(hbm_budget_bytes=4 << 30, streams=4, max_batch=8)
        self._stop = weakref.finalize(self, self.server.stop)


def prepare(case, seed):
    lib = _lib()
    kind = case["kind"]
    st = {"kind": kind, "lib": lib}
    if kind == "pi":
        st["digits"] = _digits(case, seed)
        st["out"] = np.zeros(case["digits"] + 2, np.uint8)
        return st
    ops = _operands(case, seed)
    if kind == "host":
        st["a"], st["b"] = (torch.from_numpy(x.view(np.int32)).pin_memory().numpy().view(np.uint32) for x in ops)
        st["out"] = torch.zeros(sum(x.size for x in ops), dtype=torch.int32).pin_memory().numpy().view(np.uint32)
        return st
    if kind in ("batch", "serve"):
        offs, tot = _offsets([x.size for x in ops])
        flat = np.zeros(tot, np.uint32)
        for o, x in zip(offs, ops):
            flat[o:o + x.size] = x
        pairs = _pairs(case)
        oo, otot = _offsets([na + nb for na, nb in pairs])
        st["ops"] = _dev(flat)
        st["out"] = torch.zeros(otot, dtype=torch.int32, device="cuda")
        base, obase = st["ops"].data_ptr(), st["out"].data_ptr()
        jobs = [(base + 4 * offs[2 * i], na, base + 4 * offs[2 * i + 1], nb, obase + 4 * oo[i], na + nb)
                for i, (na, nb) in enumerate(pairs)]
        if kind == "batch":
            st["lens"] = torch.zeros(len(jobs), dtype=torch.int64, device="cuda")
            lbase = st["lens"].data_ptr()
            st["batch"] = lib.Batch([j + (lbase + 8 * i,) for i, j in enumerate(jobs)], lib.BATCH_GRAPH)
        else:
            st["jobs"] = jobs
            st["server"] = _Server(lib)
        torch.cuda.synchronize()
        return st
    dev = [_dev(x) for x in ops]
    st["ops"] = dev
    if kind in ("mul", "square"):
        st["out"] = torch.zeros(case["na"] + case.get("nb", case["na"]), dtype=torch.int32, device="cuda")
        st["len"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    elif kind == "divmod":
        st["q"] = torch.zeros(case["na"] - case["nb"] + 1, dtype=torch.int32, device="cuda")
        st["r"] = torch.zeros(case["nb"], dtype=torch.int32, device="cuda")
    elif kind == "decimal":
        st["text"] = np.zeros(_decimal_room(case), np.uint8)
    elif kind == "isqrt":
        st["out"] = torch.zeros((case["na"] + 1) // 2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return st


# ---- one pass --------------------------------------------------------------------


def run(st):
    lib, kind = st["lib"], st["kind"]
    if kind == "pi":
        text = lib.compute_pi(st["digits"]).encode()
        st["out"][:len(text)] = np.frombuffer(text, np.uint8)
        return st["out"]
    if kind == "host":
        return lib.mul_ntt_cuda(st["a"], st["b"], out=st["out"])
    stream = torch.cuda.current_stream().cuda_stream
    if kind in ("mul", "square"):
        a, b = st["ops"][0], st["ops"][-1]
        lib.mul_device(a.data_ptr(), a.numel(), b.data_ptr(), b.numel(), st["out"].data_ptr(), st["out"].numel(),
                       st["len"].data_ptr(), stream)
        return st["out"], st["len"]
    if kind == "batch":
        st["batch"].launch(stream)
        return st["out"], st["lens"]
    if kind == "divmod":
        (a, b), q, r = st["ops"], st["q"], st["r"]
        ql, rl = lib.divmod_device(a.data_ptr(), a.numel(), b.data_ptr(), b.numel(), q.data_ptr(), q.numel(),
                                   r.data_ptr(), r.numel(), stream)
        q[ql:], r[rl:] = 0, 0
        return q, r
    if kind == "isqrt":
        a, out = st["ops"][0], st["out"]
        out[lib.isqrt_device(a.data_ptr(), a.numel(), out.data_ptr(), out.numel(), stream):] = 0
        return out
    if kind == "decimal":
        a = st["ops"][0]
        text = lib.to_decimal_device(a.data_ptr(), a.numel(), stream).encode()
        st["text"][:] = 0
        st["text"][:len(text)] = np.frombuffer(text, np.uint8)
        return st["text"]
    srv = st["server"].server
    tickets = [srv.submit(na, nb, a=a, b=b, out=out, out_cap=cap) for a, na, b, nb, out, cap in st["jobs"]]
    results = [srv.wait(t, 60.0) for t in tickets]
    for t in tickets:
        srv.release(t)
    return st["out"], np.array([r.out_len for r in results], np.int64), \
        np.array([r.state for r in results], np.int64)


# ---- what a pass cannot do without ------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind in ("mul", "host"):
        n = 2 * (case["na"] + case["nb"])
    elif kind == "square":
        n = 3 * case["na"]
    elif kind in ("batch", "serve"):
        n = sum(2 * (na + nb) for na, nb in _pairs(case))
    elif kind == "divmod":
        n = 2 * (case["na"] + case["nb"])
    elif kind == "isqrt":
        n = case["na"] + case["na"] // 2
    elif kind == "decimal":
        return {"bytes": 4 * case["na"] + int(case["na"] * 32 * math.log10(2)), "flops": 0}
    else:
        return {"bytes": case["digits"], "flops": 0}
    return {"bytes": 4 * n, "flops": 0}


# ---- exact results ---------------------------------------------------------------


def _int(limbs):
    return int.from_bytes(np.ascontiguousarray(limbs, "<u4").tobytes(), "little")


def _limbs(x, n=None):
    n = (x.bit_length() + 31) // 32 if n is None else n
    return np.frombuffer(x.to_bytes(4 * n, "little"), np.uint32)


def _product(a, b):
    """a * b as len(a) + len(b) limbs: Python integers when short, else 8-bit
    digits through a float64 FFT (coefficients below 2^40 here, so rounding
    to the nearest integer is exact) and an integer carry."""
    n = a.size + b.size
    if min(a.size, b.size) <= 4096:
        return _limbs(_int(a) * _int(b), n)
    size = 1 << (4 * n - 1).bit_length()
    fa = np.fft.rfft(np.ascontiguousarray(a).view(np.uint8).astype(np.float64), size)
    fa *= np.fft.rfft(np.ascontiguousarray(b).view(np.uint8).astype(np.float64), size)
    c = np.rint(np.fft.irfft(fa, size)[:4 * n]).astype(np.int64)
    total = sum(_int(((c >> (8 * k)) & 0xFF).astype(np.uint8).view(np.uint32)) << (8 * k) for k in range(6))
    return _limbs(total, n)


def _trimmed(p):
    nz = np.flatnonzero(p)
    return int(nz[-1]) + 1 if nz.size else 0


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mul", "host", "square"):
        if case["na"] + case.get("nb", case["na"]) > 1 << 22:
            return None
        ops = _operands(case, seed)
        p = _product(ops[0], ops[-1])
        n = _trimmed(p)
        return p[:n] if kind == "host" else (p.view(np.int32), np.array([n], np.int64))
    if kind in ("batch", "serve"):
        pairs = _pairs(case)
        if sum(na + nb for na, nb in pairs) > 1 << 22:
            return None
        ops = _operands(case, seed)
        oo, otot = _offsets([na + nb for na, nb in pairs])
        out, lens = np.zeros(otot, np.uint32), np.zeros(len(pairs), np.int64)
        for i, (na, nb) in enumerate(pairs):
            p = _product(ops[2 * i], ops[2 * i + 1])
            out[oo[i]:oo[i] + p.size] = p
            lens[i] = _trimmed(p)
        if kind == "batch":
            return out.view(np.int32), lens
        return out.view(np.int32), lens, np.full(len(pairs), 2, np.int64)
    if kind == "pi" or case["na"] > 20000:
        return None
    ops = _operands(case, seed)
    if kind == "divmod":
        q, r = divmod(_int(ops[0]), _int(ops[1]))
        return _limbs(q, case["na"] - case["nb"] + 1).view(np.int32), _limbs(r, case["nb"]).view(np.int32)
    if kind == "isqrt":
        return _limbs(math.isqrt(_int(ops[0])), (case["na"] + 1) // 2).view(np.int32)
    limit = sys.get_int_max_str_digits()
    sys.set_int_max_str_digits(0)
    try:
        text = np.zeros(_decimal_room(case), np.uint8)
        digits = np.frombuffer(str(_int(ops[0])).encode(), np.uint8)
        text[:digits.size] = digits
        return text
    finally:
        sys.set_int_max_str_digits(limit)
