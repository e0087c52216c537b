"""The workloads this engine is timed on, each through the public entry points.

``listed()`` names twelve of them, ``draw(rng)`` gives more of the same ranges.
A case is a dict of plain values; ``prepare(case, seed)`` makes its inputs on
the GPU, ``run(state)`` is one pass, ``work(case)`` the bytes and operations
the pass cannot do without, and ``exact(case, seed)`` its result from plain
Python integers or torch in 64 bits where that is quick.

Words are little-endian base 2^32, held in int32 tensors.
"""
from __future__ import annotations

import ctypes as C
import math
import random
import sys

import numpy as np
import torch

import piculator_b200 as P

# longest transform of the drawn NTT.h / FFT.h flows, longest drawn product
NTT_K, FFT_K, MUL_WORDS = (12, 24), (12, 21), (64, 1 << 24)


def listed():
    return [
        # Pi() as the command line runs it, the reference's text in host
        # memory.  10^4 digits: the smallest run of the tests, latency and
        # launches only; 10^6: the reference's quick run.
        {"name": "pi_10k", "op": "pi_text", "digits": 10_000},
        {"name": "pi_1m", "op": "pi_text", "digits": 1_000_000},
        # Pi() with the number left on the device (pic_pi_compute): the
        # benchmark's 10^8 and headline 10^9 digits.
        {"name": "pi_100m", "op": "pi", "digits": 100_000_000},
        {"name": "pi_1g", "op": "pi", "digits": 1_000_000_000},
        # Exact products of device words (pic_mul, tuned choice): the
        # benchmark's short 2^12-word product, an uneven one of odd lengths as
        # a truncated BigFloat::mul forms them, and the long 2^24-word one.
        {"name": "mul_4k", "op": "mul", "na": 4096, "nb": 4096},
        {"name": "mul_uneven", "op": "mul", "na": 1_048_573, "nb": 400_009},
        {"name": "mul_16m", "op": "mul", "na": 1 << 24, "nb": 1 << 24},
        # Many independent products in one call, log-uniform 1 .. 8192 words
        # (the benchmark's 8192 of them): a caller's own splitting tree.
        {"name": "mul_batch", "op": "batch", "count": 8192, "longest": 8192, "sizes": 7},
        # BigFloat division and inverse square root at one odd precision, the
        # Newton phases of Pi() used by themselves.
        {"name": "newton_300k", "op": "newton", "p": 300_007},
        # Decimal text of a number (to_string_dec).
        {"name": "to_dec_1m", "op": "dec", "digits": 1_000_000},
        # The drop-in C flows of NTT.h and FFT.h: convert two numbers, forward
        # both, multiply pointwise, back, convert to words.
        {"name": "ntt_flow_k22", "op": "ntt", "k": 22, "na": 1_048_571, "nb": 1_000_003},
        {"name": "fft_flow_k20", "op": "fft", "k": 20, "na": 131_071, "nb": 130_003},
    ]


def _between(rng, lo, hi):
    """Log-uniform whole number of [lo, hi]."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    op = rng.choice(["pi_text", "pi", "mul", "mul", "mul", "batch", "newton", "dec", "ntt", "fft"])
    if op == "pi_text":
        return {"op": op, "digits": _between(rng, 10_000, 3_000_000)}
    if op == "pi":
        return {"op": op, "digits": _between(rng, 100_000, 400_000_000)}
    if op == "mul":
        na = _between(rng, *MUL_WORDS)
        return {"op": op, "na": na, "nb": na if rng.random() < 0.3 else _between(rng, max(64, na // 16), na)}
    if op == "batch":
        return {"op": op, "count": _between(rng, 16, 8192), "longest": _between(rng, 256, 8192),
                "sizes": rng.randrange(1 << 20)}
    if op == "newton":
        return {"op": op, "p": _between(rng, 1000, 4_000_000)}
    if op == "dec":
        return {"op": op, "digits": _between(rng, 10_000, 5_000_000)}
    k = rng.randint(*(NTT_K if op == "ntt" else FFT_K))
    zw = 1 << (k - 1 if op == "ntt" else k - 2)  # words the transform's points hold
    na = rng.randint(zw // 4, zw // 2)
    return {"op": op, "k": k, "na": na, "nb": rng.randint(zw // 4, zw - na)}


# ---- inputs ------------------------------------------------------------------
def _words(n, seed):
    """n uniform words on the GPU, the top one nonzero."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    w[-1] |= 1
    return w


def _digits(case, seed):
    """The digit count itself is Pi()'s input: each seed asks for a few digits fewer."""
    return case["digits"] - seed * 7919 % max(61, case["digits"] // 4096)


def _batch_sizes(case):
    r = random.Random(case["sizes"])
    return [(_between(r, 1, case["longest"]), _between(r, 1, case["longest"])) for _ in range(case["count"])]


def _number(words):
    """A fraction with `words` as its digits: the top word above the point."""
    return P.DeviceBigFloat.from_words(True, 1 - words.numel(), words.cpu().numpy().view(np.uint32))


def _room(p):
    """Room for a product of two operands of p words and their guard words."""
    return torch.zeros(2 * p + 8, dtype=torch.int32, device="cuda")


def _ready():
    if not P._initialised:
        P.init(0)


def prepare(case, seed):
    _ready()
    op = case["op"]
    if op == "pi_text":
        # pic_pi_hex's buffer, as a C caller keeps it
        return {"op": op, "digits": _digits(case, seed), "text": np.zeros(P.pi_sizes(case["digits"])[0] + 64, np.uint8)}
    if op == "pi":
        return {"op": op, "digits": _digits(case, seed), "out": _room(P.pi_sizes(case["digits"])[1])}
    if op == "mul":
        a, b = _words(case["na"], 2 * seed), _words(case["nb"], 2 * seed + 1)
        return {"op": op, "a": a, "b": b, "z": torch.empty(a.numel() + b.numel(), dtype=torch.int32, device="cuda")}
    if op == "batch":
        sizes = _batch_sizes(case)
        total = sum(na + nb for na, nb in sizes)
        x = _words(total, seed)
        z = torch.empty(total, dtype=torch.int32, device="cuda")
        descs, at = (P.MulDesc * len(sizes))(), 0
        for i, (na, nb) in enumerate(sizes):
            descs[i] = P.MulDesc(z.data_ptr() + 4 * at, x.data_ptr() + 4 * at, x.data_ptr() + 4 * (at + na), na, nb)
            at += na + nb
        return {"op": op, "descs": descs, "x": x, "z": z}
    if op == "newton":
        p = case["p"]
        a, b = _words(p, 2 * seed), _words(p, 2 * seed + 1)
        return {"op": op, "p": p, "a": _number(a), "b": _number(b), "x": 10005 + seed % 1000, "out": [_room(p), _room(p)]}
    if op == "dec":
        return {"op": op, "digits": case["digits"], "a": _number(_words(_dec_words(case["digits"]), seed))}
    k = case["k"]
    a, b = _words(case["na"], 2 * seed), _words(case["nb"], 2 * seed + 1)
    kind = torch.int64 if op == "ntt" else torch.complex128
    return {"op": op, "k": k, "a": a, "b": b, "ta": torch.empty(1 << k, dtype=kind, device="cuda"),
            "tb": torch.empty(1 << k, dtype=kind, device="cuda"),
            "z": torch.empty(a.numel() + b.numel(), dtype=torch.int32, device="cuda")}


def _dec_words(digits):
    return int(digits * math.log2(10) / 32) + 4


# ---- one pass ----------------------------------------------------------------
def _to(out, number):
    """A BigFloat's sign, exponent, length and words, the words into the tensor `out`."""
    sign, exp, n = number.info()
    P.check(P.lib().pic_bf_to_device(number.h, out.data_ptr(), out.numel(), None))
    return [int(sign), exp, n, out]


def run(state):
    op, lib = state["op"], P.lib()
    if op == "pi_text":
        text, n = state["text"], C.c_size_t(0)
        P.check(lib.pic_pi_hex(state["digits"], P.PI_CHOSEN, C.cast(text.ctypes.data, C.c_char_p), text.size, C.byref(n), None))
        return [n.value, text]
    if op == "pi":
        h = C.c_void_p()
        P.check(lib.pic_pi_compute(state["digits"], P.PI_CHOSEN, C.byref(h), None))
        return _to(state["out"], P.DeviceBigFloat(h.value))
    if op == "mul":
        a, b, z = state["a"], state["b"], state["z"]
        P.mul_dev(z.data_ptr(), a.data_ptr(), a.numel(), b.data_ptr(), b.numel())
        return z
    if op == "batch":
        P.check(lib.pic_mul_batch(state["descs"], len(state["descs"]), P.MUL_AUTO, None))
        return state["z"]
    if op == "newton":
        q = state["a"].div(state["b"], state["p"])
        r = P.DeviceBigFloat.invsqrt(state["x"], state["p"])
        return {"div": _to(state["out"][0], q), "invsqrt": _to(state["out"][1], r)}
    if op == "dec":
        return np.frombuffer(state["a"].to_dec(state["digits"]), dtype=np.uint8)
    k, a, b, ta, tb, z = (state[n] for n in ("k", "a", "b", "ta", "tb", "z"))
    load, forward, pointwise, inverse, store = (
        (lib.pic_int_to_ntt, lib.pic_ntt_forward, lib.pic_ntt_pointwise, lib.pic_ntt_inverse, lib.pic_ntt_to_int)
        if op == "ntt" else
        (lib.pic_int_to_fft, lib.pic_fft_forward, lib.pic_fft_pointwise, lib.pic_fft_inverse, lib.pic_fft_to_int))
    for t, x in ((ta, a), (tb, b)):
        P.check(load(t.data_ptr(), k, x.data_ptr(), x.numel(), None))
        P.check(forward(t.data_ptr(), k, None))
    P.check(pointwise(ta.data_ptr(), tb.data_ptr(), k, None))
    P.check(inverse(ta.data_ptr(), k, None))
    P.check(store(ta.data_ptr(), k, z.data_ptr(), z.numel(), None))
    return {"product": z, "transform_b": tb}


# ---- what a pass cannot do without -------------------------------------------
def _product_flops(na, nb):
    """Three real FFTs of the product's 16-bit points (2.5 N log2 N each) and the pointwise product."""
    n = 2.0 * (na + nb)
    return 7.5 * n * math.log2(n) + 3 * n


def work(case):
    """Bytes: inputs read and outputs written once.  Flops: the products' FFTs
    at 16 bits a point.  Pi(): each level of the splitting tree forms four
    products over half of p words each; Newton: about five products of
    p words each for division, four for the inverse square root."""
    op = case["op"]
    if op in ("pi", "pi_text"):
        p, text = case["digits"] / 9.633, case["digits"] / 1.2041
        levels = max(1.0, math.log2(case["digits"] / 14.18))
        return {"bytes": text if op == "pi_text" else 4 * p,
                "flops": 2 * levels * _product_flops(p / 2, p / 2) + 10 * _product_flops(p, p)}
    if op == "mul":
        return {"bytes": 8.0 * (case["na"] + case["nb"]), "flops": _product_flops(case["na"], case["nb"])}
    if op == "batch":
        s = _batch_sizes(case)
        return {"bytes": sum(8.0 * (a + b) for a, b in s), "flops": sum(_product_flops(a, b) for a, b in s)}
    if op == "newton":
        return {"bytes": 16.0 * case["p"], "flops": 9 * _product_flops(case["p"], case["p"])}
    if op == "dec":
        w = _dec_words(case["digits"])
        return {"bytes": 4.0 * w + case["digits"],
                "flops": 2 * max(1.0, math.log2(w / 64)) * _product_flops(w / 2, w / 2)}
    n = float(1 << case["k"])
    point = 8 if op == "ntt" else 16
    return {"bytes": 8.0 * (case["na"] + case["nb"]) + point * n, "flops": 3 * 5 * n * case["k"] + 6 * n}


# ---- results from plain Python and torch -------------------------------------
def _as_int(words):
    return int.from_bytes(words.cpu().numpy().astype("<u4").tobytes(), "little")


def _as_words(x, n):
    return torch.from_numpy(np.frombuffer(x.to_bytes(4 * n, "little"), dtype="<i4").copy())


def _product(a, b):
    """a * b from a float64 FFT convolution of bytes (coefficients below 2^43: rounding is exact)."""
    if a.numel() + b.numel() < 20_000:
        return _as_words(_as_int(a) * _as_int(b), a.numel() + b.numel())
    n = 4 * (a.numel() + b.numel())
    size = 1 << (n - 1).bit_length()
    f, g = (torch.fft.rfft(x.view(torch.uint8).double(), n=size) for x in (a, b))
    v = torch.fft.irfft(f * g, n=size)[:n].round().to(torch.int64)
    del f, g
    while True:
        up = v >> 8
        if not bool(up.any()):
            break
        v &= 255
        v[1:] += up[:-1]
    return v.to(torch.uint8).view(torch.int32).cpu()


def _bit_reversed(x):
    n = x.numel()
    k, i, j = n.bit_length() - 1, torch.arange(n, device=x.device), torch.zeros(n, dtype=torch.int64, device=x.device)
    for b in range(k):
        j |= ((i >> b) & 1) << (k - 1 - b)
    return x[j]


def exact(case, seed):
    op = case["op"]
    if op == "mul":
        return _product(_words(case["na"], 2 * seed), _words(case["nb"], 2 * seed + 1))
    if op == "batch":
        sizes = _batch_sizes(case)
        x = _words(sum(na + nb for na, nb in sizes), seed).cpu()
        out, at = [], 0
        for na, nb in sizes:
            out.append(_as_words(_as_int(x[at:at + na]) * _as_int(x[at + na:at + na + nb]), na + nb))
            at += na + nb
        return torch.cat(out)
    if op == "dec":
        if case["digits"] > 1_500_000:
            return None
        sys.set_int_max_str_digits(0)
        w = _words(_dec_words(case["digits"]), seed)
        bits, d = 32 * (w.numel() - 1), 9 * -(-case["digits"] // 9)
        v = _as_int(w)
        whole, part = v >> bits, v & ((1 << bits) - 1)
        text = "%d.%s" % (whole, str(part * 10 ** d >> bits).zfill(d))
        return np.frombuffer(text[:2 + case["digits"]].encode(), dtype=np.uint8)
    if op in ("ntt", "fft"):
        a, b = _words(case["na"], 2 * seed), _words(case["nb"], 2 * seed + 1)
        spectrum = None
        if op == "fft":  # exp(+i theta), bit-reversed order, one byte a point
            x = torch.zeros(1 << case["k"], dtype=torch.complex128, device="cuda")
            x[:4 * b.numel()] = b.view(torch.uint8).to(torch.complex128)
            spectrum = _bit_reversed(torch.fft.ifft(x, norm="forward")).cpu()
        return {"product": _product(a, b), "transform_b": spectrum}
    return None  # Pi() and the Newton steps: their last words follow the reference's truncations
