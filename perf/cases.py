"""Timed workloads of the multiply engine, through its public entry points.

Each case is a dict of plain values; ``prepare`` makes its inputs from a seed,
``run`` is one pass as a user's program calls it, ``exact`` is the same result
from Python integers where that is quick. Limb vectors are uniform random (the
operands of every benchmark of this repository are), device vectors are torch
int32 / int64 tensors holding the limbs' bits.
"""
import math
import sys

import numpy as np
import torch

import cryptography_gb300 as g
from cryptography_gb300 import arith, engine

_MAX_LOG = 29      # transforms of up to 2^29 coefficients: the 2^28 x 2^28-limb product
_SERVER_LOG = 22   # coefficients of a serving slot (log2)
_server = None


def listed():
    return [
        # one short product of host integers (a few thousand bits): the latency of a single call
        {"name": "host_mul_96x64", "kind": "host", "na": 96, "nb": 64},
        # a short product of device operands: launches and their gaps
        {"name": "mul_1024x1000", "kind": "mul", "na": 1024, "nb": 1000, "bits": 32, "square": False},
        # a middle-sized product of odd lengths, too small to fill the GPU for long
        {"name": "mul_50021x43987", "kind": "mul", "na": 50021, "nb": 43987, "bits": 32, "square": False},
        # the 2^20 x 2^20-limb product, checked against GMP everywhere in the tests
        {"name": "mul_2pow20", "kind": "mul", "na": 1 << 20, "nb": 1 << 20, "bits": 32, "square": False},
        # a square (one forward transform), as powers are computed; an odd length
        {"name": "sqr_5000011", "kind": "mul", "na": 5000011, "nb": 5000011, "bits": 32, "square": True},
        # the largest benchmark product: 1 GiB operands
        {"name": "mul_2pow28", "kind": "mul", "na": 1 << 28, "nb": 1 << 28, "bits": 32, "square": False},
        # packed form: one 64-bit limb per coefficient, three 64-bit primes
        {"name": "packed_700001x600011", "kind": "mul", "na": 700001, "nb": 600011, "bits": 64, "square": False},
        # many short products in one call (the low levels of a product tree)
        {"name": "batch_2048_small", "kind": "batch", "count": 2048, "lo": 5.0, "hi": 10.0},
        # uneven products of very different sizes in one call
        {"name": "batch_256_uneven", "kind": "batch", "count": 256, "lo": 10.0, "hi": 20.0},
        # a burst of requests of mixed sizes to the serving loop, all waited for
        {"name": "serve_192", "kind": "serve", "count": 192, "lo": 8.0, "hi": 20.0},
        # decimal digits of a large integer: reciprocals, divisions by one divisor, cyclic products
        {"name": "decimal_250007", "kind": "decimal", "n": 250007},
        # negacyclic polynomial product with 64-bit coefficients
        {"name": "negacyclic_2pow18", "kind": "negacyclic", "log_n": 18},
    ]


def _log_size(rng, lo, hi):
    return int(2.0 ** rng.uniform(lo, hi))


def draw(rng):
    kind = rng.choice(["host", "mul", "mul", "mul", "packed", "batch", "batch", "serve", "decimal", "negacyclic"])
    if kind == "host":
        return {"kind": "host", "na": _log_size(rng, 3, 20), "nb": _log_size(rng, 3, 20)}
    if kind == "mul":
        if rng.random() < 0.25:
            n = _log_size(rng, 6, 27)
            return {"kind": "mul", "na": n, "nb": n, "bits": 32, "square": True}
        na = _log_size(rng, 6, 27)
        return {"kind": "mul", "na": na, "nb": max(1, int(na * 2.0 ** -rng.uniform(0, 3))), "bits": 32, "square": False}
    if kind == "packed":
        na = _log_size(rng, 6, 24)
        return {"kind": "mul", "na": na, "nb": max(1, int(na * 2.0 ** -rng.uniform(0, 3))), "bits": 64, "square": False}
    if kind == "batch":
        lo = rng.uniform(4, 12)
        hi = lo + rng.uniform(1, 8)
        return {"kind": "batch", "count": max(2, min(4096, _log_size(rng, 26, 28) >> int(hi + 1))), "lo": lo, "hi": hi}
    if kind == "serve":
        lo = rng.uniform(6, 12)
        hi = lo + rng.uniform(2, 8)
        return {"kind": "serve", "count": rng.randint(16, 256), "lo": lo, "hi": hi}
    if kind == "decimal":
        return {"kind": "decimal", "n": _log_size(rng, 8, 21)}
    return {"kind": "negacyclic", "log_n": rng.randint(6, 22)}


def _sizes(case):
    # the operand lengths belong to the case, the limbs to the seed
    r = np.random.default_rng(4242)
    na = np.floor(2.0 ** r.uniform(case["lo"], case["hi"], case["count"])).astype(np.int64)
    nb = np.floor(2.0 ** r.uniform(case["lo"], case["hi"], case["count"])).astype(np.int64)
    return na, nb


def _limbs(n, seed, bits):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if bits == 32:
        return torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=gen)
    x = torch.randint(-(1 << 31), 1 << 31, (2 * n,), dtype=torch.int32, device="cuda", generator=gen)
    return x.view(torch.int64)


def prepare(case, seed):
    global _server
    if not g.is_ready():
        g.init(_MAX_LOG)
    kind = case["kind"]
    if kind == "host":
        r = np.random.default_rng(seed)
        st = {"kind": kind, "a": r.integers(0, 1 << 32, case["na"], dtype=np.uint32),
              "b": r.integers(0, 1 << 32, case["nb"], dtype=np.uint32)}
    elif kind == "mul":
        a = _limbs(case["na"], 2 * seed, case["bits"])
        b = a if case["square"] else _limbs(case["nb"], 2 * seed + 1, case["bits"])
        st = {"kind": kind, "a": a, "b": b, "bits": case["bits"],
              "c": torch.empty(case["na"] + case["nb"], dtype=a.dtype, device="cuda")}
    elif kind in ("batch", "serve"):
        if kind == "serve" and _server is None:
            _server = g.Server(slots=4, slot_log=_SERVER_LOG)
        na, nb = _sizes(case)
        a = _limbs(int(na.sum()), 2 * seed, 32)
        b = _limbs(int(nb.sum()), 2 * seed + 1, 32)
        c = torch.empty(len(a) + len(b), dtype=torch.int32, device="cuda")
        at = lambda t, n: [t.data_ptr() + 4 * int(o) for o in np.concatenate([[0], np.cumsum(n)[:-1]])]  # noqa: E731
        st = {"kind": kind, "a": a, "b": b, "c": c, "pa": at(a, na), "pb": at(b, nb), "pc": at(c, na + nb),
              "na": [int(x) for x in na], "nb": [int(x) for x in nb]}
    elif kind == "decimal":
        r = np.random.default_rng(seed)
        x = r.integers(0, 1 << 32, case["n"], dtype=np.uint32)
        x[-1] = (1 << 31) + (int(x[-1]) >> 24)   # the number of decimal digits then depends on the case alone
        st = {"kind": kind, "x": int.from_bytes(x.tobytes(), "little")}
    else:
        n = 1 << case["log_n"]
        st = {"kind": kind, "f": _limbs(n, 2 * seed, 64), "g": _limbs(n, 2 * seed + 1, 64), "log_n": case["log_n"],
              "out": torch.empty(4 * n, dtype=torch.int64, device="cuda")}
    torch.cuda.synchronize()   # the engine works on its own stream
    return st


def run(st):
    kind = st["kind"]
    if kind == "host":
        return g.mul(st["a"], st["b"]).view(np.int32)
    if kind == "mul":
        a, b, c = st["a"], st["b"], st["c"]
        if st["bits"] == 32:
            g.mul_device(c.data_ptr(), a.data_ptr(), len(a), b.data_ptr(), len(b))
        else:
            engine._check(engine.lib().gbntt_mul_u64(c.data_ptr(), a.data_ptr(), len(a), b.data_ptr(), len(b), None))
        return c
    if kind == "batch":
        g.batch_mul_device(st["pc"], st["pa"], st["na"], st["pb"], st["nb"])
        return st["c"]
    if kind == "serve":
        t = [_server.submit(c, a, na, b, nb)
             for c, a, na, b, nb in zip(st["pc"], st["pa"], st["na"], st["pb"], st["nb"])]
        for ticket in t:
            _server.wait(ticket)
        return st["c"]
    if kind == "decimal":
        return np.frombuffer(arith.to_decimal(st["x"]).encode(), dtype=np.uint8)
    g.negacyclic_mul_device(st["out"].data_ptr(), st["f"].data_ptr(), st["g"].data_ptr(), st["log_n"])
    return st["out"]


def work(case):
    kind = case["kind"]
    if kind in ("host", "mul"):
        n = case["na"] + (0 if case.get("square") else case["nb"]) + case["na"] + case["nb"]
        return {"bytes": n * case.get("bits", 32) // 8, "flops": 0}
    if kind in ("batch", "serve"):
        na, nb = _sizes(case)
        return {"bytes": 8 * int(na.sum() + nb.sum()), "flops": 0}
    if kind == "decimal":
        return {"bytes": 4 * case["n"] + int(32 * case["n"] * math.log10(2)), "flops": 0}
    return {"bytes": (8 + 8 + 32) << case["log_n"], "flops": 0}


def _int(t):
    return int.from_bytes(np.ascontiguousarray(t.cpu().numpy() if isinstance(t, torch.Tensor) else t).tobytes(), "little")


def _words(v, n, dtype):
    return np.frombuffer(v.to_bytes(n * np.dtype(dtype).itemsize, "little"), dtype=dtype)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("host", "mul"):
        if (case["na"] + case["nb"]) * case.get("bits", 32) > 1 << 22:
            return None
        st = prepare(case, seed)
        dtype = np.int64 if case.get("bits") == 64 else np.int32
        return _words(_int(st["a"]) * _int(st["b"]), case["na"] + case["nb"], dtype)
    if kind in ("batch", "serve"):
        na, nb = _sizes(case)
        if float(((na + nb) ** 1.6).sum()) > 2e9:
            return None
        st = prepare(case, seed)
        a, b = st["a"].cpu().numpy(), st["b"].cpu().numpy()
        out, pa, pb = [], 0, 0
        for x, y in zip(st["na"], st["nb"]):
            out.append(_words(_int(a[pa:pa + x]) * _int(b[pb:pb + y]), x + y, np.int32))
            pa, pb = pa + x, pb + y
        return np.concatenate(out)
    if kind == "decimal":
        if case["n"] > 5000:
            return None
        sys.set_int_max_str_digits(0)
        return np.frombuffer(str(prepare(case, seed)["x"]).encode(), dtype=np.uint8)
    if case["log_n"] > 13:
        return None
    # both polynomials in slots of 24 bytes; the product's upper half comes back with the opposite sign
    n = 1 << case["log_n"]
    st = prepare(case, seed)
    slots = [np.zeros((n, 3), dtype=np.int64) for _ in range(2)]
    slots[0][:, 0], slots[1][:, 0] = st["f"].cpu().numpy(), st["g"].cpu().numpy()
    p = (_int(slots[0]) * _int(slots[1])).to_bytes(48 * n, "little")
    c = [int.from_bytes(p[24 * i:24 * i + 24], "little") for i in range(2 * n)]
    return np.concatenate([_words((c[i] - c[i + n]) % (1 << 256), 4, np.int64) for i in range(n)])
