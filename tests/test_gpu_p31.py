"""Products on the 31-bit prime set (gbntt_p31*.cu) against GMP and against
the 64-bit prime sets: both ends of every transform length, every pass size,
operands whose coefficients are largest, waves that share right operands, and
the path without pass twiddle tables."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

import oracle
from cryptography_gb300 import cudart

pytestmark = pytest.mark.gpu


def _rand(rng, n):
    return rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)


def _want(a, b):
    r = oracle.gmp_mul(a, b)
    out = np.zeros(len(a) + len(b), dtype=np.uint32)
    out[:len(r)] = r
    return out


def _waves(engine, A, B):
    # a batch whose equal right operands share one device buffer
    up = {}
    for x in A + B:
        if id(x) not in up:
            up[id(x)] = cudart.DeviceBuffer(4 * len(x))
            up[id(x)].upload(x)
    dc = [cudart.DeviceBuffer(4 * (len(a) + len(b))) for a, b in zip(A, B)]
    engine.batch_mul_device([c.ptr for c in dc], [up[id(x)].ptr for x in A], [len(x) for x in A],
                            [up[id(x)].ptr for x in B], [len(x) for x in B])
    cudart.synchronize()
    for a, b, c in zip(A, B, dc):
        assert np.array_equal(c.download(np.uint32, len(a) + len(b)), _want(a, b)), (len(a), len(b))
    for buf in list(up.values()) + dc:
        buf.free()


@pytest.mark.parametrize("L", range(5, 25))
def test_lengths(engine, L):
    # the longest and the shortest product of a 2^L-point transform, even and
    # uneven operands, a square
    rng = np.random.default_rng(3100 + L)
    top = 1 << L
    for need in (top, top // 2 + 1):
        for na in {(need + 1) // 2, max(1, need // 9)}:
            a, b = _rand(rng, na), _rand(rng, need + 1 - na)
            assert np.array_equal(engine.mul(a, b), _want(a, b)), (L, na)
    a = _rand(rng, top // 2)
    assert np.array_equal(engine.sqr(a), _want(a, a))
    full = np.full(top // 2, 0xFFFFFFFF, dtype=np.uint32)
    n = len(full)
    for c in (engine.mul(full, full), engine.mul(full, full.copy())):
        assert c[0] == 1 and not c[1:n].any() and c[n] == 0xFFFFFFFE and (c[n + 1:] == 0xFFFFFFFF).all()
    assert engine.device_errors() == 0


@pytest.mark.parametrize("plan", [[10, 10], [5, 10], [10, 5], [9, 7], [7, 9], [6, 8], [5, 5, 5], [6, 10, 6], [9, 9],
                                  [5, 6, 7, 5], [8, 5, 9]])
def test_pass_sizes(engine, plan):
    L = sum(plan)
    rng = np.random.default_rng(L)
    a, b = _rand(rng, (1 << (L - 1)) - 3), _rand(rng, (1 << (L - 1)) + 2)
    try:
        engine.set_plan(L, plan)
        assert np.array_equal(engine.mul(a, b), _want(a, b))
        assert np.array_equal(engine.sqr(a), _want(a, a))
        # waves: own, paired and shared right operands
        c, d = b[1:], b[:77]
        for B in ([b, d, c], [b, b, c, c], [b] * 3):
            _waves(engine, [a[i:] for i in range(len(B))], B)
    finally:
        engine.set_plan(L, [])
    assert engine.device_errors() == 0


@pytest.mark.parametrize("L", range(5, 13))
def test_one_cta_waves(engine, L):
    # waves of products that run in one CTA each: own, paired and shared
    # right operands, a square, one-limb operands
    rng = np.random.default_rng(41 + L)
    top = 1 << L
    a, b, c = _rand(rng, top // 2), _rand(rng, top // 2 + 1), _rand(rng, 1)
    d = _rand(rng, top - top // 3)
    _waves(engine, [a, c, d, a], [b, d, c, a])
    A = [a, a[1:], d[:top // 2], d[1:top // 2]]
    _waves(engine, A, [b, b, a, a])
    _waves(engine, A[1:], [b] * 3)
    # more products than take a cluster of CTAs each: the longest and the
    # shortest of the length, so that every carry tile boundary is met
    sizes = [(top // 2, top // 2 + 1 - i % 3) for i in range(57)] + [(top // 2 + 1, 1)] * 3
    _waves(engine, [_rand(rng, n) for n, _ in sizes], [_rand(rng, n) for _, n in sizes])
    full = np.full(top // 2, 0xFFFFFFFF, dtype=np.uint32)
    _waves(engine, [full, full], [full, full.copy()])
    assert engine.device_errors() == 0


def test_same_products_as_the_64bit_primes(engine):
    rng = np.random.default_rng(5)
    for na, nb in ((1, 1), (40, 3), (1500, 900), (70001, 333), (1 << 20, (1 << 20) + 1), (3 << 19, 3 << 19)):
        a, b = _rand(rng, na), _rand(rng, nb)
        got = engine.mul(a, b)
        engine.set_prime_set(3)
        try:
            assert np.array_equal(engine.mul(a, b), got), (na, nb)
        finally:
            engine.set_prime_set(2)


@pytest.mark.parametrize("knobs", [{"GBNTT_PASS_TABLES": "0"}, {"GBNTT_P31": "0"},
                                   {"GBNTT_PASS_TABLES": "0", "GBNTT_RADIX3_MIN_LOG": "10"}])
def test_knobs(knobs):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    body = textwrap.dedent("""
        import sys
        sys.path.insert(0, %r)
        import numpy as np
        import cryptography_gb300 as g
        import oracle
        g.init(22)
        rng = np.random.default_rng(71)
        for na, nb in [(33, 17), (2000, 100), (4096, 4095), (6000, 6000), (70000, 12345), (1 << 20, 3)]:
            a = rng.integers(0, 1 << 32, na, dtype=np.uint64).astype(np.uint32)
            b = rng.integers(0, 1 << 32, nb, dtype=np.uint64).astype(np.uint32)
            want = np.zeros(na + nb, dtype=np.uint32)
            r = oracle.gmp_mul(a, b)
            want[:len(r)] = r
            assert np.array_equal(g.mul(a, b), want), (na, nb)
        assert g.device_errors() == 0
        print("fine")
    """ % root)
    r = subprocess.run([sys.executable, "-c", body], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, **knobs))
    assert r.returncode == 0 and "fine" in r.stdout, r.stderr[-2000:]


@pytest.mark.parametrize("log_n", [5, 6, 8, 10, 11, 13, 17, 19, 22, 23])
def test_negacyclic(engine, log_n):
    # three products of 32-bit halves (gbntt_p31_nega.cu) against the three
    # 64-bit primes: random and largest coefficients, squares
    n = 1 << log_n
    rng = np.random.default_rng(log_n)
    f = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    g = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    full = np.full(n, 0xFFFFFFFFFFFFFFFF, dtype=np.uint64)
    f[::7] = 0xFFFFFFFF00000000
    bufs = []
    for x in (f, g, full):
        bufs.append(cudart.DeviceBuffer(8 * n))
        bufs[-1].upload(x)
    out = cudart.DeviceBuffer(32 * n)
    for x, y in ((0, 1), (0, 0), (2, 2), (2, 1), (1, 2)):
        got = []
        for primes in (2, 3):
            engine.set_prime_set(primes)
            try:
                engine.negacyclic_mul_device(out.ptr, bufs[x].ptr, bufs[y].ptr, log_n)
                cudart.synchronize()
                got.append(out.download(np.uint64, 4 * n))
            finally:
                engine.set_prime_set(2)
        assert np.array_equal(*got), (x, y)
    for b in bufs + [out]:
        b.free()
    assert engine.device_errors() == 0
