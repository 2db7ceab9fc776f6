"""Packed products with one 64-bit limb per coefficient over the three 64-bit
primes. The default set runs them as 32-bit limbs wherever the engine is long
enough, so the packed tests run once more with prime set 3, which keeps the
64-bit decomposition and its carries."""
import numpy as np
import pytest

import oracle
import test_gpu_packed
from cryptography_gb300 import cudart
from test_gpu_packed import (test_packed_2pow22, test_packed_length_boundaries, test_packed_limbs_above_primes,  # noqa: F401
                             test_packed_small_and_sweep, test_packed_square_and_equivalence)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def engine(engine):
    engine.set_prime_set(3)
    yield engine
    engine.set_prime_set(2)


def test_bigint_api_packed_mode(monkeypatch):
    monkeypatch.setenv("GBNTT_PRIMES", "3")
    test_gpu_packed.test_bigint_api_packed_mode()


@pytest.mark.parametrize("n", [1, 16, 17, 2048, 2049, (1 << 20) + 1])
def test_packed_all_ones(engine, n):
    # the largest coefficients, a square and two operands: (beta^n - 1)^2
    full = np.full(n, (1 << 64) - 1, dtype=np.uint64)
    for b in (full, full.copy()):
        c = engine.mul64(full, b)
        want = np.full(2 * n, (1 << 64) - 1, dtype=np.uint64)
        want[:n] = 0
        want[0] += 1
        want[n] -= 1
        assert np.array_equal(c, want), n
    assert engine.device_errors() == 0


def test_one_coefficient_per_limb_runs(engine):
    # 2^17 64-bit limbs are 2^17 points here (each prime with launches of its
    # own), and 2^18 points of 32-bit limbs on the default set
    n = 1 << 16
    a, c = cudart.DeviceBuffer(8 * n), cudart.DeviceBuffer(16 * n)
    x = np.random.default_rng(3).integers(0, 1 << 64, n, dtype=np.uint64)
    a.upload(x)
    firsts = []
    for primes in (3, 2):
        engine.set_prime_set(primes)
        try:
            engine.launch_log(True)
            assert engine.lib().gbntt_mul_u64(c.ptr, a.ptr, n, a.ptr, n, None) == 0
            cudart.synchronize()
            firsts.append([r[0] for r in engine.launch_records()].count("fwd_pass_first"))
        finally:
            engine.launch_log(False)
            engine.set_prime_set(3)
        want = oracle.gmp_mul(x.view(np.uint32), x.view(np.uint32))
        got = c.download(np.uint32, 4 * n)
        assert np.array_equal(got[:len(want)], want) and not got[len(want):].any(), primes
    assert firsts == [3, 1], firsts
    for b in (a, c):
        b.free()
    assert engine.device_errors() == 0
