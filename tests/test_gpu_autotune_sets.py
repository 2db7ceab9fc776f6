"""The autotuner installs a plan only for the primes whose passes it timed:
lengths whose product runs none of 2^L points on the 31-bit primes (whole in
one CTA, or through the outer stage) keep the plan that was set, and tuning
the 31-bit primes leaves the 64-bit ones their plans."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def big(engine):
    engine.teardown()
    engine.init(26)
    yield engine
    engine.teardown()
    engine.init(24)


@pytest.mark.parametrize("L,plan", [(5, [5]), (11, [6, 5]), (12, [7, 5]), (26, [5, 5, 6, 10])])
def test_lengths_without_passes_keep_their_plan(big, L, plan):
    try:
        big.set_plan(L, plan)
        got, ms = big.autotune(L, L, reps=1)[L]
        assert got == plan and ms > 0
        for primes in (2, 3):
            big.set_prime_set(primes)
            assert big.plan(L) == plan, primes
    finally:
        big.set_prime_set(2)
        big.set_plan(L, [])


def test_each_set_keeps_its_own_plan(big):
    lo, hi = 13, 16
    hand = {13: [8, 5], 14: [9, 5], 15: [10, 5], 16: [5, 5, 6]}
    rng = np.random.default_rng(26)
    try:
        for L, p in hand.items():
            big.set_plan(L, p)
        tuned = {L: p for L, (p, _) in big.autotune(lo, hi, reps=2).items()}
        assert all(big.plan(L) == tuned[L] for L in hand)
        big.set_prime_set(3)
        assert all(big.plan(L) == hand[L] for L in hand)     # the 64-bit primes: as set by hand
        tuned64 = {L: p for L, (p, _) in big.autotune(lo, hi, reps=2).items()}
        for primes, plans in ((3, tuned64), (2, tuned)):
            big.set_prime_set(primes)
            for L in hand:
                assert big.plan(L) == plans[L], (primes, L)
                a = rng.integers(0, 1 << 32, (1 << (L - 1)) - 3, dtype=np.uint64).astype(np.uint32)
                b = rng.integers(0, 1 << 32, (1 << (L - 1)) + 2, dtype=np.uint64).astype(np.uint32)
                want = np.zeros(len(a) + len(b), dtype=np.uint32)
                r = oracle.gmp_mul(a, b)
                want[:len(r)] = r
                assert np.array_equal(big.mul(a, b), want), (primes, L)
    finally:
        big.set_prime_set(2)
        for L in hand:
            big.set_plan(L, [])
        assert all(big.plan(L) != hand[L] for L in hand)
    assert big.device_errors() == 0
