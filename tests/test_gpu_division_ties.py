"""Divisions whose remainders sit next to multiples of the divisor, where the
multiple taken from the top limbs may fall one short, against Python
integers: exact multiples, one below and one above, divisors of one to many
limbs, with top limbs of one bit and of all ones."""
import random

import pytest

from cryptography_gb300 import arith

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 31, 32, 33, 64, 96, 97, 129, 2048, 2049, 40000, 300001])
def test_remainders_next_to_multiples(engine, bits):
    rng = random.Random(bits)
    for d in (1 << (bits - 1), (1 << bits) - 1, rng.getrandbits(bits) | 1 << (bits - 1)):
        for qbits in (1, 40, bits, 2 * bits + 5):
            q = rng.getrandbits(qbits) | 1 << (qbits - 1)
            for r in (0, d - 1, min(1, d - 1), rng.randrange(d)):
                assert arith.div_newton(q * d + r, d) == (q, r), (bits, qbits, r)
        x = arith.newton_reciprocal(d)
        assert x == (1 << (2 * d.bit_length())) // d


@pytest.mark.parametrize("k", [1, 9, 18, 4608, 36864, 73728, 200000])
def test_powers_of_ten(engine, k):
    assert arith.to_decimal(10 ** k) == "1" + "0" * k
    assert arith.to_decimal(10 ** k - 1) == "9" * k
    assert arith.to_decimal(10 ** k + 1) == "1" + "0" * (k - 1) + "1"
