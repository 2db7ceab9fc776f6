"""The 31-bit prime set's constants (gbntt_p31.cuh), checked on the host: the
primes, their 2- and 3-adicity, generators and inverses, and that their
product exceeds every coefficient of a product whose transform they take."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cryptography_gb300", "csrc")


def _array(name):
    src = open(os.path.join(CSRC, "gbntt_p31.cuh")).read()
    body = re.search(r"%s\[3\] = \{([^}]*)\}" % name, src).group(1)
    return [int(x.strip().rstrip("u")) for x in body.split(",")]


def _prime(n):
    return n > 1 and all(n % d for d in range(2, int(n ** 0.5) + 1))


def test_primes_and_roots():
    P, inv, gen = _array("kP31"), _array("kP31Inv"), _array("kP31Gen")
    assert len(set(P)) == 3
    for p, i, g in zip(P, inv, gen):
        assert _prime(p) and 1 << 30 < p < 1 << 31
        assert (p - 1) % (3 << 25) == 0                    # transforms of 2^25 and 3 2^25 points
        assert p * i % (1 << 32) == 1
        assert 3 * p > 1 << 32                             # a limb is reduced by 2 p and p
        odd = [q for q in (2, 3, 5, 7) if (p - 1) % q == 0]
        assert all(pow(g, (p - 1) // q, p) != 1 for q in odd)
        m = p - 1
        for q in odd:
            while m % q == 0:
                m //= q
        assert m == 1


@pytest.mark.parametrize("points", [1 << 25, 3 << 25])
def test_modulus_exceeds_every_coefficient(points):
    P = _array("kP31")
    shorter = (points + 1) // 2                            # n_a + n_b - 1 <= points
    assert P[0] * P[1] * P[2] > shorter * ((1 << 32) - 1) ** 2
    # Garner's partial sum p0 a1 + a0 + lo(p0 p1) a2 stays below 2^64
    assert P[0] * (P[1] - 1) + P[0] - 1 + ((1 << 32) - 1) * (P[2] - 1) < 1 << 64
