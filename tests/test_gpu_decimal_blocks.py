"""Decimal conversions on both sides of the lines between one in-memory piece
per multiprocessor and more, and between pieces split by launches of their own
and in one, digit for digit: D random digits, D a multiple of
a block's digits and one off, and all nines."""
import random
import sys

import pytest

from cryptography_gb300 import arith

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("top,pieces", [(0, 1), (0, 152), (0, 153), (3, 151), (3, 152), (3, 153), (3, 400), (7, 40),
                                        (7, 170), (11, 1), (11, 2), (8, 20), (8, 75), (8, 76), (8, 77), (9, 37), (9, 39), (10, 5), (11, 5), (12, 1)])
def test_pieces_per_multiprocessor(engine, top, pieces, monkeypatch):
    monkeypatch.setenv("GBNTT_DEC_TOP", str(top))
    if hasattr(sys, "set_int_max_str_digits"):
        sys.set_int_max_str_digits(0)
    rng = random.Random(1000 * top + pieces)
    full = pieces * (9 << (top + 1))
    for digits in (full - 1, full, full + 1):
        s = str(rng.randrange(1, 10)) + "".join(rng.choice("0123456789") for _ in range(digits - 1))
        assert arith.to_decimal(int(s)) == s
    assert arith.to_decimal(10 ** full - 1) == "9" * full
