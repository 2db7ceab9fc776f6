"""The integer arrays of a batch call: every iterable gives what the ctypes
constructor gives for it, whichever way it is converted."""
import ctypes

import numpy as np
import pytest

from cryptography_gb300 import engine

CASES = [
    [3, 1, 4], (3, 1, 4), [], np.array([3, 1, 4], dtype=np.uint64), range(3), bytes([3, 1, 4]), bytearray(range(8)),
    bytes(range(16)), [-1, 5], [1 << 64, 2], [np.int64(7), True],
]


@pytest.mark.parametrize("make", [lambda v: v, lambda v: iter(v)], ids=["itself", "iterator"])
@pytest.mark.parametrize("values", CASES, ids=repr)
@pytest.mark.parametrize("more", [0, 2])
def test_same_as_ctypes(values, make, more):
    n = len(values) + more   # (a short iterable leaves zeros)
    want = list((ctypes.c_uint64 * n)(*values))
    assert list(engine._c_array(ctypes.c_uint64, "Q", n, make(values))) == want


@pytest.mark.parametrize("values,error", [([1.0], TypeError), (["1"], TypeError), ("1", TypeError), ([1, 2], IndexError),
                                          (iter([1, 2]), IndexError), ([None], TypeError)])
def test_refused(values, error):
    with pytest.raises(error):
        engine._c_array(ctypes.c_uint64, "Q", 1, values)
