"""Host products whose operands are read in place or copied beside the first
operand's transform, against the same product of device operands: pinned and
pageable operands, squares, pointers off 16 bytes, on both sides of the lines
between one transform, the radix-3 stage and the outer stage."""
import ctypes

import numpy as np
import pytest

from cryptography_gb300 import cudart, synth

pytestmark = pytest.mark.gpu

M = 1 << 25
u32p = ctypes.POINTER(ctypes.c_uint32)


@pytest.fixture(scope="module")
def big(engine):
    engine.teardown()
    engine.init(28)
    yield engine
    engine.teardown()
    engine.init(24)


@pytest.mark.parametrize("na,nb", [(1 << 16, 60001), (1 << 21, 1 << 21), (M // 2, M // 2), (M + 5, M), (3 * M, 70001),
                                   (2 * M + 3, M + 1), (3 * M + 1, 0)])
@pytest.mark.parametrize("pinned", ["ab", "a", "b", ""])
def test_host_operands(big, na, nb, pinned):
    # nb = 0: the square
    square = nb == 0
    nb = nb or na
    xa = synth.operand(na, 51)
    xb = xa if square else synth.operand(nb, 52)
    da, dc = cudart.DeviceBuffer(4 * na), cudart.DeviceBuffer(4 * (na + nb))
    da.upload(xa)
    db = da
    if not square:
        db = cudart.DeviceBuffer(4 * nb)
        db.upload(xb)
    big.mul_device(dc.ptr, da.ptr, na, db.ptr, nb)
    cudart.synchronize()
    want = dc.download(np.uint32, na + nb)
    for b in (da, dc) if square else (da, db, dc):
        b.free()
    held = []

    def place(x, pin):
        if not pin:
            return np.ascontiguousarray(x)
        p = cudart.PinnedBuffer(len(x) + 1, np.uint32)
        held.append(p)
        p.array[1:] = x
        return p.array[1:]

    a = place(xa, "a" in pinned)
    b = a if square else place(xb, "b" in pinned)
    c = place(np.zeros(na + nb, dtype=np.uint32), "a" in pinned)
    rc = big.lib().gbntt_mul_u32_host(*(z for x in ((c,), (a, na), (b, nb))
                                        for z in (x[0].ctypes.data_as(u32p),) + x[1:]))
    assert rc == 0
    assert np.array_equal(c, want)
    for p in held:
        p.free()
