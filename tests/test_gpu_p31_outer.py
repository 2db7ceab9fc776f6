"""Products of more than 2^25 coefficients on the 31-bit primes (the outer
stage over several 2^25-point transforms, gbntt_p31_outer.cu) against the
three 64-bit primes, whose products test_gpu_fullsize.py and
test_gpu_maxsize.py compare with GMP: both ends of a block count, operands of
one block, squares, and all-ones operands (the largest coefficients)."""
import numpy as np
import pytest

from cryptography_gb300 import cudart, synth

pytestmark = pytest.mark.gpu

M = 1 << 25


@pytest.fixture(scope="module")
def big(engine):
    engine.teardown()
    engine.init(29)
    yield engine
    engine.teardown()
    engine.init(24)


def _device(x):
    b = cudart.DeviceBuffer(4 * len(x))
    b.upload(x)
    return b


def _kinds(engine, call):
    engine.launch_log(True)
    try:
        call()
        return {r[0] for r in engine.launch_records()}
    finally:
        engine.launch_log(False)


@pytest.mark.parametrize("na,nb", [(M, M // 2 + M // 4), (M + 1, M), (3 * M, 9), (2 * M, 2 * M), (3 * M + 7, M + 2),
                                   (5 * M - 9, M // 3), (4 * M + 1, 2 * M + 1), (8 * M, 8 * M - 3)])
def test_outer_stage(big, na, nb):
    a, b = synth.operand(na, na), synth.operand(nb, nb + 1)
    da, db, dc = _device(a), _device(b), cudart.DeviceBuffer(4 * (na + nb))
    got = []
    for primes in (2, 3):
        big.set_prime_set(primes)
        try:
            kinds = _kinds(big, lambda: (big.mul_device(dc.ptr, da.ptr, na, db.ptr, nb), cudart.synchronize()))
            assert ("outer_fwd" in kinds) == (primes == 2), kinds
            got.append(dc.download(np.uint32, na + nb))
        finally:
            big.set_prime_set(2)
    assert np.array_equal(*got)
    for x in (da, db, dc):
        x.free()
    assert big.device_errors() == 0


@pytest.mark.parametrize("n", [M, 2 * M, 3 * M + M // 2, 8 * M])
def test_outer_stage_largest_coefficients(big, n):
    full = np.full(n, 0xFFFFFFFF, dtype=np.uint32)
    da, dc = _device(full), cudart.DeviceBuffer(8 * n)
    db = _device(full)
    for right in (da, db):   # a square, and two operands
        big.mul_device(dc.ptr, da.ptr, n, right.ptr, n)
        cudart.synchronize()
        c = dc.download(np.uint32, 2 * n)
        assert c[0] == 1 and not c[1:n].any() and c[n] == 0xFFFFFFFE and (c[n + 1:] == 0xFFFFFFFF).all()
    for x in (da, db, dc):
        x.free()
    assert big.device_errors() == 0


def test_batch_of_long_products(big):
    # a batch whose long products run one after the other beside a wave
    sizes = [(M + 1, M), (M // 2, M), (1000, 900), (M + 1, M)]
    A = [synth.operand(n, 50 + i) for i, (n, _) in enumerate(sizes)]
    B = [synth.operand(n, 60 + i) for i, (_, n) in enumerate(sizes)]
    da, db = [_device(x) for x in A], [_device(x) for x in B]
    db[3] = db[0]   # the same right operand
    dc = [cudart.DeviceBuffer(4 * (x + y)) for x, y in sizes]
    one = cudart.DeviceBuffer(4 * (2 * M + 1))
    big.batch_mul_device([c.ptr for c in dc], [x.ptr for x in da], [n for n, _ in sizes], [x.ptr for x in db],
                         [n for _, n in sizes])
    cudart.synchronize()
    for i, (x, y) in enumerate(sizes):
        big.set_prime_set(3)
        try:
            big.mul_device(one.ptr, da[i].ptr, x, db[i].ptr, y)
            cudart.synchronize()
        finally:
            big.set_prime_set(2)
        assert np.array_equal(dc[i].download(np.uint32, x + y), one.download(np.uint32, x + y)), i
    for buf in {id(b): b for b in da + db + dc + [one]}.values():
        buf.free()
    assert big.device_errors() == 0
