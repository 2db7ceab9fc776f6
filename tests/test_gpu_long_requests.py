"""Served requests longer than the 31-bit primes' transforms (above 3 2^25
points): they run as waves on q0 with p3, beside shorter ones on the 31-bit
primes, and equal the 64-bit primes' products."""
import numpy as np
import pytest

from cryptography_gb300 import cudart, synth

pytestmark = pytest.mark.gpu

M = 1 << 25


@pytest.fixture(scope="module")
def big(engine):
    engine.teardown()
    engine.init(27)
    yield engine
    engine.teardown()
    engine.init(24)


def test_long_served_requests(big):
    # 2^26 points twice and by one right operand, 3 2^25 and 2^27 points,
    # and requests on the 31-bit primes between them
    sizes = [(M + 1, M), (1000, 900), (M + M // 2, M // 3), (2 * M, M), (M // 2, M // 2), (2 * M + 3, M + 9)]
    A = [synth.operand(n, 10 + i) for i, (n, _) in enumerate(sizes)]
    B = [synth.operand(n, 20 + i) for i, (_, n) in enumerate(sizes)]
    bufs = []

    def up(x):
        bufs.append(cudart.DeviceBuffer(4 * len(x)))
        bufs[-1].upload(x)
        return bufs[-1]

    reqs = [(up(a), len(a), up(b), len(b)) for a, b in zip(A, B)]
    reqs.append(reqs[0][:1] + (M - 7,) + reqs[0][2:])   # a prefix of A by the same right operand
    out = [cudart.DeviceBuffer(4 * (na + nb)) for _, na, _, nb in reqs]
    srv = big.Server(slots=2, slot_log=27)
    try:
        t = [srv.submit(c.ptr, a.ptr, na, b.ptr, nb) for c, (a, na, b, nb) in zip(out, reqs)]
        for ticket in t:
            srv.wait(ticket, 120.0)
        assert srv.stats()["device_errors"] == 0
    finally:
        srv.stop()
    one = cudart.DeviceBuffer(4 * max(na + nb for _, na, _, nb in reqs))
    big.set_prime_set(3)
    try:
        for c, (a, na, b, nb) in zip(out, reqs):
            big.mul_device(one.ptr, a.ptr, na, b.ptr, nb)
            cudart.synchronize()
            assert np.array_equal(c.download(np.uint32, na + nb), one.download(np.uint32, na + nb)), (na, nb)
    finally:
        big.set_prime_set(2)
    for x in bufs + out + [one]:
        x.free()
    assert big.device_errors() == 0
