"""A batch that is refused computes none of its products: also not one that is
too long for a wave and runs by itself."""
import numpy as np
import pytest

from cryptography_gb300 import cudart, synth

pytestmark = pytest.mark.gpu

M = 1 << 25


@pytest.fixture(scope="module")
def big(engine):
    engine.teardown()
    engine.init(26)
    yield engine
    engine.teardown()
    engine.init(24)


@pytest.mark.parametrize("na,nb", [(1000, 900), (M, M - 5)])
def test_refused_batch_writes_nothing(big, na, nb):
    a, b = cudart.DeviceBuffer(4 * na), cudart.DeviceBuffer(4 * nb)
    c = cudart.DeviceBuffer(4 * (na + nb))
    a.upload(synth.operand(na, 1))
    b.upload(synth.operand(nb, 2))
    mark = np.full(na + nb, 0x5A5A5A5A, dtype=np.uint32)
    c.upload(mark)
    # the second product would need 2^27 coefficients (its operands are not read)
    with pytest.raises(big.EngineError) as ei:
        big.batch_mul_device([c.ptr, c.ptr], [a.ptr, a.ptr], [na, 1 << 26], [b.ptr, b.ptr], [nb, 1 << 26])
    assert ei.value.code == big.GBNTT_ERR_SIZE
    cudart.synchronize()
    assert np.array_equal(c.download(np.uint32, na + nb), mark)
    big.batch_mul_device([c.ptr], [a.ptr], [na], [b.ptr], [nb])
    cudart.synchronize()
    got = c.download(np.uint32, na + nb)
    big.mul_device(c.ptr, a.ptr, na, b.ptr, nb)
    cudart.synchronize()
    assert np.array_equal(c.download(np.uint32, na + nb), got) and not np.array_equal(got, mark)
    for x in (a, b, c):
        x.free()
    assert big.device_errors() == 0
