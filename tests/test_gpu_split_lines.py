"""Batch products on both sides of the lines of the split rule: the longer
operand 16 times the shorter, a shorter operand of 64 limbs, and products that
fit one CTA (2^12 coefficients), which are never split. The launch log shows
which were split: into chunk products of four times the shorter operand's
length (all in one CTA here) instead of one of the product's own."""
import numpy as np
import pytest

import oracle
from cryptography_gb300 import cudart

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb,split", [
    (8192, 512, True), (8191, 512, False), (512, 8192, True), (512, 8191, False),   # 16 x the shorter
    (1 << 17, 64, True), (1 << 17, 63, False),                                      # 64 limbs
    (4033, 64, False), (4034, 64, True), (64, 4033, False), (64, 4034, True),       # 2^12 coefficients
])
def test_split_lines(engine, na, nb, split):
    rng = np.random.default_rng(na * 31 + nb)
    full = lambda n: np.full(n, 0xFFFFFFFF, dtype=np.uint32)  # noqa: E731
    rnd = lambda n: rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)  # noqa: E731
    for a, b in ((rnd(na), rnd(nb)), (full(na), full(nb))):
        da, db, dc = (cudart.DeviceBuffer(4 * n) for n in (na, nb, na + nb))
        da.upload(a)
        db.upload(b)
        engine.launch_log(True)
        try:
            engine.batch_mul_device([dc.ptr], [da.ptr], [na], [db.ptr], [nb])
            cudart.synchronize()
            launches = [r[:2] for r in engine.launch_records()]
        finally:
            engine.launch_log(False)
        L = (na + nb - 2).bit_length()
        chunks = (4 * min(na, nb) - 1).bit_length()   # (log2; the last chunk may be shorter)
        blocks = [p for kind, p in launches if kind == "block_product"]
        if split:
            assert len(blocks) == len(launches) and max(blocks) == chunks < L, launches
        elif L <= 12:
            assert launches == [("block_product", L)], launches
        else:
            assert not blocks and launches[-1][0] == "garner_carry", launches
        want = np.zeros(na + nb, dtype=np.uint32)
        r = oracle.gmp_mul(a, b)
        want[:len(r)] = r
        assert np.array_equal(dc.download(np.uint32, na + nb), want), (na, nb)
        for x in (da, db, dc):
            x.free()
    assert engine.device_errors() == 0
