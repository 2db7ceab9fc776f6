"""Products of 2 2^25 + 1 to 3 2^25 coefficients: the radix-3 stage takes
them, and with it switched off the outer stage, whose products then equal the
64-bit primes'."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("knobs,stage", [({}, "radix3"), ({"GBNTT_RADIX3": "0"}, "outer"),
                                         ({"GBNTT_RADIX3_MIN_LOG": "26"}, "outer")])
def test_three_blocks(knobs, stage):
    body = textwrap.dedent("""
        import sys
        sys.path.insert(0, %r)
        import numpy as np
        import cryptography_gb300 as g
        from cryptography_gb300 import cudart, synth
        g.init(27)
        M = 1 << 25
        for na, nb in ((M + 2, M), (2 * M, M), (2 * M + 5, 2 * M // 3)):
            da, db, dc = (cudart.DeviceBuffer(4 * n) for n in (na, nb, na + nb))
            da.upload(synth.operand(na, 1))
            db.upload(synth.operand(nb, 2))
            got = []
            for primes in (2, 3):
                g.set_prime_set(primes)
                g.launch_log(True)
                g.mul_device(dc.ptr, da.ptr, na, db.ptr, nb)
                cudart.synchronize()
                kinds = {r[0] for r in g.launch_records()}
                g.launch_log(False)
                if primes == 2:
                    assert {k[:-4] for k in kinds if k.startswith(("outer", "radix3"))} == {%r}, kinds
                got.append(dc.download(np.uint32, na + nb))
            assert np.array_equal(*got), (na, nb)
            for x in (da, db, dc):
                x.free()
        assert g.device_errors() == 0
        print("fine")
    """ % (ROOT, stage))
    r = subprocess.run([sys.executable, "-c", body], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, **knobs))
    assert r.returncode == 0 and "fine" in r.stdout, r.stderr[-2000:]
