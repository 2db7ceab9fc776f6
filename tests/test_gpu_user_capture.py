"""Products captured on a caller's own stream and replayed as a CUDA graph,
with other operands in the same buffers: every route of gbntt_mul_u32 (one
CTA, a cluster of CTAs, the pass chain with programmatic dependent launches,
the radix-3 and the outer stage), packed and negacyclic products. The first
capture of a length finds no pass twiddle tables and may build none. Replays
equal the 64-bit primes' products, which the other tests compare with GMP."""
import ctypes

import numpy as np
import pytest

from cryptography_gb300 import cudart

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fresh(engine):
    engine.teardown()
    engine.init(26)
    yield engine
    engine.teardown()
    engine.init(24)


def _capture(call):
    # the graph of call(stream) twice over, captured on a new stream
    rt = cudart.rt()
    stream, graph, ex = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    cudart.check(rt.cudaStreamCreate(ctypes.byref(stream)))
    cudart.check(rt.cudaStreamBeginCapture(stream, 2))   # relaxed
    try:
        call(stream)
        call(stream)
    finally:
        rc = rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
    cudart.check(rc)
    cudart.check(rt.cudaGraphInstantiate(ctypes.byref(ex), graph, ctypes.c_ulonglong(0)))
    cudart.check(rt.cudaGraphDestroy(graph))
    return stream, ex


def _check(g, call, ins, out, words, dtype, seed):
    # captured before the length has been run, and again after it
    rng = np.random.default_rng(seed)
    cudart.synchronize()
    for turn in range(2):
        stream, ex = _capture(call)
        for _ in range(2):
            for buf, n in ins:
                buf.upload(rng.integers(0, 1 << (8 * np.dtype(dtype).itemsize), n, dtype=np.uint64).astype(dtype))
            got = []
            cudart.check(cudart.rt().cudaMemset(out.ptr, 0, words * np.dtype(dtype).itemsize))
            cudart.check(cudart.rt().cudaGraphLaunch(ex, stream))
            cudart.synchronize()
            got.append(out.download(dtype, words))
            for primes in (2, 3):
                g.set_prime_set(primes)
                try:
                    call(None)
                    cudart.synchronize()
                finally:
                    g.set_prime_set(2)
                got.append(out.download(dtype, words))
            assert np.array_equal(got[0], got[2]) and np.array_equal(got[1], got[2]), turn
        cudart.check(cudart.rt().cudaGraphExecDestroy(ex))
        cudart.check(cudart.rt().cudaStreamDestroy(stream))
    for buf, _ in ins:
        buf.free()
    out.free()
    assert g.device_errors() == 0


@pytest.mark.parametrize("na,nb", [(100, 90), (1000, 1024), (3000, 1000), (50021, 43987), (1 << 18, 1 << 17),
                                   (3 << 17, 3 << 17), ((1 << 25) + 5, (1 << 25) - 7)])
def test_mul(fresh, na, nb):
    a, b, c = (cudart.DeviceBuffer(4 * n) for n in (na, nb, na + nb))
    _check(fresh, lambda st: fresh.mul_device(c.ptr, a.ptr, na, b.ptr, nb, st), [(a, na), (b, nb)], c, na + nb,
           np.uint32, na)


def test_packed(fresh):
    na, nb = 70001, 60011
    a, b, c = (cudart.DeviceBuffer(8 * n) for n in (na, nb, na + nb))

    def call(st):
        assert fresh.lib().gbntt_mul_u64(c.ptr, a.ptr, na, b.ptr, nb, st) == 0

    _check(fresh, call, [(a, na), (b, nb)], c, na + nb, np.uint64, na)


@pytest.mark.parametrize("log_n", [6, 10, 14, 19])
def test_negacyclic(fresh, log_n):
    n = 1 << log_n
    f, h, o = (cudart.DeviceBuffer(8 * k) for k in (n, n, 4 * n))
    _check(fresh, lambda st: fresh.negacyclic_mul_device(o.ptr, f.ptr, h.ptr, log_n, st), [(f, n), (h, n)], o, 4 * n,
           np.uint64, log_n)
