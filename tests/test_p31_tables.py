"""The tables of powers that every engine initialisation fills (p31_powers,
gbntt_p31.cuh): compiled for the host and compared with Python's powers, at
lengths that are and are not powers of two, for every prime."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cryptography_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
P, GEN = (2013265921, 1811939329, 2113929217), (31, 13, 5)
LENGTHS = (1, 2, 3, 5, 64, 1000, 1024, 3 * 1024, 1 << 15)

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "gbntt_p31.cuh"
int main()
{
    unsigned long long n, w, p;
    while (scanf("%llu %llu %llu", &n, &w, &p) == 3) {
        std::vector<uint32_t> t(n + 1, 0xdeadbeefu);
        gbntt::p31_powers(t.data(), n, w, p);
        for (uint32_t x : t) printf("%u\n", x);
    }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("powers")
    (d / "powers.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, "-I", os.path.join(CSRC, "..", "..", "include"), "-I",
                    os.path.join(CUDA, "include"), "powers.cpp", "-o", "powers"], cwd=d, check=True)
    return str(d / "powers")


def test_powers(program):
    cases = []
    for p, g in zip(P, GEN):
        root = pow(g, (p - 1) >> 25, p)
        for n in LENGTHS:
            cases += [(n, w, p) for w in (1, p - 1, g, root, pow(root, p - 2, p), pow(root, 1 << 15, p))]
    text = "".join("%d %d %d\n" % c for c in cases)
    out = iter(subprocess.run([program], input=text, capture_output=True, text=True, check=True).stdout.split())
    for n, w, p in cases:
        x = 1
        for i in range(n):
            assert int(next(out)) == (x << 32) % p, (n, w, p, i)
            x = x * w % p
        assert int(next(out)) == 0xdeadbeef, (n, w, p)   # nothing beyond the table
    assert next(out, None) is None
