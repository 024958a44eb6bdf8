"""Sums of the Arnoldi step and of the cycle start (csrc/arnoldi.cu) over long complex64 vectors, by a host program of their
own (tests/c_host/arnoldi_sums.cu) that is linked with the library.

The vectors repeat one value, so every addition of a chain rounds the same way and a chain's error shows at its full size.
A thread adds up to 16 squares in FP32: the i-th addition is off by at most half a unit in the last place of i squares, each
square by half of its own, so the sum by at most ((1 + ... + 16) / 16 + 1) 2^-24 = 5.7e-7.  (One chain over a thread's part of
the longest vectors here has 498.)
"""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(g2lib, tmp_path_factory):
    from giem2g_b200 import build as b
    exe = str(tmp_path_factory.mktemp("sums") / "arnoldi_sums")
    libdir = os.path.dirname(b.LIB)
    cmd = [b.NVCC, *b.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I", b.CSRC, "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", "c_host", "arnoldi_sums.cu"), "-L", libdir, "-lgiem2g_b200",
           "-Xlinker", "-rpath", "-Xlinker", libdir, "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return exe


@pytest.mark.parametrize("elements,basis,instances", [(3 * 256 * 256 * 48, 10, 2), (3 * 128 * 128 * 32, 4, 4),
                                                      (3 * 128 * 128 * 32, 11, 2), (3 * 128 * 128 * 32, 31, 4),
                                                      (3 * 64 * 64 * 16, 1, 1), (12, 2, 1)])
def test_sums_of_one_repeated_value(program, elements, basis, instances):
    for re, im in ((1.0, 0.7), (0.3, 0.9), (1.1, 0.2), (0.77, 0.61)):
        r = subprocess.run([program, str(elements), str(basis), str(instances), str(re), str(im)], capture_output=True,
                           text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        err, step, start = r.stdout.split()[-3:]
        assert int(err) == 0 and float(step) < 5.7e-7 and float(start) < 5.7e-7, (re, im, step, start)
