"""The device's inverse mod q (binary extended gcd), compiled for the CPU, against
Python integers: small values, powers of two, values around q and random ones."""
import random
import shutil
import subprocess

import pytest

from test_ring_emulation import CSRC, ROOT, _cuda_include

Q = (1 << 112) - 75


def test_inverse_matches_fermat(tmp_path):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = tmp_path / "inverse"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(inc), "-I", str(CSRC), "-x", "c++",
                    str(ROOT / "tests" / "native" / "field_inverse.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    rng = random.Random(5)
    xs = [0] + [x % Q for k in range(113) for x in ((1 << k) - 1, 1 << k, (1 << k) + 1, Q - (1 << k), Q // (k + 1))]
    xs += [rng.randrange(Q) for _ in range(20000)]
    out = subprocess.run([str(exe)], input="\n".join("%x" % x for x in xs), capture_output=True, text=True,
                         check=True).stdout.split("\n")[:len(xs)]
    for x, line in zip(xs, out):
        got, same = line.split()
        assert int(got, 16) == (pow(x, -1, Q) if x else 0) and same == "1", x
