"""The kernels' CRT into Z_q over its whole declared range, |X| <= 2^250 (the
largest commitment sum), on the CPU against Python integers."""
import random
import shutil
import subprocess
from math import prod

import pytest

from test_ring_emulation import CSRC, ROOT, _cuda_include

Q = (1 << 112) - 75


@pytest.mark.parametrize("bits", [0, 1, 27, 28, 111, 112, 113, 224, 246, 249, 250])
def test_crt_recovers_every_sum(tmp_path, bits):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = tmp_path / "crt"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(inc), "-I", str(CSRC), "-x", "c++",
                    str(ROOT / "tests" / "native" / "crt_residues.cpp"), str(CSRC / "dm_tables.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    primes = [int(p) for p in subprocess.run([str(exe)], input="", capture_output=True, text=True).stdout.split()]
    assert prod(primes) > 1 << 251
    rng = random.Random(bits)
    top = 1 << bits
    xs = [0, 1, top - 1, top] + [rng.randrange(top + 1) for _ in range(2000)]
    # sums whose residues are extreme: multiples of all primes but one, plus or minus one
    xs += [k * (prod(primes) // p) + e for p in primes for k in (1, p // 8) for e in (-1, 0, 1)]
    xs = [x for x in xs if 0 <= x <= top]
    xs += [-x for x in xs]
    lines = "\n".join(" ".join(str(x % p) for p in primes) for x in xs)
    out = subprocess.run([str(exe)], input=lines, capture_output=True, text=True, check=True).stdout.split()[9:]
    assert [int(o, 16) for o in out] == [x % Q for x in xs]
