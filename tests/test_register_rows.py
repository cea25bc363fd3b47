"""Transforms of a whole row in registers at rings 2^0 .. 2^5, on the CPU, against
evaluation at the slots' points."""
import shutil
import subprocess

import pytest

from test_ring_emulation import CSRC, ROOT, _cuda_include


def test_register_rows(tmp_path):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = tmp_path / "register_rows"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(inc), "-I", str(CSRC), "-x", "c++",
                    str(ROOT / "tests" / "native" / "register_rows.cpp"), str(CSRC / "dm_tables.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
