"""The transforms' padded shared-memory exchanges (every word distinct, inside its
row's range, no bank conflict, base plus constant) and the stored slot order, at
every ring size, on the CPU."""
import shutil
import subprocess

import pytest

from test_ring_emulation import CSRC, ROOT, _cuda_include


def test_row_layouts(tmp_path):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = tmp_path / "row_layouts"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(inc), "-I", str(CSRC), "-x", "c++",
                    str(ROOT / "tests" / "native" / "row_layouts.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
