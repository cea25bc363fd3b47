"""Whole ring products through the transforms' padded exchanges and stored slot order, as
the radix-16 kernels take them, on the CPU at every ring size from 2^5 on."""
import shutil
import subprocess

import pytest

from test_ring_emulation import CSRC, ROOT, _cuda_include


def test_products_through_padded_exchanges(tmp_path):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = tmp_path / "padded_transforms"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(inc), "-I", str(CSRC), "-x", "c++",
                    str(ROOT / "tests" / "native" / "padded_transforms.cpp"), str(CSRC / "dm_tables.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout
