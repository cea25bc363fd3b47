"""Kernels that are launched beside another one start without waiting for what came
before, so an SM's L1 may hold the words that were at their inputs' addresses earlier:
those inputs have no load but one past L1 (on the CPU, by their type), and bursts that
take the same buffers again and again, with several ring sizes in a wave and more last
rounds than one launch takes, give the round-by-round prover's bytes (on the GPU)."""
import shutil
import subprocess

import pytest

from test_ring_emulation import CSRC, ROOT, _cuda_include


def test_inputs_are_read_past_l1(tmp_path):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    res = subprocess.run([cxx, "-std=c++17", "-I", str(inc), "-I", str(CSRC), "-x", "c++", "-c",
                          str(ROOT / "tests" / "native" / "beside_reads.cpp"), "-o", str(tmp_path / "beside_reads.o")],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr


@pytest.mark.gpu
def test_bursts_over_the_same_buffers():
    import damascus000_gb300 as D
    from damascus000_gb300 import synth
    epoch = bytes([6]) * 32
    # 20 of depth 6 (three launches of last rounds), and rings up to 2^9 in the same waves;
    # every file ends within a block, which takes the byte-wise unpacking
    sizes = [1_000 + 2_600 * i for i in range(20)] + [200_000, 213_100, 700_001, 900_000]
    with D.Context(0) as c, D.Engine(c) as eng:
        for turn in range(4):  # the same sizes, so the pool hands out the same memory
            files = [synth.random_file(120 + turn, n, i) for i, n in enumerate(sizes)]
            want = []
            for data, seed in files:
                p = D.DamascusProver(c, data, seed, epoch)
                n = p.rounds_total()
                records = [p.fold_round(r) for r in range(n)]
                want.append(p.statement() + n.to_bytes(8, "little") + b"".join(records) + p.final_opening())
                del p
            assert eng.prove_batch([(data, seed, epoch) for data, seed in files]) == want
            assert [c.prove(data, seed, epoch) for data, seed in files[:3] + files[-2:]] == want[:3] + want[-2:]
