"""Commitments whose columns are summed in 1 .. 16 parts (a part has eight columns or
more, and the finish loads four at a time), in rings on both sides of 2^10, against the
oracle."""
import random

import pytest

import damascus000_gb300 as D

pytestmark = pytest.mark.gpu

Q = (1 << 112) - 75


@pytest.mark.parametrize("n", [16, 64, 1024, 2048])
@pytest.mark.parametrize("N", [8, 9, 24, 25, 33, 40, 65, 129])
def test_commit_by_parts(ctx, oracle_lib, N, n):
    rng = random.Random(N * 10_007 + n)
    w = D.fe_vec([Q - 1] * n + [rng.randrange(Q) for _ in range(N * n - n)])
    seed = rng.randbytes(32)
    g = oracle_lib.derive_generators(oracle_lib.derive_subseed(seed, b"g0"), N, n)
    assert ctx.commit_witness(w, N, n, seed) == oracle_lib.commit_with_generators(w, g, N, n, threads=8)
