"""Commitments whose witness is copied beside the generators' expansion (above 128 KiB)
against the oracle, on both sides of the line and from two threads of one context."""
import random
import threading

import pytest

import damascus000_gb300 as D

pytestmark = pytest.mark.gpu


Q = (1 << 112) - 75


def _case(N, n):
    rng = random.Random(N * 10_007 + n)
    w = D.fe_vec([Q - 1, 0] + [rng.randrange(Q) for _ in range(N * n - 2)])
    return w, rng.randbytes(32)


@pytest.mark.parametrize("N,n", [(16, 512), (17, 512), (1, 8192), (3, 4096), (129, 64), (4097, 2)])
def test_commit_around_the_line(ctx, oracle_lib, N, n):
    w, seed = _case(N, n)
    g = oracle_lib.derive_generators(oracle_lib.derive_subseed(seed, b"g0"), N, n)
    assert ctx.commit_witness(w, N, n, seed) == oracle_lib.commit_with_generators(w, g, N, n, threads=8)


def test_two_threads_of_one_context(ctx):
    cases = [(40, 256), (9, 1024)]
    data = [_case(*c) for c in cases]
    want = [ctx.commit_witness(w, *c, seed) for c, (w, seed) in zip(cases, data)]
    got = [[], []]

    def work(i):
        w, seed = data[i]
        got[i] = [ctx.commit_witness(w, *cases[i], seed) for _ in range(20)]

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [[want[0]] * 20, [want[1]] * 20]
