"""Kernels of a stage that run side by side (the file's hash, unpacking and generators;
the finishes of two ring sizes) against the round-by-round prover: files around one
hash group (128 chunks: one or two hash kernels), and an engine burst with more jobs of
a kind than one launch takes."""
import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([6]) * 32


def _round_by_round(ctx, data, seed):
    p = D.DamascusProver(ctx, data, seed, EPOCH)
    n = p.rounds_total()
    records = [p.fold_round(r) for r in range(n)]
    return p.statement() + n.to_bytes(8, "little") + b"".join(records) + p.final_opening()


@pytest.mark.parametrize("n", [131_071, 131_072, 131_073, 262_145])
def test_around_a_hash_group(ctx, n):
    data, seed = synth.random_file(91, n, n % 7)
    want = _round_by_round(ctx, data, seed)
    for _ in range(3):
        assert ctx.prove(data, seed, EPOCH) == want


def test_burst_of_more_jobs_than_a_launch(ctx):
    files = [synth.random_file(92, 53_000 + 7_000 * (i % 9), i) for i in range(90)]
    want = [ctx.prove(data, seed, EPOCH) for data, seed in files]
    with D.Engine(ctx) as eng:
        tickets = [eng.submit(data, seed, EPOCH) for data, seed in files]
        done = {t: proof for t, proof, _ in eng.as_completed(tickets)}
    assert [done[t] for t in tickets] == want
