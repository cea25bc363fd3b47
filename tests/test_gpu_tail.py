"""The last rounds in one launch against the round-by-round prover (challenges on the
host, a kernel per operation): whole proofs of depth 6 from it, and the last six
rounds of deeper ones, over witnesses with few, half and all columns nonzero, of the
largest and smallest coefficients, and with the generators in a cache."""
import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([7]) * 32


def _round_by_round(ctx, data, seed):
    p = D.DamascusProver(ctx, data, seed, EPOCH)
    n = p.rounds_total()
    records = [p.fold_round(r) for r in range(n)]
    return p.statement() + n.to_bytes(8, "little") + b"".join(records) + p.final_opening()


FILES = {
    "empty": b"",
    "one column": synth.random_file(71, 13 * 64, 0)[0],
    "past half the columns": synth.random_file(72, 13 * 64 * 32 + 1, 1)[0],
    "depth 6 in full": synth.random_file(73, 13 * 64 * 64, 2)[0],
    "zeros": bytes(50_000),
    "ones": b"\xff" * 53_248,
    "depth 7": synth.random_file(74, 13 * 64 * 64 + 1, 3)[0],
    "depth 8, sparse": bytes(400_000) + b"\x01",
}


@pytest.mark.parametrize("name", FILES)
def test_tail_equals_round_by_round(ctx, name):
    data, seed = FILES[name], bytes([len(name)]) * 32
    proof = ctx.prove(data, seed, EPOCH)
    assert proof == _round_by_round(ctx, data, seed)
    assert ctx.verify(proof, EPOCH)


def test_tail_reads_cached_generators(ctx):
    seed = bytes([5]) * 32
    files = [FILES["one column"], FILES["depth 6 in full"], FILES["depth 7"]]
    want = [ctx.prove(f, seed, EPOCH) for f in files]
    with D.Context(0) as c:
        c.set_generator_cache(1 << 30)
        assert [c.prove(f, seed, EPOCH) for f in files + files] == want + want
        # a family is noted at its first use, filled at its second and hit from its third on:
        # depth 6 is used four times, depth 7 twice
        assert c.generator_cache_stats()["hits"] == 2
