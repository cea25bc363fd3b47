"""Last rounds in one launch inside the engine: proofs of depth 6 (from the Init stage
on) and deeper (from a polynomial stage on) together, more than one launch takes, with
a generator cache, against the round-by-round prover's bytes; and with the launch trace
on, which runs them stage by stage."""
import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth
from test_gpu_tail import _round_by_round

pytestmark = pytest.mark.gpu
EPOCH = bytes([7]) * 32  # test_gpu_tail's
SIZES = [0, 1, 20_000, 53_248, 53_249, 213_000, 213_100, 900_000]


@pytest.mark.parametrize("copies,cache", [(1, False), (3, True)])
def test_engine_tail_equals_round_by_round(ctx, copies, cache):
    seed = bytes([8]) * 32
    files = [synth.random_file(95, n, n % 5)[0] for n in SIZES]
    want = [_round_by_round(ctx, f, seed) for f in files]
    with D.Context(0) as c:
        if cache:
            c.set_generator_cache(1 << 30)
        with D.Engine(c) as eng:
            assert eng.prove_batch([(f, seed, EPOCH) for f in files] * copies) == want * copies
            c.trace_start()
            assert eng.prove_batch([(f, seed, EPOCH) for f in files]) == want
            kinds = {r[0] for r in c.trace_read(stop=True)}
        assert "last_rounds" not in kinds
