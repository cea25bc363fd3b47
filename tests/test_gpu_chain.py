"""prove()'s chain of launches (challenges on the device) against the round-by-round
prover, whose challenges the host computes: the same proof bytes at every depth and
around the layout's edges, under a budget without room for the chain's buffers, and
with the generator cache filling and hitting."""
import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([3]) * 32


def _round_by_round(ctx, data, seed):
    p = D.DamascusProver(ctx, data, seed, EPOCH)
    n = p.rounds_total()
    records = [p.fold_round(r) for r in range(n)]
    return p.statement() + n.to_bytes(8, "little") + b"".join(records) + p.final_opening()


# one byte, depth 6's last coefficient and the next depth's first, up to rings of
# 2^10; the largest also spreads a challenge's chunks over several blocks
@pytest.mark.parametrize("n", [0, 1, 53_248, 53_249, 13 * 128 * 128, 13 * 128 * 128 + 1, 700_001, 851_968, 900_000,
                               3_500_000])
def test_chain_equals_round_by_round(ctx, n):
    data, seed = synth.random_file(61, n, n % 997)
    assert ctx.prove(data, seed, EPOCH) == _round_by_round(ctx, data, seed)


def test_without_room_for_the_chain(ctx):
    data, seed = synth.random_file(62, 300_000, 1)
    want = ctx.prove(data, seed, EPOCH)
    with D.Context(0, hbm_budget_bytes=D.prover_footprint(len(data))) as tight:
        assert tight.prove(data, seed, EPOCH) == want
        assert tight.reserved == 0
    with D.Context(0, hbm_budget_bytes=D.prover_footprint(len(data)) - 256) as small:
        with pytest.raises(D.DamascusError) as e:
            small.prove(data, seed, EPOCH)
        assert e.value.code == D.ENOMEM_BUDGET and small.reserved == 0


def test_chain_with_generator_cache(ctx):
    files = [synth.random_file(63, n, i)[0] for i, n in enumerate([300_000, 500_000, 300_000])]
    seed = bytes([9]) * 32
    want = [ctx.prove(f, seed, EPOCH) for f in files]
    with D.Context(0) as c:
        c.set_generator_cache(4 << 30)
        assert [c.prove(f, seed, EPOCH) for f in files + files] == want + want
        assert c.generator_cache_stats()["hits"] >= 4
