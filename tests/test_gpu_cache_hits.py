"""A verification that reads its generators from the provers' cache counts one hit,
through the service and by itself, with the transcript on the host (depth 7) and on the
device (depth 8)."""
import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([3]) * 32
SEED = bytes([9]) * 32


@pytest.mark.parametrize("n", [100_000, 300_000])
def test_one_hit_a_verification(n):
    files = [synth.random_file(151, n - i, i)[0] for i in range(5)]
    with D.Context(0) as c:
        c.set_generator_cache(1 << 30)
        proofs = [c.prove(f, SEED, EPOCH) for f in files]  # noted, filled, then hit
        hits = lambda: c.generator_cache_stats()["hits"]
        assert hits() == 3
        for i, p in enumerate(proofs):
            assert c.verify(p, EPOCH) and hits() == 4 + i
        with D.VerifyService(c) as svc:
            assert svc.verify_batch(proofs, EPOCH) == [True] * 5
        assert hits() == 13
