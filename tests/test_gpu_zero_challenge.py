"""What follows when a challenge candidate computed on the device is zero, which the
transcript's counter then resolves on the host: prove() starts over stage by stage, an
engine goes on from where its last rounds began, a verification replays on the host.  No
input gives such a candidate; the library is told to take finished chains for ones with
it, and proofs and verdicts have to be the same."""
import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([3]) * 32
SEED = bytes([9]) * 32
SIZES = [1, 20_000, 53_248, 60_000, 213_000, 300_000]  # depths 6, 7 and 8


def _pretend(c, n):
    c.check(c._lib.damascus_test_zero_challenges(c.handle, n), "pretend")


@pytest.fixture(scope="module")
def files(ctx):
    data = [synth.random_file(161, n, i)[0] for i, n in enumerate(SIZES)]
    return data, [ctx.prove(f, SEED, EPOCH) for f in data]


@pytest.mark.parametrize("cache", [False, True])
def test_prove_starts_over(files, cache):
    data, want = files
    with D.Context(0) as c:
        if cache:
            c.set_generator_cache(1 << 30)
        for _ in range(3):  # the family noted, filled and hit
            for f, w in zip(data, want):
                _pretend(c, 1)
                c.set_profiling(True)
                c.reset_stats()
                assert c.prove(f, SEED, EPOCH) == w
                # the chain, then the stages: the file is hashed in both
                assert c.kernel_stat("last_rounds")[0] == 1 and c.kernel_stat("file_hash")[0] >= 2
                assert c.prove(f, SEED, EPOCH) == w  # not pretended
                assert c.kernel_stat("last_rounds")[0] == 2


# some and all of a batch's last rounds
@pytest.mark.parametrize("zeros", [1, 4, 100])
@pytest.mark.parametrize("cache", [False, True])
def test_engine_goes_on(files, zeros, cache):
    data, want = files
    with D.Context(0) as c:
        if cache:
            c.set_generator_cache(1 << 30)
        with D.Engine(c) as eng:
            for _ in range(3):
                _pretend(c, zeros)
                assert eng.prove_batch([(f, SEED, EPOCH) for f in data * 2]) == want * 2
            st = eng.stats()
        assert st["failed"] == 0 and st["completed"] == 6 * len(data)


@pytest.mark.parametrize("cache", [False, True])
def test_verification_replays_on_the_host(files, cache):
    proof = files[1][SIZES.index(300_000)]
    wrong = proof[:-16] + bytes([proof[-16] ^ 1]) + proof[-15:]
    with D.Context(0) as c:
        if cache:
            c.set_generator_cache(1 << 30)
            for f in files[0][-1:] * 2:
                c.prove(f, SEED, EPOCH)
        c.set_profiling(True)
        for _ in range(3):
            for p, ok in ((proof, True), (wrong, False)):
                _pretend(c, 1)
                assert c.verify(p, EPOCH) == ok
                assert c.verify(p, EPOCH) == ok
        # on the device every time: a call that goes on to the host gives its place back
        assert c.kernel_stat("transcript")[0] == 12
        with D.VerifyService(c) as svc:
            for _ in range(3):
                _pretend(c, 3)
                assert svc.verify_batch([proof, wrong] * 3, EPOCH) == [True, False] * 3
