"""Verifications by several threads of one context, more than take their transcript on
the device at once, and a service with and without cached families: the same verdicts
on both routes, and the count of device transcripts back at zero (a later single call
gives its verdict as before)."""
import threading

import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([9]) * 32


@pytest.fixture(scope="module")
def proofs(ctx):
    out = []
    for i in range(6):
        data, seed = synth.random_file(97, 300_000 + 200_000 * i, i)
        good = ctx.prove(data, seed, EPOCH)
        out += [(good, True), (good[:-16] + bytes([good[-16] ^ 1]) + good[-15:], False)]
    return out


def test_threads_of_one_context(ctx, proofs):
    got = [[] for _ in proofs]

    def work(i):
        got[i] = [ctx.verify(proofs[i][0], EPOCH) for _ in range(6)]

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(proofs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [[ok] * 6 for _, ok in proofs]
    assert [ctx.verify(p, EPOCH) for p, _ in proofs] == [ok for _, ok in proofs]


@pytest.mark.parametrize("cache", [0, 8 << 30])
def test_service_with_and_without_families(ctx, proofs, cache):
    with D.VerifyService(ctx, cache_bytes=cache) as s:
        for _ in range(3):  # host, host and filling the cache, device (with a cache)
            assert s.verify_batch([p for p, _ in proofs], EPOCH) == [ok for _, ok in proofs]
