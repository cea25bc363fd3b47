"""Single verifications of depth 11, whose transcript is on the device only for a call
with no other beside it: threads' verdicts, and a lone call after them, which is on the
device again once every place has been given back."""
import threading

import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([3]) * 32


def test_threads_then_alone(ctx):
    data, seed = synth.random_file(171, 14_000_000, 1)
    assert D.layout_for_byte_len(len(data))[0] == 11
    proof = ctx.prove(data, seed, EPOCH)
    wrong = proof[:-16] + bytes([proof[-16] ^ 1]) + proof[-15:]
    with D.Context(0) as c:
        bad = []

        def work(t):
            for _ in range(6):
                for p, ok in ((proof, True), (wrong, False), (proof[:-1], None)):
                    try:
                        got = c.verify(p, EPOCH)
                    except D.DamascusError as e:
                        got = None if e.code == D.EDESERIALIZE else e.code
                    if got is not ok and not (ok is None and got is False):
                        bad.append((t, ok, got))

        ts = [threading.Thread(target=work, args=(t,)) for t in range(4)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert bad == []
        c.set_profiling(True)
        c.reset_stats()
        assert c.verify(proof, EPOCH) and not c.verify(wrong, EPOCH)
        assert c.kernel_stat("transcript")[0] == 2 and c.reserved == 0
