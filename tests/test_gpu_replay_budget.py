"""What one verification holds is its generators and the first fold's half and nothing
besides: in a budget of exactly that its transcript still runs on the device, and as
many calls at once as the budget has such footprints all run."""
import threading

import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([3]) * 32


def _footprint(dim):
    family = dim * 8 * dim * 16
    return family + ((family // 2 + 16 + 255) & ~255)


# depths 8, where the room beside the folds is tightest, to 10
@pytest.mark.parametrize("n", [300_000, 900_000, 3_500_000])
def test_transcript_runs_in_one_footprint(ctx, n):
    data, seed = synth.random_file(141, n, 1)
    _, dim = D.layout_for_byte_len(n)
    proof = ctx.prove(data, seed, EPOCH)
    wrong = proof[:-16] + bytes([proof[-16] ^ 1]) + proof[-15:]
    with D.Context(0, hbm_budget_bytes=_footprint(dim)) as tight:
        tight.set_profiling(True)
        assert tight.verify(proof, EPOCH) and not tight.verify(wrong, EPOCH)
        # the opening's check follows the transcript and the folds on the device
        assert [(tight.kernel_stat(k) or (0,))[0] for k in ("transcript", "opening")] == [2, 2]
        assert tight.reserved == 0


def test_calls_at_once_under_as_many_footprints(ctx):
    threads, calls = 3, 60
    files = [synth.random_file(142, 300_000 - t, t) for t in range(threads)]
    _, dim = D.layout_for_byte_len(300_000)
    proofs = [ctx.prove(data, seed, EPOCH) for data, seed in files]
    wrong = []
    with D.Context(0, hbm_budget_bytes=threads * _footprint(dim)) as tight:
        start = threading.Barrier(threads)

        def work(t):
            start.wait()
            for _ in range(calls):
                rc = tight._lib.damascus_verify(tight.handle, proofs[t], len(proofs[t]), EPOCH)
                if rc:
                    wrong.append(rc)

        ts = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert wrong == []
        assert tight.reserved == 0
