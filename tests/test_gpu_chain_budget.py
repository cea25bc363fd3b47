"""What one prove() call holds is its footprint and nothing besides: in a budget of
exactly that it still runs as one chain of launches, and as many calls at once as the
budget has footprints all run."""
import threading

import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([3]) * 32


# depth 6 (no challenge before the last rounds) to 10, host and device files
@pytest.mark.parametrize("n", [1, 53_248, 200_000, 900_000, 3_500_000])
def test_chain_runs_in_one_footprint(ctx, n):
    import torch
    data, seed = synth.random_file(131, n, 1)
    want = ctx.prove(data, seed, EPOCH)
    file = torch.frombuffer(bytearray(data), dtype=torch.uint8).cuda()
    torch.cuda.synchronize()
    with D.Context(0, hbm_budget_bytes=D.prover_footprint(n)) as tight:
        tight.set_profiling(True)
        assert tight.prove(data, seed, EPOCH) == want
        assert tight.prove_device(file.data_ptr(), n, seed, EPOCH) == want
        stat = tight.kernel_stat("last_rounds")
        assert stat and stat[0] == 2  # one launch of last rounds in each
        assert tight.reserved == 0


def test_calls_at_once_under_as_many_footprints(ctx):
    n, threads, calls = 300_000, 3, 40
    files = [synth.random_file(132, n - t, t) for t in range(threads)]
    want = [ctx.prove(data, seed, EPOCH) for data, seed in files]
    wrong = []
    with D.Context(0, hbm_budget_bytes=threads * D.prover_footprint(n)) as tight:
        start = threading.Barrier(threads)

        def work(t):
            start.wait()
            for _ in range(calls):
                try:
                    if tight.prove(*files[t], EPOCH) != want[t]:
                        wrong.append("proof")
                except D.DamascusError as e:
                    wrong.append(e.code)

        ts = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert wrong == []
        assert tight.reserved == 0


def test_chain_beside_cached_families(ctx):
    """A budget filled by families that another proof may need again: they give way to the
    call's footprint and to no more."""
    seed = bytes([9]) * 32
    small = [synth.random_file(133, 60_000, i)[0] for i in range(3)]
    big = synth.random_file(133, 900_000, 9)[0]
    want = [ctx.prove(f, seed, EPOCH) for f in small + [big]]
    with D.Context(0, hbm_budget_bytes=D.prover_footprint(len(big))) as c:
        c.set_generator_cache(1 << 30)
        assert [c.prove(f, seed, EPOCH) for f in small] == want[:3]
        assert c.generator_cache_stats()["fills"] == 1
        c.set_profiling(True)
        assert c.prove(big, seed, EPOCH) == want[3]
        assert c.kernel_stat("last_rounds")[0] == 1
        assert c.generator_cache_stats()["bytes"] == 0 and c.reserved == 0
