"""Verification of proofs of depth 8, the smallest whose transcript the device takes,
and of depth 11, whose first stages hash several passes' worth of chunks per block,
against the round-by-round verifier: honest proofs and one changed byte per part."""
import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth
from test_gpu_replay import EPOCH, _offsets, _round_by_round, _verify

pytestmark = pytest.mark.gpu


# depth 8's smallest and largest file, and a file of depth 11
@pytest.mark.parametrize("n", [13 * 128 * 128 + 1, 13 * 256 * 256, 13 * 1024 * 1024 + 1])
def test_first_and_last_sizes(ctx, n):
    data, seed = synth.random_file(81, n, 2)
    _, dim = D.layout_for_byte_len(n)
    proof = ctx.prove(data, seed, EPOCH)
    assert _verify(ctx, proof) == _round_by_round(ctx, proof, dim) == 0
    for what, at in _offsets(dim).items():
        bad = bytearray(proof)
        bad[at] ^= 1
        assert _verify(ctx, bytes(bad)) == D.EVERIFY, what
