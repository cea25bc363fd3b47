"""Verification with the transcript on the device (depth 9 on) against the
round-by-round verifier, whose transcript the host replays: the same verdict for
honest proofs, for changes in every part of a proof, for words at or above q, and
for proofs that only the host path takes."""
import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
EPOCH = bytes([3]) * 32
Q = (1 << 112) - 75


def _verify(ctx, proof, epoch=EPOCH):
    return ctx._lib.damascus_verify(ctx.handle, proof, len(proof), epoch)


def _round_by_round(ctx, proof, dim, epoch=EPOCH):
    st = D.statement_size(dim)
    v = D.DamascusVerifier(ctx, proof[:st], epoch)
    at, n = st + 8, dim
    while n > 1:
        size = D.record_size(n, n // 2)
        rc = v.update_commitment(proof[at:at + size])
        if rc:
            return rc
        at, n = at + size, n // 2
    return v.verify_final_opening(proof[at:at + 16])


@pytest.fixture(scope="module", params=[900_000, 5_000_000])  # rings of 2^9 and 2^10
def case(ctx, request):
    data, seed = synth.random_file(71, request.param, 1)
    _, dim = D.layout_for_byte_len(len(data))
    return ctx.prove(data, seed, EPOCH), dim


def test_honest_and_wrong_epoch(ctx, case):
    proof, dim = case
    assert _verify(ctx, proof) == _round_by_round(ctx, proof, dim) == 0
    other = bytes([4]) * 32
    assert _verify(ctx, proof, other) == _round_by_round(ctx, proof, dim, other) == D.EVERIFY
    assert _verify(ctx, proof + b"tail") == 0  # what follows the opening is not read


def _offsets(dim):
    st = D.statement_size(dim)
    module = lambda n: 8 + 8 * (8 + 16 * n)
    at = {"file id": 3, "com_0": 48 + 16, "com_0 end": st - 32 - 16, "seed": st - 7}
    r, n, j = st + 8, dim, 0
    while n > 1:
        if j in (0, 1, 5) or n == 2:
            at.update({f"l_vec {j}": r + 8 + 16, f"r_vec {j}": r + 8 + 2 * module(n) - 16,
                       f"l_poly {j}": r + 8 + 2 * module(n) + 16,
                       f"r_poly {j}": r + D.record_size(n, n // 2) - 16})
        r, n, j = r + D.record_size(n, n // 2), n // 2, j + 1
    at["opening"] = r
    return at


def test_changed_bytes_are_rejected(ctx, case):
    proof, dim = case
    for what, at in _offsets(dim).items():
        bad = bytearray(proof)
        bad[at] ^= 4
        bad = bytes(bad)
        assert _verify(ctx, bad) == _round_by_round(ctx, bad, dim) == D.EVERIFY, what


def test_words_above_q_are_reduced(ctx, case):
    """Deserialisation takes any 128-bit word mod q, and the transcript absorbs the
    reduced one."""
    proof, dim = case
    same = bytearray(proof)
    for what, at in _offsets(dim).items():
        if what in ("file id", "seed"):
            continue
        v = int.from_bytes(proof[at:at + 16], "little")
        assert v < Q
        same[at:at + 16] = (v + (3 + at % 1000) * Q).to_bytes(16, "little")
    assert _verify(ctx, bytes(same)) == _round_by_round(ctx, bytes(same), dim) == 0


def test_proofs_of_another_shape(ctx, case):
    proof, dim = case
    st, first = D.statement_size(dim), D.record_size(dim, dim // 2)
    count = bytearray(proof)
    count[st] -= 1
    renumbered = bytearray(proof)
    renumbered[st + 8] = 1
    assert _verify(ctx, bytes(renumbered)) == D.EVERIFY  # round mismatch
    assert _verify(ctx, bytes(count)) == D.EVERIFY       # the opening before every round
    assert _verify(ctx, proof[:st + 8 + first + 100]) == D.EDESERIALIZE
    assert _verify(ctx, proof[:-1]) == D.EDESERIALIZE
    length = bytearray(proof)
    length[st + 8 + 8] = 7  # a commitment of rank 7
    assert _verify(ctx, bytes(length)) == D.EDESERIALIZE


def test_without_room_for_the_transcript(ctx, case):
    proof, dim = case
    family = dim * 8 * dim * 16
    need = family + ((family // 2 + 16 + 255) & ~255)
    with D.Context(0, hbm_budget_bytes=need) as tight:
        assert tight.verify(proof, EPOCH) and tight.reserved == 0
    with D.Context(0, hbm_budget_bytes=need - 256) as small:
        assert _verify(small, proof) == D.ENOMEM_BUDGET and small.reserved == 0
