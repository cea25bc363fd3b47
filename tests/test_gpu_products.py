"""Ring products in one kernel (rings up to 2^10) against the oracle and against the
general path, which an output overlapping a factor takes: every ring size, counts
around a block's products, elements below 2^112 (q and above among them), the product in place of a factor, and the
budget the general path's scratch asks for."""
import random

import pytest
import torch

import damascus000_gb300 as D

pytestmark = pytest.mark.gpu
Q = (1 << 112) - 75


def _words(count, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randint(-(1 << 63), (1 << 63) - 1, (count, n, 2), dtype=torch.int64, device="cuda", generator=g)
    w[..., 1] &= (1 << 48) - 1
    w[0, 0] = torch.tensor([-1, (1 << 48) - 1])  # 2^112 - 1 = q + 74
    return w


def _ints(t):
    b = t.cpu().numpy().tobytes()
    return [int.from_bytes(b[i:i + 16], "little") for i in range(0, len(b), 16)]


def _mul(ctx, a, b, out, n, count):
    ctx.ring_mul_batch_device(a.data_ptr(), b.data_ptr(), out.data_ptr(), n, count)


@pytest.mark.parametrize("L", range(0, 11))
def test_products_match_oracle(ctx, oracle_lib, L):
    n, per = 1 << L, 32 if L < 5 else max(1, 512 >> L)
    # the last: more blocks than SMs, where a block takes one factor after the other
    for count in sorted({1, per, per + 1, 3 * per - 1, 200 * per + 1}):
        a, b = _words(count, n, 7 * L + count), _words(count, n, 7 * L + count + 1)
        out = torch.empty_like(a)
        _mul(ctx, a, b, out, n, count)
        x, y, z = _ints(a), _ints(b), _ints(out)
        for i in sorted({0, count // 2, count - 1}):
            at = slice(i * n, (i + 1) * n)
            assert z[at] == oracle_lib.negacyclic_multiply([v % Q for v in x[at]], [v % Q for v in y[at]]), (n, count, i)


@pytest.mark.parametrize("n", [2, 16, 256, 1024])
def test_in_place_and_overlapping(ctx, n):
    count = 67
    a, b = _words(count, n, n), _words(count, n, n + 1)
    want = torch.empty_like(a)
    _mul(ctx, a, b, want, n, count)
    for which in (0, 1):
        f = [a.clone(), b.clone()]
        _mul(ctx, f[0], f[1], f[which], n, count)
        assert torch.equal(f[which], want)
    both = torch.empty(count + 1, n, 2, dtype=torch.int64, device="cuda")
    both[1:] = a
    _mul(ctx, both[1:], b, both, n, count)  # one polynomial below the first factor
    assert torch.equal(both[:count], want)
    both[:count] = b
    _mul(ctx, a, both, both[1:], n, count)
    assert torch.equal(both[1:], want)


def test_budget_as_for_the_general_path():
    n, count = 512, 100
    a, b = _words(count, n, 3), _words(count, n, 4)
    out = torch.empty_like(a)
    scratch = 2 * count * 9 * n * 4
    with D.Context(0, hbm_budget_bytes=scratch - 1) as c:
        with pytest.raises(D.DamascusError) as e:
            _mul(c, a, b, out, n, count)
        assert e.value.code == D.ENOMEM_BUDGET and c.reserved == 0
    with D.Context(0, hbm_budget_bytes=scratch) as c:
        _mul(c, a, b, out, n, count)
        assert c.reserved == 0
