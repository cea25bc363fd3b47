"""Ring products in place of a factor where the one kernel has more blocks than SMs, so
that a block takes one factor after the other (rings of 2^4 to 2^9), and in the small
rings' kernel."""
import pytest
import torch

import damascus000_gb300 as D
from damascus000_gb300.autotune import NTT_RADIX
from test_gpu_products import _mul, _words

pytestmark = pytest.mark.gpu


# blocks of 32, 8 and 1 products; at 2^9 the rule's last count, and the first of the general path
@pytest.mark.parametrize("n,count", [(8, 6001), (64, 2001), (512, 153), (512, 8 * 152), (512, 8 * 152 + 1)])
def test_in_place_with_many_blocks(ctx, n, count):
    a, b = _words(count, n, n + count), _words(count, n, n + count + 1)
    want = torch.empty_like(a)
    _mul(ctx, a, b, want, n, count)
    with D.Context(0) as c:  # the general path: radix-32 passes take no other
        if n >= 32:
            c.tuning_set(NTT_RADIX, n.bit_length() - 1, 32)
            general = torch.empty_like(a)
            _mul(c, a, b, general, n, count)
            assert torch.equal(general, want)
    for which in (0, 1):
        f = [a.clone(), b.clone()]
        _mul(ctx, f[0], f[1], f[which], n, count)
        assert torch.equal(f[which], want)
    square = a.clone()
    _mul(ctx, a, a, want, n, count)
    _mul(ctx, square, square, square, n, count)
    assert torch.equal(square, want)
