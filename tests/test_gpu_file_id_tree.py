"""The file id's tree at its block edges: groups of 128 chunks merged in a block,
the levels above in one block (through memory beyond 1024 groups), ragged last
chunks and groups, and device buffers at any byte alignment.  Bit-exact with the
oracle."""
import ctypes

import pytest

import damascus000_gb300 as D
from damascus000_gb300 import synth

pytestmark = pytest.mark.gpu
GROUP = 128 << 10  # bytes of one block's chunks
SIZES = [GROUP - 1, GROUP, GROUP + 1, GROUP + 1025, 2 * GROUP, 3 * GROUP - 1023, 5 * GROUP + 63, 127 * GROUP + 3,
         (129 << 20) + 7]


@pytest.mark.parametrize("n", SIZES)
def test_file_id_at_group_edges(ctx, oracle_lib, n):
    data, _ = synth.random_file(91, n, n % 1000)
    assert ctx.file_id(data) == oracle_lib.blake3(data)


@pytest.mark.parametrize("n", [1, 700, 1024 + 65, GROUP + 1025])
@pytest.mark.parametrize("offset", [0, 1, 4, 8])
def test_file_id_of_unaligned_device_buffers(ctx, oracle_lib, n, offset):
    torch = pytest.importorskip("torch")
    data, _ = synth.random_file(92, n, n % 1000)
    dev = torch.frombuffer(bytearray(bytes(offset) + data), dtype=torch.uint8).cuda()
    out = torch.zeros(32, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream()
    assert D.load().damascus_file_id_noalloc(ctypes.c_void_p(dev.data_ptr() + offset), n,
                                             ctypes.c_void_p(out.data_ptr()),
                                             ctypes.c_void_p(stream.cuda_stream)) == D.OK
    stream.synchronize()
    assert bytes(out.cpu().tolist()) == oracle_lib.blake3(data)
