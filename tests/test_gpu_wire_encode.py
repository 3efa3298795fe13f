"""The wire format's encoder on the device gives the host encoder's bytes: symbol types and alphabets on either side of a byte,
blocks that end off every boundary, tables from a few slots to 2^16, arrays around the length that is staged."""
import numpy as np
import pytest
import torch

from eoq_quantization_b200.core import rans as R
from eoq_quantization_b200.core.rans_blocked import BlockedRANSDecoder, BlockedRANSEncoder
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,block,p,alphabet,dtype", [
    (1 << 16, 256, 14, 15, np.int64), ((1 << 16) + 1, 256, 16, 3, np.int8), (70001, 250, 12, 15, np.uint8), (70001, 1, 8, 2, np.int32),
    (131073, 4096, 12, 256, np.int64), (100003, 1 << 20, 14, 255, np.int16), (99999, 77, 16, 257, np.uint16), (200000, 264, 14, 4096, np.uint32),
    (1 << 20, 256, 14, 15, np.int8)])
def test_device_encoder_gives_the_host_encoders_bytes(n, block, p, alphabet, dtype):
    torch.zeros(1, device="cuda")
    rng = np.random.default_rng(n + p)
    sym = np.minimum((np.abs(rng.standard_normal(n)) * alphabet / 5).astype(np.int64), alphabet - 1)
    if alphabet == 3:
        sym[:] = 1                                            # one symbol that takes nearly all slots
    if dtype == np.int8:
        sym = np.minimum(sym, 127)
    sym = sym.astype(dtype)
    staged, counts = R.stage_symbols(sym, alphabet)
    assert staged is not None and np.array_equal(counts, np.bincount(sym.astype(np.int64), minlength=alphabet))
    freq = R.RANSEncoder(counts, p).freq
    want, offsets = R.encode_blocks(freq, p, sym, block)
    got, at = R.encode_blocks(freq, p, sym, block, staged)
    assert got == want and at == offsets
    if alphabet == 15:
        # and through the entry point, against the oracle and back
        data = BlockedRANSEncoder(block, p).encode(sym, alphabet)
        blocked = O.encode_blocked(sym.astype(np.int64), alphabet, block, p)
        assert data.compressed_blocks == bytes(blocked.compressed_blocks) and np.array_equal(BlockedRANSDecoder().decode_all(data), sym)


def test_what_is_not_staged_and_calls_beside_a_recording():
    torch.zeros(1, device="cuda")
    sym = np.zeros(1 << 17, np.int64)
    assert R.stage_symbols(sym[:1000], 15)[0] is None and R.stage_symbols(sym, 5000)[0] is None and R.stage_symbols(sym[::2], 15)[0] is None
    sym[12345] = 15
    assert R.stage_symbols(sym, 15)[0] is None and R.stage_symbols(sym, 15, 0, True)[0] is not None
    with pytest.raises(ValueError, match="got range"):
        BlockedRANSEncoder().encode(sym, 15)
    # bytes go up as they are and are looked at there
    low = np.zeros(70001, np.int8)
    low[70000], low[3] = 20, -9
    assert R.stage_symbols(low, 15)[0] is None
    assert R.stage_symbols(low, 15, 7, True)[1].tolist() == R.count_symbols(low, 15, 7, True)[0].tolist()
    sym = np.random.default_rng(0).integers(0, 15, 1 << 17)
    want = BlockedRANSEncoder().encode(sym, 15).compressed_blocks
    x, graph = torch.ones(8, device="cuda"), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = x + 1
        got = BlockedRANSEncoder().encode(sym, 15).compressed_blocks
        y = y * 2
    graph.replay()
    assert got == want and y.tolist() == [4.0] * 8
