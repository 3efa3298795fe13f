"""The wire format's encoder on the device gives the host encoder's bytes: symbol types and alphabets on either side of a byte,
blocks that end off every boundary, tables from a few slots to 2^16, arrays around the length that is staged."""
import ctypes as C
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

from eoq_quantization_b200 import _lib as L
from eoq_quantization_b200.core import rans as R
from eoq_quantization_b200.core.rans_bitpacked import compress_tensor_rans
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


@pytest.mark.parametrize("n,short,long", [(1 << 16, 645, 646), (70001, 256, 70001)])
def test_few_long_blocks_are_the_hosts_and_give_the_same_bytes(n, short, long):
    torch.zeros(1, device="cuda")
    sym = np.minimum(np.abs(np.random.default_rng(n).standard_normal(n) * 3).astype(np.int64), 14)
    for block, on_device in ((short, True), (long, False)):
        staged, _ = R.stage_symbols(sym, 15, block_size=block)
        assert (staged is not None) == on_device
        data, want = BlockedRANSEncoder(block, 14).encode(sym, 15), O.encode_blocked(sym, 15, block, 14)
        assert data.compressed_blocks == bytes(want.compressed_blocks) and list(data.block_offsets) == list(want.block_offsets)


def test_scratch_is_bounded_and_given_back():
    torch.zeros(1, device="cuda")
    lib = L.lib()
    assert lib.eoq_b200_tune(b"release_scratch", 0) == 0
    before = torch.cuda.mem_get_info()[0]
    BlockedRANSEncoder().encode(np.zeros(1 << 23, np.uint8), 15)                        # some 50 MB
    kept = before - torch.cuda.mem_get_info()[0]
    assert 0 < kept <= 64 << 20
    big, at_first = np.zeros(80 << 20, np.uint8), BlockedRANSEncoder().encode(np.zeros(1 << 17, np.uint8), 15).compressed_blocks
    BlockedRANSEncoder().encode(big, 15)                                                # more than 256 MB of scratch: not kept
    assert before - torch.cuda.mem_get_info()[0] <= 256 << 20
    assert lib.eoq_b200_tune(b"release_scratch", 0) == 0
    assert before - torch.cuda.mem_get_info()[0] <= 4 << 20                             # (the side stream and its kernels stay)
    assert BlockedRANSEncoder().encode(np.zeros(1 << 17, np.uint8), 15).compressed_blocks == at_first


def test_two_threads_encode_at_once():
    torch.zeros(1, device="cuda")
    arrays = [np.random.default_rng(i).integers(0, 15, (1 << 18) + 1000 * i).astype(t) for i, t in enumerate((np.uint8, np.int64, np.int32))]
    want = [BlockedRANSEncoder().encode(a, 15).compressed_blocks for a in arrays]
    with ThreadPoolExecutor(3) as pool:
        for _ in range(8):
            assert list(pool.map(lambda a: BlockedRANSEncoder().encode(a, 15).compressed_blocks, arrays)) == want


def test_an_array_beside_another_ones_staged_symbols():
    torch.zeros(1, device="cuda")
    sym = np.random.default_rng(2).integers(0, 15, 1 << 17).astype(np.uint8)
    staged, counts = R.stage_symbols(sym, 15)
    freq = R.RANSEncoder(counts, 14).freq
    for other in (sym[:70000], np.concatenate([sym, sym])):
        assert R.encode_blocks(freq, 14, other, 256, staged) == R.encode_blocks(freq, 14, other, 256)
    assert R.encode_blocks(freq, 14, sym, 256, staged) == R.encode_blocks(freq, 14, sym, 256)


def test_threads_that_fetch_beside_a_recording():
    torch.zeros(1, device="cuda")
    sym = np.random.default_rng(1).integers(0, 15, 1 << 23).astype(np.int8)             # 4 MB of blocks: several threads
    want = BlockedRANSEncoder().encode(sym, 15).compressed_blocks
    for size in (1 << 23, (1 << 23) - 5):                                               # and once with scratch that is there already
        x, graph = torch.ones(8, device="cuda"), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = x + 1
            got = BlockedRANSEncoder().encode(sym[:size], 15).compressed_blocks
            y = y * 2
        graph.replay()
        assert (size < 1 << 23 or got == want) and y.tolist() == [4.0] * 8


@pytest.mark.parametrize("step", [1, 2, 3, 4, 5])
def test_what_the_device_refuses_the_host_encodes(step):
    torch.zeros(1, device="cuda")
    codes = torch.from_numpy(np.random.default_rng(step).integers(-7, 8, 1 << 17).astype(np.int8))
    sym = codes.numpy().astype(np.int64) + 7
    want, record = BlockedRANSEncoder().encode(sym, 15), compress_tensor_rans("w", codes, torch.ones(1024), 4, 128, (1 << 17,))
    try:
        assert L.lib().eoq_b200_tune(b"symbols_refused", step) == 0
        got, again = BlockedRANSEncoder().encode(sym, 15), compress_tensor_rans("w", codes, torch.ones(1024), 4, 128, (1 << 17,))
    finally:
        L.lib().eoq_b200_tune(b"symbols_refused", 0)
    assert got.compressed_blocks == want.compressed_blocks and list(got.block_offsets) == list(want.block_offsets)
    assert again.rans_bytes == record.rans_bytes and np.array_equal(got.freq_table, want.freq_table)


def test_more_than_two_to_the_27_blocks():
    torch.zeros(1, device="cuda")
    n = (1 << 27) + 77
    sym, lib = np.ones(n, np.uint8), L.lib()
    sym[:1000] = 0
    freq = np.array([100, 156], np.uint32)
    lib.eoq_b200_symbols_stage.restype, lib.eoq_b200_symbols_stage.argtypes = C.c_void_p, [C.c_void_p, C.c_int, C.c_size_t, C.c_int64, C.c_int, C.c_uint32]
    s = C.c_void_p(lib.eoq_b200_symbols_stage(sym.ctypes.data, R._ELEMENTS[sym.dtype], n, 0, 0, 2))
    assert s.value
    counts, size, want = np.zeros(2, np.uint64), C.c_size_t(), C.c_size_t()
    try:
        assert lib.eoq_b200_symbols_count(s, C.c_void_p(counts.ctypes.data)) == L.EOQ_OK and counts.tolist() == [1000, n - 1000]
        assert lib.eoq_b200_symbols_encode(s, C.c_void_p(freq.ctypes.data), 2, 8, 1, C.byref(size)) == L.EOQ_OK
        got, at = np.zeros(size.value, np.uint8), np.zeros(n, np.uint32)
        assert lib.eoq_b200_symbols_fetch(s, C.c_void_p(got.ctypes.data), C.c_void_p(at.ctypes.data)) == L.EOQ_OK
    finally:
        lib.eoq_b200_symbols_free(s)
    # every block is one symbol: a zero's bytes, then a one's for all the others
    h = C.c_void_p()
    assert lib.eoq_b200_wire_encode(sym[999:].ctypes.data, R._ELEMENTS[sym.dtype], 2, 0, 0, freq.ctypes.data, 2, 8, 1, C.byref(h), C.byref(want)) == L.EOQ_OK
    pair, offs = np.zeros(want.value, np.uint8), np.zeros(2, np.uint32)
    lib.eoq_b200_wire_take(h, pair.ctypes.data, offs.ctypes.data)
    zero, one = pair[:offs[1]], pair[offs[1]:]
    assert np.array_equal(at, np.where(np.arange(n) < 1000, np.arange(n) * len(zero), 1000 * len(zero) + (np.arange(n) - 1000) * len(one)))
    assert np.array_equal(got[:1000 * len(zero)].reshape(1000, -1), np.tile(zero, (1000, 1)))
    assert (got[1000 * len(zero):].reshape(-1, len(one)) == one).all()
