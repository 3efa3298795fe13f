"""Blocks of a wire-format stream that are not well-formed, found on the device, give the codes that the checks on the host give;
symbols in device memory of any alignment give the same tiles."""
import ctypes as C

import numpy as np
import pytest
import torch

from eoq_quantization_b200 import _lib as L
from eoq_quantization_b200.core.rans import _normalize_frequencies
from eoq_quantization_b200.core.rans_blocked import BlockedRANSEncoder, serialize_blocked_rans
from eoq_quantization_b200.fused import EOQWeight

pytestmark = pytest.mark.gpu
N, K = 96, 512


def _stream(block=256):
    sym = np.random.default_rng(3).integers(0, 15, N * K)
    data = BlockedRANSEncoder(block, 14).encode(sym, 15)
    return sym, data


@pytest.mark.parametrize("what", ["fine", "order", "past the end", "last past the end", "state longer than the block", "wide state", "both"])
@pytest.mark.parametrize("at", [0, 7, -1])
@pytest.mark.parametrize("block", [256, 12, 8])                # 192 and 4096 blocks (checked on the host), 6144
def test_corrupt_blocks_give_the_hosts_codes(what, at, block):
    sym, data = _stream(block)
    offs, raw = np.array(data.block_offsets, np.uint32), bytearray(data.compressed_blocks)
    nb = len(offs)
    at = nb - 1 if at < 0 else at
    if what == "order":
        offs[at] = offs[min(at + 1, nb - 1)] + (5 if at + 1 < nb else len(raw))
    elif what == "past the end":
        offs[at] = 0xFFFFFFF0
    elif what == "last past the end":
        offs[-1] = len(raw) + 1
    elif what == "state longer than the block":
        raw[offs[at]] = 255
    elif what in ("wide state", "both"):
        raw[offs[at]] = 5
        if what == "both":                                    # the earlier block decides
            raw[offs[nb // 2]] = 255
    lib, freq = L.lib(), np.ascontiguousarray(_normalize_frequencies(data.freq_table, 14)[0], dtype=np.uint32)
    buf, out = np.frombuffer(bytes(raw), np.uint8), np.zeros(N * K, np.uint8)
    want = lib.eoq_b200_decode_blocked(freq.ctypes.data, 15, 14, buf.ctypes.data, buf.size, offs.ctypes.data, nb, block, N * K, out.ctypes.data, 1, 0, None)
    assert (want == L.EOQ_OK) == (what == "fine")
    got = L.native().decode_symbols(freq, 14, bytes(raw), offs, block, np.zeros(N * K, np.int64), 6, 0)
    assert (0 if got is None else got) == want
    # the container, at an address off every boundary
    data.compressed_blocks, data.block_offsets = bytes(raw), offs.tolist()
    whole = np.frombuffer(b"x" + serialize_blocked_rans(data), np.uint8)[1:]
    opts, keep = EOQWeight._opts(L.KIND_INT4_ABSMAX, N, K, 128, 0, 0, 0, None)
    scales, h = np.ones(N * K // 128, np.float16), C.c_void_p()
    rc = lib.eoq_b200_weight_from_rans(whole.ctypes.data, whole.size, scales.ctypes.data, C.byref(opts), C.byref(h))
    assert rc == want
    if rc == L.EOQ_OK:
        assert np.array_equal(EOQWeight(h.value, L.KIND_INT4_ABSMAX).decode_symbols().cpu().numpy().ravel(), sym)


@pytest.mark.parametrize("pinned_refused", [0, 1])
@pytest.mark.parametrize("what", ["order", "state longer than the block", "wide state"])
@pytest.mark.parametrize("block", [12, 8])                     # 4096 blocks (checked on the host), 6144
def test_a_refused_stream_leaves_the_result_alone(block, what, pinned_refused):
    sym, data = _stream(block)
    offs, raw = np.array(data.block_offsets, np.uint32), bytearray(data.compressed_blocks)
    if what == "order":
        offs[-2] = offs[-1] + 1
    else:
        raw[offs[-1]] = 255 if what == "state longer than the block" else 5
    freq = np.ascontiguousarray(_normalize_frequencies(data.freq_table, 14)[0], dtype=np.uint32)
    try:
        L.lib().eoq_b200_tune(b"pinned_refused", pinned_refused)
        for dtype, code in ((np.int8, 0), (np.int64, 6)):
            out = np.full(N * K, 77, dtype)
            got = L.native().decode_symbols(freq, 14, bytes(raw), offs, block, out, code, 0)
            assert got == (L.EOQ_ERR_UNSUPPORTED if what == "wide state" else L.EOQ_ERR_CORRUPT_STREAM) and (out == 77).all()
            assert L.native().decode_symbols(freq, 14, data.compressed_blocks, np.array(data.block_offsets, np.uint32), block, out, code, 0) is None
            assert np.array_equal(out, sym)
    finally:
        L.lib().eoq_b200_tune(b"pinned_refused", 0)


@pytest.mark.parametrize("offset", [0, 4, 8, 5])
def test_tiles_from_symbols_of_any_alignment(offset):
    sym, _ = _stream()
    held = torch.zeros(N * K + 16, dtype=torch.uint8, device="cuda")
    held[offset:offset + N * K] = torch.from_numpy(sym.astype(np.uint8)).cuda()
    w = EOQWeight.from_device_symbols(held[offset:offset + N * K].view(N, K), np.ones(N * K // 128, np.float16))
    assert np.array_equal(w.decode_symbols().cpu().numpy().ravel(), sym)
