"""The wire codec on symbols of every integer type, read and written where they lie: the encoder (four blocks side by side,
divisions by reciprocal) byte for byte against the oracle's at the edges of its ranges, the decoder's typed host output."""
import numpy as np
import pytest
import torch

from eoq_quantization_b200.core import rans as R
from eoq_quantization_b200.core import rans_blocked as RB
from eoq_quantization_b200.core.rans_bitpacked import compress_tensor_rans, decompress_tensor_rans
from oracle import oracle as O


@pytest.mark.parametrize("p,a", [(8, 3), (12, 15), (14, 255), (16, 1), (16, 255), (16, 4000)])
@pytest.mark.parametrize("n,bs", [(1, 7), (255, 64), (256, 64), (70001, 256), (300000, 4096)])
def test_encoder_is_byte_exact_for_every_type(p, a, n, bs):
    rng = np.random.default_rng(n + a)
    sym = np.minimum(rng.geometric(min(0.9, 4.0 / a), n) - 1, a - 1).astype(np.int64)
    # on a table that sums to 2^p every normaliser is the identity, whatever its tie order
    table = O.Table(R._normalize_frequencies(np.bincount(sym, minlength=a), p)[0], p)
    want = [table.encode(sym[i:i + bs]) for i in range(0, n, bs)]
    starts = np.cumsum([0] + [len(b) for b in want])[:-1].tolist()
    for dt in (np.int8, np.uint8, np.int16, np.uint16, np.int32, np.uint32, np.int64):
        if a - 1 > np.iinfo(dt).max:
            continue
        got = RB.BlockedRANSEncoder(block_size=bs, precision_bits=p).encode(sym.astype(dt), a)
        assert got.compressed_blocks == b"".join(want) and got.block_offsets == starts, dt
    with pytest.raises(ValueError):
        RB.BlockedRANSEncoder(block_size=bs, precision_bits=p).encode(np.append(sym, a), a)
    with pytest.raises(R._lib.EOQError):                      # a symbol outside the table
        R.encode_blocks(R._normalize_frequencies(np.ones(a), p)[0], p, np.append(sym, a), bs)


def test_compressed_tensor_clips_like_the_reference():
    codes = torch.from_numpy(np.random.default_rng(0).integers(-9, 10, 5000).astype(np.int32))
    ct = compress_tensor_rans("t", codes, torch.ones(40), 4, 128, (5000,))
    want = O.encode_blocked(np.clip(codes.numpy().astype(np.int64) + 7, 0, 14), 15, 256, 14)
    assert ct.rans_bytes == O.serialize_rans_v1(want)
    empty = compress_tensor_rans("e", codes[:0], torch.ones(0), 4, 128, (0,))
    assert RB.deserialize_blocked_rans(empty.rans_bytes).num_symbols == 0 and decompress_tensor_rans(empty)[0].numel() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("a,p", [(15, 12), (255, 14), (3000, 16)])
@pytest.mark.parametrize("n", [1, 262143, 262145, 3000001])
def test_decoded_symbols_in_every_type(a, p, n):
    rng = np.random.default_rng(n + a)
    sym = rng.integers(0, a, n)
    d = RB.BlockedRANSEncoder(block_size=1024, precision_bits=p).encode(sym, a)
    freq = R._normalize_frequencies(d.freq_table, p)[0]
    for dt, shift in ((np.int64, 0), (np.int64, -a), (np.int8, -7), (np.uint8, 0), (np.int16, -3), (np.uint16, 5), (np.int32, -a)):
        got = R.decode_blocks(freq, p, d.compressed_blocks, d.block_offsets, 1024, n, dt, shift)
        assert got.dtype == dt and np.array_equal(got, (sym + shift).astype(dt)), (dt, shift)


@pytest.mark.gpu
def test_codec_without_page_locked_memory():
    """Where the system has no page-locked memory to give, streams and symbols are copied without it, to the same results,
    and the refusal does not come back as the error of a launch."""
    rng = np.random.default_rng(5)
    n = 3000001                                               # a stream that several threads would stage (from 2 MB on)
    sym = rng.integers(0, 255, n)
    d = RB.BlockedRANSEncoder(block_size=1024, precision_bits=14).encode(sym, 255)
    assert len(d.compressed_blocks) > 2 << 20
    freq = R._normalize_frequencies(d.freq_table, 14)[0]
    lib = R._lib.lib()
    assert lib.eoq_b200_tune(b"pinned_refused", 1) == 0
    try:
        for dt, shift in ((np.int64, 0), (np.int8, -127)):
            got = R.decode_blocks(freq, 14, d.compressed_blocks, d.block_offsets, 1024, n, dt, shift)
            assert np.array_equal(got, (sym + shift).astype(dt)), dt
    finally:
        lib.eoq_b200_tune(b"pinned_refused", 0)
