"""Single-stream rANS front end with the interface of the reference's
``core/rans.py``: table helpers on the host, encoding in the library (on the
device where long arrays are staged there, else on the host), decoding on the GPU."""
from __future__ import annotations

import ctypes as C

import numpy as np

from .. import _lib


#: integer types the library reads symbols in and writes them in, where they lie
_ELEMENTS = {np.dtype(np.int8): 0, np.dtype(np.uint8): 1, np.dtype(np.int16): 2, np.dtype(np.uint16): 3,
             np.dtype(np.int32): 4, np.dtype(np.uint32): 5, np.dtype(np.int64): 6}


def _native(result, where: str):
    """A result of the native front, or its error code raised."""
    if isinstance(result, int):
        _lib.check(result, where)
    return result


def readable(symbols: np.ndarray) -> bool:
    return symbols.dtype in _ELEMENTS and symbols.flags.c_contiguous and symbols.dtype.isnative


def count_symbols(symbols: np.ndarray, alphabet_size: int, shift: int = 0, clamp: bool = False):
    """(int64 counts, least, greatest) of value + shift over an array of one of the types above."""
    counts, lo, hi = _native(_lib.native().count_symbols(symbols, _ELEMENTS[symbols.dtype], shift, int(clamp), alphabet_size), "count_symbols")
    return np.array(counts, dtype=np.int64), lo, hi


def stage_symbols(symbols: np.ndarray, alphabet_size: int, shift: int = 0, clamp: bool = False, block_size: int = 0):
    """(staged, int64 counts): the array on the device, counted there, to be handed to `encode_blocks` or `encode_container`
    beside it; or (None, None) where the host counts and encodes (short arrays, few long blocks where `block_size` is given, no
    device in use, symbols outside the alphabet)."""
    if not readable(symbols) or not 0 < alphabet_size <= 4096:
        return None, None
    got = _lib.native().stage_symbols(symbols, _ELEMENTS[symbols.dtype], shift, int(clamp), alphabet_size, block_size)
    return (None, None) if got is None else (got[0], np.array(got[1], dtype=np.int64))


def compute_frequency_table(symbols: np.ndarray, alphabet_size: int) -> np.ndarray:
    """Histogram of symbol values (core/rans.py:32-55); ValueError if out of range."""
    symbols = np.asarray(symbols).ravel()
    if symbols.size == 0:
        return np.zeros(alphabet_size, dtype=np.int64)
    if readable(symbols) and 0 < alphabet_size <= 1 << 20:
        counts, lo, hi = count_symbols(symbols, alphabet_size)
    else:
        counts, lo, hi = None, symbols.min(), symbols.max()
    if lo < 0 or hi >= alphabet_size:
        raise ValueError(f"Symbols must be in [0, {alphabet_size}), got range [{lo}, {hi}]")
    return np.bincount(symbols, minlength=alphabet_size).astype(np.int64)[:alphabet_size] if counts is None else counts


def estimate_compressed_size(freq_table: np.ndarray, num_symbols: int) -> int:
    """ceil(H * n / 8) with H the Shannon entropy of the table (core/rans.py:58-78)."""
    f = np.asarray(freq_table, dtype=np.float64)
    tot = f.sum()
    if tot == 0 or num_symbols == 0:
        return 0
    pr = f[f > 0] / tot
    return int(np.ceil(-float(np.sum(pr * np.log2(pr))) * num_symbols / 8))


def _normalize_frequencies(raw_freq: np.ndarray, precision_bits: int):
    """(freq, cdf) summing to ``2**precision_bits``, every symbol >= 1.

    Same arithmetic as core/rans.py:85-153 -- float64 proportional scaling,
    truncation, then the residual dealt out round-robin over the symbols in
    descending order of scaled frequency.  The order comes from
    ``np.argsort(-scaled)`` exactly as in the reference, so a table built here
    agrees with one built by the reference on the same machine even where ties
    make that order implementation-defined (alphabets above 16 symbols).
    """
    M = 1 << precision_bits
    raw = np.asarray(raw_freq, dtype=np.int64).copy()
    a = len(raw)
    if a == 0:
        raise ValueError("Frequency table must not be empty")
    if a > M:
        raise ValueError(f"Alphabet size ({a}) exceeds probability space (2**{precision_bits} = {M}).  "
                         "Use a larger precision_bits.")
    raw = np.maximum(raw, 1)
    scaled = np.maximum((raw.astype(np.float64) / raw.sum() * M).astype(np.int64), 1)
    residual = int(M - scaled.sum())
    if residual > 0:                        # nobody is passed over: whole rounds, then one more for the first ones
        order = np.argsort(-scaled)
        scaled += residual // a
        scaled[order[:residual % a]] += 1
    elif residual:
        order = np.argsort(-scaled)
        at = 0
        while residual:
            if scaled[order[at]] > 1:
                scaled[order[at]] -= 1
                residual += 1
            at = (at + 1) % a
    cdf = np.zeros(a + 1, dtype=np.int64)
    np.cumsum(scaled, out=cdf[1:])
    return scaled, cdf


def _check_precision(p: int) -> None:
    if p < 8 or p > 20:
        raise ValueError(f"precision_bits must be in [8, 20], got {p}")


def encode_blocks(freq_norm: np.ndarray, precision_bits: int, symbols: np.ndarray, block_size: int, staged=None):
    """Encoder of the library (on the device for `staged` symbols) -> (bytes, offsets), wire format of core/rans.py:210-276."""
    sym = np.asarray(symbols).ravel()
    if sym.size == 0:
        return b"", []
    f = np.ascontiguousarray(freq_norm, dtype=np.uint32)
    if precision_bits <= 16 and readable(sym):
        return _native(_lib.native().encode_symbols(sym, _ELEMENTS[sym.dtype], 0, 0, f, precision_bits, block_size, None, None, staged),
                       "eoq_b200_wire_encode")
    sym = np.ascontiguousarray(sym.astype(np.uint32))
    nb = (sym.size + block_size - 1) // block_size
    cap = C.c_size_t(3 * sym.size + 16 * nb + 64)
    out = np.empty(cap.value, np.uint8)
    offs = np.empty(nb, np.uint32)
    _lib.check(_lib.lib().eoq_b200_encode_blocked(f.ctypes.data, f.size, precision_bits, sym.ctypes.data, sym.size,
                                                  block_size, out.ctypes.data, C.byref(cap), offs.ctypes.data),
               "eoq_b200_encode_blocked")
    return out[:cap.value].tobytes(), offs.astype(np.int64).tolist()


def encode_container(symbols: np.ndarray, shift: int, freq_norm: np.ndarray, precision_bits: int, block_size: int, head: bytes,
                     counts: np.ndarray, staged=None) -> bytes:
    """A whole `RANS` container (core/rans_blocked.py:176-214) of value + shift, clipped to the alphabet: `head` up to the
    data size, the counts, the offsets and the blocks."""
    table = np.asarray(counts).astype("<u4")
    if symbols.size == 0:
        return head + b"\0\0\0\0" + table.tobytes()
    return _native(_lib.native().encode_symbols(symbols, _ELEMENTS[symbols.dtype], shift, 1, np.ascontiguousarray(freq_norm, dtype=np.uint32),
                                                precision_bits, block_size, head, table, staged), "eoq_b200_wire_encode")


def decode_blocks(freq_norm: np.ndarray, precision_bits: int, data: bytes, offsets, block_size: int, n: int,
                  dtype=np.int64, shift: int = 0) -> np.ndarray:
    """GPU decode of wire-format blocks -> symbols + shift (core/rans.py:368-419 per block), int64 unless asked otherwise."""
    if n == 0 or len(data) == 0:
        return np.empty(0, dtype=dtype)
    if precision_bits > 16:
        raise NotImplementedError("the GPU decoder keeps a 32-bit state: precision_bits must be <= 16")
    f = np.ascontiguousarray(freq_norm, dtype=np.uint32)
    if f.size > 65536:
        raise NotImplementedError("alphabets above 65536 symbols are not supported")
    out = np.empty(n, dtype)
    offs = offsets if type(offsets) is list else np.ascontiguousarray(np.asarray(offsets, dtype=np.uint32))
    _native(_lib.native().decode_symbols(f, precision_bits, data, offs, block_size, out, _ELEMENTS[out.dtype], shift), "eoq_b200_decode_blocked")
    return out


class RANSEncoder:
    """core/rans.py:160-314."""

    def __init__(self, freq_table: np.ndarray, precision_bits: int = 16) -> None:
        _check_precision(precision_bits)
        self.precision_bits = precision_bits
        self.M = 1 << precision_bits
        freq_table = np.asarray(freq_table, dtype=np.int64)
        self.alphabet_size = len(freq_table)
        self.freq, self.cdf = _normalize_frequencies(freq_table, precision_bits)

    def encode(self, symbols: np.ndarray) -> bytes:
        symbols = np.asarray(symbols).ravel()
        if symbols.size == 0:
            return b""
        data, _ = encode_blocks(self.freq, self.precision_bits, symbols, max(int(symbols.size), 1))
        return data

    def encode_blocked(self, symbols: np.ndarray, block_size: int = 256):
        symbols = np.asarray(symbols).ravel()
        return encode_blocks(self.freq, self.precision_bits, symbols, block_size)


class RANSDecoder:
    """core/rans.py:321-439."""

    def __init__(self, freq_table: np.ndarray, precision_bits: int = 16) -> None:
        _check_precision(precision_bits)
        self.precision_bits = precision_bits
        self.M = 1 << precision_bits
        freq_table = np.asarray(freq_table, dtype=np.int64)
        self.alphabet_size = len(freq_table)
        self.freq, self.cdf = _normalize_frequencies(freq_table, precision_bits)

    def decode(self, data: bytes, num_symbols: int) -> np.ndarray:
        if num_symbols == 0 or len(data) == 0:
            return np.empty(0, dtype=np.int64)
        return decode_blocks(self.freq, self.precision_bits, bytes(data), [0], max(num_symbols, 1), num_symbols)

    def decode_block(self, data: bytes, offset: int, block_size: int) -> np.ndarray:
        return self.decode(data[offset:], block_size)
