"""Which of two ways a call goes, where both were measured on either side of the line: the rules of the library, asked without a device."""
import ctypes as C

import pytest

from eoq_quantization_b200 import _lib as L


def _rule(name, n):
    fn = getattr(L.lib(), name)
    fn.restype, fn.argtypes = C.c_int, [C.c_uint32] * n
    return fn


@pytest.mark.parametrize("bits,group,n,k,warp_level", [
    # bytes: few rows of many columns are the product kernel's
    (8, 64, 512, 4096, 1), (8, 32, 512, 5120, 0), (8, 32, 1024, 4096, 1), (8, 64, 2048, 3072, 1), (8, 64, 2048, 4096, 0), (8, 64, 2048, 8192, 0),
    (8, 64, 3072, 4096, 1), (8, 32, 3072, 5120, 0), (8, 64, 4096, 4096, 1), (8, 64, 4096, 8192, 0), (8, 32, 5120, 8192, 1), (8, 64, 14336, 8192, 1),
    # packed: fewer rows of more columns
    (4, 64, 1024, 6144, 1), (4, 64, 1024, 8192, 0), (4, 32, 1536, 11008, 0), (4, 64, 2048, 11008, 1), (4, 64, 2048, 28672, 0), (4, 32, 3072, 28672, 1),
    (2, 64, 1024, 11008, 1), (2, 64, 1024, 14336, 0), (2, 64, 2048, 14336, 1), (2, 64, 2048, 28672, 0), (2, 64, 4096, 28672, 1),
    # whole spans: always; what the warp-level kernel does not take: never
    (8, 128, 512, 28672, 1), (4, 256, 256, 28672, 1), (8, 64, 11008, 8320, 0), (2, 32, 4096, 4096, 0), (4, 48, 4096, 4608, 0), (4, 64, 4096, 4160, 0)])
def test_a_few_rows_of_16_bit_activations(bits, group, n, k, warp_level):
    assert _rule("eoq_b200_gemv_packed_preferred", 4)(n, k, bits, group) == warp_level


@pytest.mark.parametrize("n,k,rows,rotated", [
    (8192, 4096, 32, 0), (8192, 4096, 33, 1), (8193, 4096, 64, 0), (8193, 4096, 65, 1), (28672, 8192, 112, 1), (12288, 4096, 113, 0), (12288, 4096, 128, 0),
    (12288, 4096, 129, 1), (11008, 8192, 128, 1), (14336, 2048, 128, 1), (28672, 8192, 144, 0), (28672, 8192, 145, 1), (20480, 8192, 144, 1), (28672, 11008, 144, 1)])
def test_polar_rows_that_rotate_the_weight(n, k, rows, rotated):
    assert _rule("eoq_b200_polar_rotates", 3)(n, k, rows) == rotated


@pytest.mark.parametrize("n,block,on_device", [
    (65535, 256, 0), (1 << 16, 1, 1), (1 << 16, 256, 1), (1 << 16, 645, 1), (1 << 16, 646, 0), (1 << 16, 1 << 16, 0), (1 << 18, 1024, 1), (1 << 18, 4096, 0),
    (1 << 20, 4096, 1), (1 << 20, 16384, 0), (1 << 20, 1 << 40, 0), (1 << 24, 16384, 1), (1 << 24, 65536, 0), (1 << 24, 1 << 24, 0)])
def test_blocks_that_are_encoded_on_the_device(n, block, on_device):
    fn = L.lib().eoq_b200_symbols_preferred
    fn.restype, fn.argtypes = C.c_int, [C.c_size_t, C.c_uint64]
    assert fn(n, block) == on_device
