"""Polar weights in blocks of 64 against many 16-bit rows, where the kernel rotates the weight: around the rows and weight sizes
where that begins, an odd number of blocks, a token tile's edges, every magnitude of a row that its type holds."""
import pytest
import torch

from eoq_quantization_b200 import _lib as L
from eoq_quantization_b200.core.polar_quant import hadamard_matrix
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,rows", [(1, 64, (33, 513)), (129, 704, (32, 33, 64, 65, 256, 257)), (8192, 128, (33, 64)), (8193, 192, (64, 65, 144))])
@pytest.mark.parametrize("bits", [1, 5, 8])
def test_rotated_weight(bits, n, k, rows):
    g = torch.Generator(device="cuda").manual_seed(bits + n)
    codes = torch.randint(0, 1 << bits, (n, k), generator=g, device="cuda").to(torch.uint8)
    norms = (torch.rand(n * k // 64, generator=g, device="cuda") * 2 + 0.1).half()
    norms[3:: 7] = 0
    cent = torch.sort(torch.randn(1 << bits, generator=g, device="cuda"))[0]
    bias = torch.randn(n, generator=g, device="cuda").half()
    dense = ((cent.double()[codes.long()].view(-1, 64) / 8) @ hadamard_matrix(64).cuda().double() * norms.double()[:, None]).view(n, k)
    for m in rows:
        for dt, code, sizes in ((torch.float16, L.F16, (1.0, 1e-3, 1e3)), (torch.bfloat16, L.BF16, (1.0, 1e-30, 1e30))):
            x = torch.randn(m, k, generator=g, device="cuda").to(dt)
            for i, size in enumerate(sizes):
                x[i::3] *= size
            x[5] = 0
            y, scratch = torch.empty(m, n, device="cuda"), torch.empty(m * (k + 1), device="cuda")
            assert L.lib().eoq_b200_linear_polar_codes(codes.data_ptr(), norms.data_ptr(), cent.data_ptr(), n, k, bits, 64, x.data_ptr(), code, m, scratch.data_ptr(),
                                                       y.data_ptr(), L.F32, bias.data_ptr(), L.F16, torch.cuda.current_stream().cuda_stream) == L.EOQ_OK
            want = x.double() @ dense.T + bias.double()
            # fp32 sums of K products (2e-6 where the tests of the other forms have it), to each row's own magnitude; one output
            # alone may be a difference of large ones: to the sum of its products' magnitudes, which its error is a part of 2^-22 of
            size = want.norm(dim=1) if n > 1 else (x.double().abs() @ dense.abs().T + bias.double().abs()).norm(dim=1)
            err = (y.double() - want).norm(dim=1) / size
            assert err.max().item() < 2e-6, (m, dt)
    assert L.lib().eoq_b200_linear_status() == 0


def _product(codes, norms, cent, n, k, x, code, m):
    y, scratch = torch.empty(m, n, device="cuda"), torch.empty(m * (k + 1), device="cuda")
    assert L.lib().eoq_b200_linear_polar_codes(codes.data_ptr(), norms.data_ptr(), cent.data_ptr(), n, k, 5, 64, x.data_ptr(), code, m, scratch.data_ptr(),
                                               y.data_ptr(), L.F32, None, L.F16, torch.cuda.current_stream().cuda_stream) == L.EOQ_OK
    return y


@pytest.mark.parametrize("dt,code", [(torch.float16, L.F16), (torch.bfloat16, L.BF16)])
@pytest.mark.parametrize("m", [33, 130])
def test_rows_that_are_not_finite_or_not_aligned(m, dt, code):
    n, k = 200, 192
    g = torch.Generator(device="cuda").manual_seed(m)
    codes = torch.randint(0, 32, (n, k), generator=g, device="cuda").to(torch.uint8)
    norms, cent = (torch.rand(n * k // 64, generator=g, device="cuda") + 0.1).half(), torch.sort(torch.randn(32, generator=g, device="cuda"))[0]
    held = torch.randn(m * k + 8, generator=g, device="cuda").to(dt)
    x = held[:m * k].view(m, k)
    want = _product(codes, norms, cent, n, k, x, code, m)
    # an infinity or a NaN leaves its own row without a finite result (the weight goes in as two halves of either sign) and the others as they were
    bad = x.clone()
    bad[3, 5], bad[17, 64], bad[32, 191], bad[m - 1, 0] = float("inf"), float("-inf"), float("nan"), float("inf")
    y, rows = _product(codes, norms, cent, n, k, bad, code, m), torch.ones(m, dtype=torch.bool, device="cuda")
    rows[[3, 17, 32, m - 1]] = False
    assert torch.equal(y[rows], want[rows]) and not torch.isfinite(y[~rows]).any()
    # one element off a 16-byte boundary: fp16 rows then take the form that rotates them
    off = held[1:1 + m * k].view(m, k)
    dense = ((cent.double()[codes.long()].view(-1, 64) / 8) @ hadamard_matrix(64).cuda().double() * norms.double()[:, None]).view(n, k)
    assert O.rel_l2(_product(codes, norms, cent, n, k, off, code, m).double().cpu().numpy(), (off.double() @ dense.T).cpu().numpy()) < 2e-6
