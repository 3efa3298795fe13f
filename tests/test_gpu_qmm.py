"""``eoq_b200_linear_packed`` / ``eoq_b200_linear_polar_codes``: activations times weights that stay quantised, on tcgen05 tensor
cores, against the dequantised product in fp64 at the edges of its tiles: weight rows around 128, tokens around the token
tiles of every variant, column counts that end inside a block or a weight copy, groups of half a block to several."""
import numpy as np
import pytest
import torch

from eoq_quantization_b200 import _lib as L
from eoq_quantization_b200.core.polar_quant import hadamard_matrix
from eoq_quantization_b200.core.quantized_linear import QuantizedLinear
from oracle import oracle as O

pytestmark = pytest.mark.gpu
CODE = {torch.float16: L.F16, torch.bfloat16: L.BF16, torch.float32: L.F32}


def _pack(c, bits):
    if bits == 8:
        return c.to(torch.int8).contiguous()
    u = (c + (1 << (bits - 1)) - 1).to(torch.uint8)
    per = 8 // bits
    return sum(u[:, i::per] << (bits * i) for i in range(per)).to(torch.uint8).contiguous()


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("bits", [2, 4, 8])
@pytest.mark.parametrize("n,k,group", [(1, 128, 32), (127, 192, 64), (300, 1344, 96), (129, 4096, 256), (1000, 2816, 128), (2500, 1024, 1024)])
def test_packed_product(bits, n, k, group):
    g = torch.Generator(device="cuda").manual_seed(bits + n)
    qmax = (1 << (bits - 1)) - 1
    c = torch.randint(-qmax, qmax + 1, (n, k), generator=g, device="cuda")
    s = (torch.rand(n, k // group, generator=g, device="cuda") * 0.01 + 1e-3).half()
    dense = (c.double().view(n, -1, group) * s.double()[:, :, None]).view(n, k) if k % group == 0 else None
    packed, bias = _pack(c, bits), torch.randn(n, generator=g, device="cuda")
    for dt in CODE:
        for m in (1, 16, 17, 32, 33, 64, 65, 128, 129, 257, 600):
            x = torch.randn(m, k, generator=g, device="cuda").to(dt)
            y = torch.empty(m, n, dtype=torch.float32, device="cuda")
            scratch = torch.empty(m * (k + 1), device="cuda")
            rc = L.lib().eoq_b200_linear_packed(packed.data_ptr(), s.data_ptr(), n, k, bits, group, x.data_ptr(), CODE[dt], m, scratch.data_ptr(),
                                                y.data_ptr(), L.F32, bias.data_ptr(), _stream())
            if k % (64 if bits == 2 else 32 if bits == 4 else 16):
                assert rc == L.EOQ_ERR_UNSUPPORTED
                continue
            assert rc == L.EOQ_OK
            want = x.double() @ dense.T + bias.double()
            # exact codes and fp32 scales, or (more than 128 rows of 16-bit activations) one rounding of code x scale
            tol = 2e-6 if m <= 128 or dt == torch.float32 else 4e-4 if dt == torch.float16 else 3e-3
            assert O.rel_l2(y.cpu().numpy(), want.cpu().numpy()) < tol, (dt, m)
    assert L.lib().eoq_b200_linear_status() == 0


@pytest.mark.parametrize("bits,block", [(3, 64), (5, 64), (8, 128), (4, 256)])
@pytest.mark.parametrize("n,k", [(1, 256), (130, 1280), (700, 4096)])
def test_polar_product(bits, block, n, k):
    g = torch.Generator(device="cuda").manual_seed(bits + n)
    codes = torch.randint(0, 1 << bits, (n, k), generator=g, device="cuda").to(torch.uint8)
    norms = (torch.rand(n * k // block, generator=g, device="cuda") * 2 + 0.1).half()
    cent = torch.sort(torch.randn(1 << bits, generator=g, device="cuda"))[0]
    H = hadamard_matrix(block).cuda().double()
    dense = ((cent.double()[codes.long()].view(-1, block) / block ** 0.5) @ H * norms.double()[:, None]).view(n, k)
    bias = torch.randn(n, generator=g, device="cuda").half()
    for dt in CODE:
        for m, size in ((1, 1.0), (16, 1e-5), (33, 1.0), (128, 1e5), (200, 1.0)):          # rows of any magnitude
            x = (torch.randn(m, k, generator=g, device="cuda") * (size if dt != torch.float16 else 1.0)).to(dt)
            y = torch.empty(m, n, dtype=torch.float32, device="cuda")
            scratch = torch.empty(m * (k + 1), device="cuda")
            assert L.lib().eoq_b200_linear_polar_codes(codes.data_ptr(), norms.data_ptr(), cent.data_ptr(), n, k, bits, block, x.data_ptr(), CODE[dt], m,
                                                       scratch.data_ptr(), y.data_ptr(), L.F32, bias.data_ptr(), L.F16, _stream()) == L.EOQ_OK
            want = x.double() @ dense.T + bias.double()
            assert O.rel_l2(y.cpu().numpy(), want.cpu().numpy()) < 2e-6, (dt, m)
    assert L.lib().eoq_b200_linear_status() == 0


@pytest.mark.parametrize("n,k,group", [(96, 128, 32), (97, 256, 64), (1000, 1024, 128), (2305, 640, 128), (5000, 4096, 128)])
def test_entropy_coded_product(n, k, group):
    """EOQWeight.linear beyond the fused GEMV's rows: codes decoded two per byte, then the same product; the packed codes
    themselves against the symbols, odd numbers of row blocks and rows past the matrix among them."""
    from eoq_quantization_b200.fused import EOQWeight
    rng = np.random.default_rng(n)
    codes, scales = O.quantize_absmax((rng.standard_normal((n, k)) * 0.02).astype(np.float32), 4, group)
    s16 = scales.astype(np.float16)
    w = EOQWeight.from_symbols((codes + 7).astype(np.uint8), s16, group=group)
    assert np.array_equal(w.decode_symbols(packed=True).cpu().numpy(), O.pack_int4_rows(codes))
    dense = torch.from_numpy((codes.reshape(-1, group).astype(np.float64) * s16.astype(np.float64)[:, None]).reshape(n, k)).cuda()
    bias = torch.randn(n, device="cuda")
    for dt in CODE:
        for m in (1, 2, 3, 5, 8, 9, 40, 130, 300):
            x = torch.randn(m, k, device="cuda").to(dt)
            want = x.double() @ dense.T + bias.double()
            tol = 1e-5 if dt == torch.float32 else 1e-3 if dt == torch.float16 else 6e-3
            for _ in range(2):
                assert O.rel_l2(w.linear(x, bias).double().cpu().numpy(), want.cpu().numpy()) < tol, (dt, m)
    assert w.status() == 0 and L.lib().eoq_b200_linear_status() == 0


def test_modules_fall_back_outside_the_native_route():
    """Gradients through x, activations that are not contiguous or not aligned, no rows: the Python path, same results."""
    torch.manual_seed(1)
    ql = QuantizedLinear.from_float(torch.nn.Linear(256, 96), bits=4, block_size=64).cuda()
    w = ql._dequantize_weight()
    x = torch.randn(40, 256, device="cuda")
    want = torch.nn.functional.linear(x, w, ql.bias_param)
    for arg in (x, torch.randn(256, 40, device="cuda").copy_(x.T).T, torch.cat([x.flatten(), x.flatten()[:1]])[1:].view(40, 256)):
        ref = want if arg is x or arg.shape == x.shape and torch.equal(arg, x) else torch.nn.functional.linear(arg, w, ql.bias_param)
        assert O.rel_l2(ql(arg).cpu().numpy(), ref.cpu().numpy()) < 1e-5
    assert ql(x[:0]).shape == (0, 96)
    xg = x.clone().requires_grad_()
    ql(xg).sum().backward()
    assert O.rel_l2(xg.grad.cpu().numpy(), w.sum(0).expand(40, -1).cpu().numpy()) < 1e-5


@pytest.mark.parametrize("n,k", [(2047, 136), (2049, 264), (41, 136), (2048, 136)])
def test_rows_that_end_inside_a_scale_group(n, k):
    """A dequantised copy with rows added until y's rows are 16-byte multiples: around the sizes where that starts."""
    torch.manual_seed(n)
    for bits in (2, 4, 8):
        ql = QuantizedLinear.from_float(torch.nn.Linear(k, n), bits=bits, block_size=128).cuda()
        w, b = ql._dequantize_weight().double(), ql.bias_param.double()
        for dt, tol in ((torch.float16, 1e-3), (torch.bfloat16, 8e-3), (torch.float32, 1e-5)):
            for m in (1, 8, 32, 33):
                x = torch.randn(2, m, k, device="cuda").to(dt) if m > 8 else torch.randn(m, k, device="cuda").to(dt)
                y = ql(x)
                assert y.dtype == dt and y.shape == (*x.shape[:-1], n) and y.is_contiguous()
                assert O.rel_l2(y.double().cpu().numpy(), (x.double() @ w.T + b).cpu().numpy()) < tol, (bits, dt, m)


@pytest.mark.parametrize("bits,block,n,k", [(5, 64, 130, 192), (8, 256, 77, 512), (3, 64, 300, 4160), (1, 128, 129, 384)])
def test_polar_product_many_rows(bits, block, n, k):
    """Centroid x norm as two halves: norms of one row four decades apart, rows all zero, token tiles around their sizes."""
    g = torch.Generator(device="cuda").manual_seed(bits + n)
    codes = torch.randint(0, 1 << bits, (n, k), generator=g, device="cuda").to(torch.uint8)
    norms = (10 ** (torch.rand(n, k // block, generator=g, device="cuda") * 4 - 3)).half()
    norms[n // 2] = 0
    cent = torch.sort(torch.randn(1 << bits, generator=g, device="cuda"))[0]
    H = hadamard_matrix(block).cuda().double()
    dense = ((cent.double()[codes.long()].view(-1, block) / block ** 0.5) @ H * norms.double().view(-1, 1)).view(n, k)
    for m in (112, 113, 255, 256, 257, 520):
        x = torch.randn(m, k, generator=g, device="cuda")
        y = torch.empty(m, n, device="cuda")
        scratch = torch.empty(m * (k + 1), device="cuda")
        assert L.lib().eoq_b200_linear_polar_codes(codes.data_ptr(), norms.data_ptr(), cent.data_ptr(), n, k, bits, block, x.data_ptr(), L.F32, m,
                                                   scratch.data_ptr(), y.data_ptr(), L.F32, None, L.F32, _stream()) == L.EOQ_OK
        want = x.double() @ dense.T
        err = (y.double() - want).norm(dim=0) / want.norm(dim=0).clamp_min(1e-30)          # each row of the weight by itself
        assert err.max().item() < 3e-6, m
    assert L.lib().eoq_b200_linear_status() == 0


@pytest.mark.parametrize("n,k", [(2400, 384), (2369, 1024), (9488, 640), (14224, 128), (16400, 256)])
def test_packed_gemv_warp_counts(n, k):
    """Few rows by the warp-level kernel where its CTAs have idle warps, an odd number of warps, or need a second round."""
    g = torch.Generator(device="cuda").manual_seed(n)
    for bits in (2, 4, 8):
        qmax = (1 << (bits - 1)) - 1
        c = torch.randint(-qmax, qmax + 1, (n, k), generator=g, device="cuda")
        s = (torch.rand(n, k // 128, generator=g, device="cuda") * 0.01 + 1e-3).half()
        dense, packed = (c.double().view(n, -1, 128) * s.double()[:, :, None]).view(n, k), _pack(c, bits)
        for m in (1, 8):
            x = torch.randn(m, k, generator=g, device="cuda").half()
            y = torch.empty(m, n, device="cuda")
            assert L.lib().eoq_b200_gemv_packed(packed.data_ptr(), s.data_ptr(), n, k, bits, 128, x.data_ptr(), L.F16, m, None, y.data_ptr(), L.F32,
                                                None, _stream()) == L.EOQ_OK
            assert O.rel_l2(y.cpu().numpy(), (x.double() @ dense.T).cpu().numpy()) < 2e-6, (bits, m)


def test_errors_of_the_library_are_raised():
    """A call that the library refuses or fails is an exception, not a second attempt by another route."""
    x = torch.randn(1, 256, device="cuda").half()
    native = L.native()
    for rows in (1, 40):                                      # a weight that is gone: the fused GEMV, the decode to a dense matrix
        with pytest.raises(L.EOQError) as e:
            native.weight_linear(0, x.get_device(), 96, 256, 4, 8, x.expand(rows, 256).contiguous(), None)
        assert e.value.code == L.EOQ_ERR_NULL_PTR


@pytest.mark.parametrize("bits,group", [(4, 128), (8, 32)])
def test_fp32_rows_with_infinities(bits, group):
    """A row with infinities among its values: infinite or NaN exactly where the dequantised product is, and the other rows untouched."""
    torch.manual_seed(bits)
    ql = QuantizedLinear.from_float(torch.nn.Linear(512, 200), bits=bits, block_size=group).cuda()
    w = ql._dequantize_weight().double()
    for m in (1, 12, 40, 200):
        x = torch.randn(m, 512, device="cuda") * 1e5
        x[0, 7] = float("inf")
        if m > 2:
            x[2, 100], x[2, 101] = float("inf"), float("-inf")
        y, want = ql(x), x.double() @ w.T + ql.bias_param.double()
        assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isinf(y), torch.isinf(want))
        assert torch.equal(y[torch.isinf(y)].sign(), want[torch.isinf(want)].sign().float())
        finite = [i for i in range(m) if i not in (0, 2)]
        if finite:
            assert O.rel_l2(y[finite].cpu().numpy(), want[finite].cpu().numpy()) < 1e-5
