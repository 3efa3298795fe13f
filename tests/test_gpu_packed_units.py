"""A few 16-bit rows against packed codes whose scale groups are not whole 128-column spans: groups of one to several units of 32 and
64 columns, tiles and spans at their edges, byte codes on either side of the row length where another kernel takes them."""
import numpy as np
import pytest
import torch

from eoq_quantization_b200.core.quantized_linear import QuantizedLinear
from eoq_quantization_b200.fused import gemv_packed, packed_gemv_applies
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("n,k,group", [(1, 128, 32), (17, 128, 64), (130, 384, 96), (33, 1152, 192), (1000, 4096, 64), (300, 2560, 32), (47, 8192, 64), (47, 8320, 64)])
def test_units_of_a_span(bits, n, k, group):
    g = torch.Generator(device="cuda").manual_seed(bits + n + k)
    qmax = (1 << (bits - 1)) - 1
    c = torch.randint(-qmax, qmax + 1, (n, k), generator=g, device="cuda")
    layer = QuantizedLinear(k, n, bias=True, bits=bits, block_size=group).cuda()
    if bits in (2, 4):
        per, u = 8 // bits, (c + qmax).to(torch.uint8)
        layer.packed_weight.copy_(sum(u[:, i::per] << (bits * i) for i in range(per)).to(torch.uint8).view(layer.packed_weight.shape))
    else:
        layer.packed_weight.copy_(c)
    layer.scales.copy_(torch.rand(layer.scales.shape, generator=g, device="cuda") * 0.01 + 1e-3)
    layer.bias_param.data.copy_(torch.randn(n, generator=g, device="cuda"))
    dense = (c.double().view(n, -1, group) * layer.scales.double().view(n, -1, 1)).view(n, k)
    for dt in (torch.float16, torch.bfloat16):
        for m in (1, 2, 7, 8, 9):
            x = torch.randn(m, k, generator=g, device="cuda").to(dt)
            want = x.double() @ dense.T + layer.bias_param.double()
            with torch.no_grad():
                y = layer(x)
            # one rounding of the result (of one value where the layer has one output)
            assert O.rel_l2(y.double().cpu().numpy(), want.cpu().numpy()) < (2 ** -11 if dt == torch.float16 else 2 ** -8), (dt, m)
            if m <= 8 and packed_gemv_applies(k, bits, group, dt, m):
                y = gemv_packed(layer.packed_weight, layer.scales, n, k, bits, group, x, layer.bias_param, out_dtype=torch.float32)
                assert O.rel_l2(y.cpu().numpy(), want.cpu().numpy()) < 1e-6, (dt, m)


@pytest.mark.parametrize("bits,group", [(4, 64), (4, 32), (2, 64), (8, 64), (8, 32)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_rows_that_are_not_finite(bits, group, dt):
    n, k, m = 40, 256, 8
    g = torch.Generator(device="cuda").manual_seed(bits + group)
    qmax = (1 << (bits - 1)) - 1
    c = torch.randint(-qmax, qmax + 1, (n, k), generator=g, device="cuda")
    packed = c.to(torch.int8) if bits == 8 else sum((c + qmax)[:, i::8 // bits].to(torch.uint8) << (bits * i) for i in range(8 // bits)).to(torch.uint8)
    scales, x = (torch.rand(n, k // group, generator=g, device="cuda") + 0.1).half(), torch.randn(m, k, generator=g, device="cuda").to(dt)
    want = gemv_packed(packed, scales, n, k, bits, group, x, out_dtype=torch.float32)
    x[1, 7], x[4, group], x[6, 255] = float("inf"), float("-inf"), float("nan")
    y = gemv_packed(packed, scales, n, k, bits, group, x, out_dtype=torch.float32)
    assert torch.equal(y[[0, 2, 3, 5, 7]], want[[0, 2, 3, 5, 7]]) and torch.isnan(y[6]).all()
    inf = float("inf")
    for row, col, sign in ((1, 7, 1), (4, group, -1)):            # a zero code times infinity is NaN, others take its sign
        expect = torch.where(c[:, col] == 0, torch.full((n,), float("nan"), device="cuda"), sign * torch.sign(c[:, col]) * inf)
        assert torch.equal(torch.nan_to_num(y[row], 123.0), torch.nan_to_num(expect, 123.0))
