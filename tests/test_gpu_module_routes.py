"""The routes of the modules' forward calls for what a program makes of them: the same kernels, straight from the codes, whatever
the activations' layout, the types that a cast left in the module, and the mode the call is made in.  A dense copy of the weight
shows in the allocator's peak, an entropy-coded one in the module."""
import numpy as np
import pytest
import torch

from eoq_quantization_b200.core.eoq_linear import EOQLinear
from eoq_quantization_b200.core.polar_quant import hadamard_matrix
from eoq_quantization_b200.core.quantized_linear import QuantizedLinear
from eoq_quantization_b200.core.quantized_matmul import QuantizedLinearFast
from eoq_quantization_b200.fused import EOQWeight
from eoq_quantization_b200.kernels.polar_engine import PolarLinear
from oracle import oracle as O

pytestmark = pytest.mark.gpu
N, K = 2048, 4096                                             # a dense 16-bit copy of the weight: 16 MB
TOL = {torch.float16: 1e-3, torch.bfloat16: 8e-3, torch.float32: 1e-5}      # the result's rounding (and one of code x scale beyond 128 rows)
ROWS = (1, 8, 24, 200)


def _layer(kind, bias=True):
    torch.manual_seed(3)
    lin = torch.nn.Linear(K, N, bias=bias)
    if kind == "packed":
        return QuantizedLinear.from_float(lin, bits=4, block_size=128).cuda()
    if kind == "fast":
        return QuantizedLinearFast.from_linear(lin, bits=4, block_size=128).cuda()
    if kind == "polar":
        return PolarLinear.from_linear(lin.cuda(), bits=5, block_size=64)
    q = QuantizedLinear.from_float(lin, bits=4, block_size=128).cuda()
    return EOQLinear(EOQWeight.from_int4_packed(q.packed_weight, q.scales, K), q.bias_param)


def _dense(layer):
    """The weight in 64 bits, of the scales, norms and centroids as the module holds them."""
    if isinstance(layer, PolarLinear):
        values = layer.centroids.double()[layer.codes.long()].view(-1, layer.block_size) / layer.block_size ** 0.5
        return (values @ hadamard_matrix(layer.block_size).cuda().double() * layer.norms.double()[:, None]).view(N, K)
    return (QuantizedLinear._dequantize_weight(layer) if isinstance(layer, QuantizedLinearFast) else layer._dequantize_weight()).double()


def _taken(layer, x):
    """(result, bytes of device memory that the call needed at its peak)."""
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    y = layer(x)
    return y, torch.cuda.max_memory_allocated() - before


def _check(layer, x, dense, plain, extra=0, dtype=None):
    """The product within the result's type, without an entropy-coded copy of the weight, and without a dense one where `plain`
    (bytes the plain call on a plain module takes) has none: at most `extra` bytes more (and two megabytes, the allocator's rounding)."""
    y, taken = _taken(layer, x)
    dtype = dtype or (torch.float16 if isinstance(layer, PolarLinear) else x.dtype)
    assert y.dtype == dtype and y.shape == (*x.shape[:-1], N)
    want = x.detach().double() @ dense.T + (0 if layer.bias is None else layer.bias.double())
    tol = TOL[torch.float16] if isinstance(layer, PolarLinear) else TOL[dtype]           # PolarLinear: fp16 before the bias is added
    assert O.rel_l2(y.detach().double().cpu().numpy(), want.cpu().numpy()) < tol, (x.shape, x.dtype)
    assert taken <= plain + extra + (2 << 20), (taken, plain, x.shape, x.dtype)
    assert getattr(layer, "_eoq", None) is None
    return y


def _plain(layer):
    """What the plain call takes for every number of rows and type: no dense copy up to 24 rows."""
    took = {(m, dt): _taken(layer, torch.randn(m, K, device="cuda").to(dt))[1] for m in ROWS for dt in TOL}
    assert max(v for (m, _), v in took.items() if m <= 24) < N * K
    return took


def _odd(x, how):
    """The same values, strided or off the 16-byte grid."""
    if how == "strided":
        return torch.stack([x, x], dim=-1)[..., 0]
    if how == "transposed":
        return x.T.contiguous().T
    return torch.cat([x.flatten(), x.flatten()[:1]])[1:].view_as(x) if how == "misaligned" else x


@pytest.mark.parametrize("kind", ["packed", "fast", "eoq", "polar"])
@pytest.mark.parametrize("how", ["strided", "transposed", "misaligned"])
def test_activations_that_are_not_plain_take_the_codes_route(kind, how):
    layer = _layer(kind)
    dense, plain = _dense(layer), _plain(layer)
    for rows, dt in plain:
        x = _odd(torch.randn(rows, K, device="cuda").to(dt), how)
        _check(layer, x, dense, plain[rows, dt], extra=x.numel() * x.element_size())          # the copy of the activations


class _Sub(torch.Tensor):
    pass


def test_tensor_subclasses_take_the_codes_route():
    layer = _layer("packed")
    dense = _dense(layer)
    for rows in (1, 8, 24):
        x = torch.randn(rows, K, device="cuda").half().as_subclass(_Sub)
        assert O.rel_l2(layer(x).as_subclass(torch.Tensor).double().cpu().numpy(),
                        (x.as_subclass(torch.Tensor).double() @ dense.T + layer.bias_param.double()).cpu().numpy()) < 1e-3
        assert layer._eoq is None


@pytest.mark.parametrize("kind", ["packed", "fast", "eoq", "polar"])
@pytest.mark.parametrize("to", [torch.float16, torch.bfloat16, torch.float32, torch.float64])
def test_modules_that_were_cast_take_the_codes_route(kind, to):
    layer = _layer(kind)
    plain = _plain(layer)
    layer = layer.to(to)
    dense = _dense(layer)
    result = torch.promote_types(torch.float16, to) if kind == "polar" else None         # fp16, to which the bias is added
    for rows, dt in plain:
        if kind == "polar" and rows > 32 and to in (torch.float32, torch.float64):
            continue                                          # norms wider than the kernels' are not rounded for a prompt
        y = _check(layer, torch.randn(rows, K, device="cuda").to(dt), dense, plain[rows, dt], extra=rows * N * 8 * (result not in (None, torch.float16)),
                   dtype=result)
        del y


def test_scales_converted_for_a_call_are_complete_when_they_are_read():
    """A cast module's scales are converted in front of every call; kernels that start under the one before them wait for that."""
    layer = _layer("packed", bias=False).bfloat16()
    scales = [layer.scales, layer.scales * 2]
    x = torch.randn(1, K, device="cuda").half()
    want = []
    for s in scales:
        layer.scales = s
        torch.cuda.synchronize()
        want.append(layer(x))
    torch.cuda.synchronize()
    got = []
    for i in range(400):                                      # back to back: the conversion's memory is the last call's, with other values
        layer.scales = scales[i % 2]
        got.append(layer(x))
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 2]), i


@pytest.mark.parametrize("kind", ["packed", "fast", "eoq", "polar"])
def test_gradients_of_the_bias_and_of_the_activations(kind):
    layer = _layer(kind)
    dense = _dense(layer).float()
    x = torch.randn(40, K, device="cuda")
    like = _taken(layer, x)[1]
    layer.bias.requires_grad_()
    g = torch.randn(40, N, device="cuda")
    y, taken = _taken(layer, x)
    assert taken <= like + (2 << 20) and like < N * K
    y.backward(g.to(y.dtype))
    assert O.rel_l2(layer.bias.grad.double().cpu().numpy(), g.sum(0).double().cpu().numpy()) < 1e-3       # an fp16 bias's gradient
    layer.bias.requires_grad_(False)
    x.requires_grad_()
    y = layer(x)
    y.backward(g.to(y.dtype))
    assert O.rel_l2(x.grad.cpu().numpy(), (g @ dense).cpu().numpy()) < (1e-3 if kind == "polar" else 1e-5)      # polar: fp16 results' gradient


@pytest.mark.parametrize("kind", ["packed", "fast", "eoq", "polar"])
@pytest.mark.parametrize("rows", [1, 40])
def test_forward_mode_tangents_are_carried(kind, rows):
    layer = _layer(kind)
    dense = _dense(layer).float()
    x, v = torch.randn(rows, K, device="cuda"), torch.randn(rows, K, device="cuda")
    with torch.autograd.forward_ad.dual_level():
        y, t = torch.autograd.forward_ad.unpack_dual(layer(torch.autograd.forward_ad.make_dual(x, v)))
        assert t is not None and O.rel_l2(t.float().cpu().numpy(), (v @ dense.T).cpu().numpy()) < (1e-3 if kind == "polar" else 1e-5)
        assert O.rel_l2(y.float().cpu().numpy(), layer(x).float().cpu().numpy()) < (1e-3 if kind == "polar" else 1e-5)


@pytest.mark.parametrize("kind", ["packed", "eoq"])
@pytest.mark.parametrize("rows", [1, 40])
def test_vmap_runs_over_the_layers(kind, rows):
    layer = _layer(kind)
    x = torch.randn(3, rows, K, device="cuda")
    y = torch.vmap(layer)(x)
    assert O.rel_l2(y.cpu().numpy(), layer(x).cpu().numpy()) < 1e-5


@pytest.mark.parametrize("kind", ["packed", "eoq", "polar"])
def test_calls_under_autocast_take_the_codes_route(kind):
    """Results of the autocast type, as torch.nn.Linear gives them, but for the few rows of the fused GEMV (and PolarLinear's fp16)."""
    layer = _layer(kind)
    dense, plain = _dense(layer), _plain(layer)
    for rows, dt in plain:
        for to in (torch.float16, torch.bfloat16):
            few = rows <= (8 if dt == torch.float32 else 4)
            result = torch.float16 if kind == "polar" else dt if few else to
            with torch.autocast("cuda", dtype=to):
                y, taken = _taken(layer, x := torch.randn(rows, K, device="cuda").to(dt))
            assert y.dtype == result and getattr(layer, "_eoq", None) is None
            want = x.double() @ dense.T + layer.bias.double()
            tol = max(TOL[y.dtype], 0 if few or kind == "polar" else 2 * TOL[to])             # x is rounded to the autocast type, too
            assert O.rel_l2(y.double().cpu().numpy(), want.cpu().numpy()) < tol, (rows, dt, to)
            like = plain[rows, dt if few or kind == "polar" else to]
            assert taken <= like + x.numel() * 4 + (2 << 20), (taken, like, rows, dt, to)


@pytest.mark.parametrize("kind", ["packed", "fast", "eoq"])
@pytest.mark.parametrize("rows", [1, 3, 24])
def test_calls_that_want_gradients_take_the_codes_route(kind, rows):
    layer = _layer(kind)
    dense, plain = _dense(layer), _plain(layer)
    for dt in TOL:
        x = torch.randn(rows, K, device="cuda").to(dt).requires_grad_()
        y, taken = _taken(layer, x)
        like = _taken(layer, x.detach())[1]
        assert y.dtype == dt and taken <= like + (2 << 20) and like < N * K and getattr(layer, "_eoq", None) is None
        g = torch.randn(rows, N, device="cuda").to(dt)
        y.backward(g)
        assert x.grad.dtype == dt
        assert O.rel_l2(x.grad.double().cpu().numpy(), (g.double() @ dense).cpu().numpy()) < TOL[dt], dt
    if kind == "packed":
        y = layer(x)
        layer.scales.mul_(2)
        with pytest.raises(RuntimeError):                     # the weight that y was made with is gone
            y.backward(g)
