"""The work that a program using this package has it do, as cases that can be timed and compared.

A case is a dict of plain values; its ``path`` says which entry point it goes through:

  eoq           ``EOQLinear`` layers (entropy-coded weights resident on the GPU), what an ``.eoq`` model runs
  packed        ``QuantizedLinear`` layers (packed codes resident on the GPU), what ``replace_linear_with_quantized`` leaves
  polar         a ``PolarLinear`` layer (PolarQuant codes and norms)
  load          one tensor of an ``.eoq`` file to an ``EOQLinear``, and the layer's first prompt
  wire_decode   compressed bytes on the host to codes on the host
  wire_encode   codes on the host to compressed bytes on the host

``eoq`` and ``packed`` cases with ``block`` set run the seven linears of one decoder block (q, k, v, o, gate, up, down),
as a decode step calls them; their inputs stand for what attention and activation leave in a user's program.
"""
import math

import numpy as np
import torch

from eoq_quantization_b200.core.eoq_linear import EOQLinear
from eoq_quantization_b200.core.polar_quant import _ensure_centroids, polar_quantize
from eoq_quantization_b200.core.quantized_linear import QuantizedLinear
from eoq_quantization_b200.core.rans_bitpacked import CompressedTensorData, compress_tensor_rans, decompress_tensor_rans
from eoq_quantization_b200.core.rans_blocked import (BlockedRANSDecoder, BlockedRANSEncoder, deserialize_blocked_rans,
                                                     serialize_blocked_rans)
from eoq_quantization_b200.core.utils import quantize_absmax
from eoq_quantization_b200.eoq_file import EOQTensorRecord
from eoq_quantization_b200.fused import EOQWeight
from eoq_quantization_b200.kernels.polar_engine import PolarLinear

DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}
BYTES = {"float16": 2, "bfloat16": 2, "float32": 4}
# entropy of the absmax codes of Gaussian weights, bits per weight
ENTROPY = {2: 0.9, 3: 2.2, 4: 3.4, 5: 4.5, 6: 5.6, 8: 7.6}


def _linear(path, n, k, m, dtype, bits=4, group=128, bias=False, block=False, kv=0):
    """n x k layer on m rows; with block: hidden size k, intermediate size n, kv rows in the k and v projections."""
    return {"path": path, "n": n, "k": k, "m": m, "dtype": dtype, "bits": bits, "group": group, "bias": bias, "block": block, "kv": kv}


def _wire(path, n, bits, block, precision, api):
    return {"path": path, "n": n, "bits": bits, "block_size": block, "precision": precision, "api": api}


def listed():
    return [
        # one projection at one token: the smallest call there is, launch and host time show
        dict(_linear("eoq", 4096, 4096, 1, "float16"), name="eoq projection, 1 row"),
        # a decode step's linears of a 7B-shape decoder block, entropy-coded weights
        dict(_linear("eoq", 11008, 4096, 1, "float16", block=True, kv=4096), name="eoq block, decode"),
        # a long prompt through the widest projection of a 70B-shape model
        dict(_linear("eoq", 28672, 8192, 2048, "bfloat16"), name="eoq wide layer, prefill"),
        # the same decode step from packed codes
        dict(_linear("packed", 11008, 4096, 1, "float16", block=True, kv=4096), name="packed block, decode"),
        # some two dozen sequences decoded together
        dict(_linear("packed", 11008, 4096, 24, "bfloat16"), name="packed layer, batch 24"),
        # a model kept at eight bits with finer scales, fp32 activations, a few rows, an output width of no round size
        dict(_linear("packed", 3001, 2752, 5, "float32", bits=8, group=64, bias=True), name="packed 8-bit, fp32"),
        # a prompt on a packed layer
        dict(_linear("packed", 4096, 11008, 777, "float16", bias=True), name="packed layer, prefill"),
        # PolarQuant: a small batch decoded, and a prompt
        dict(_linear("polar", 14336, 4096, 4, "float16", bits=5, group=64), name="polar layer, batch 4"),
        dict(_linear("polar", 14336, 4096, 512, "float16", bits=5, group=64, bias=True), name="polar layer, prefill"),
        # a layer out of a model file on the disk's side of memory, to its first prompt
        dict(_linear("load", 11008, 4096, 16, "float16"), name="load and first prompt"),
        # the reference's container: a square layer in blocks of 4096 symbols decoded, and codes compressed as the
        # bit-packed pipeline does by default (blocks of 256)
        dict(_wire("wire_decode", 4096 * 4096, 4, 4096, 12, "blocked"), name="container to codes"),
        dict(_wire("wire_encode", 2048 * 2048, 4, 256, 14, "tensor"), name="codes to container"),
    ]


def _log(rng, lo, hi):
    """An integer from lo to hi, spread evenly over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges: every path, layers of a few hundred to 28672 rows and columns, one row to
    2048, each activation type, code width and group size, sizes off every power of two among them."""
    kind = rng.choice(["eoq", "eoq", "eoq prefill", "eoq block", "packed", "packed", "packed prefill", "packed block",
                       "polar", "polar prefill", "load", "wire_decode", "wire_encode"])
    path = kind.split()[0]
    dtype = rng.choice(["float16", "float16", "bfloat16", "bfloat16", "float32"])
    bias = rng.random() < 0.3
    if path in ("wire_decode", "wire_encode"):
        bits = rng.choice([4, 4, 4, 2, 3, 8])
        api = rng.choice(["blocked", "tensor"])
        block, precision = (256, 14) if api == "tensor" else rng.choice([(4096, 12), (1024, 14), (256, 16), (256, 14)])
        return _wire(path, _log(rng, 1 << 16, 1 << 22 if path == "wire_encode" else 1 << 24), bits, block, precision, api)
    if path == "polar":
        block = rng.choice([64, 64, 128])
        m = rng.randint(1, 32) if kind == "polar" else _log(rng, 33, 512)
        return _linear(path, _log(rng, 512, 14336), block * _log(rng, 512 // block, 8192 // block), m, dtype,
                       rng.choice([3, 4, 5, 5]), block, bias)
    group = rng.choice([128, 128, 64]) if path in ("eoq", "load") else rng.choice([128, 128, 128, 64, 32])
    bits = rng.choice([4, 4, 4, 2, 8]) if path == "packed" else 4
    if kind.endswith("block"):
        hidden = 128 * _log(rng, 8, 32)
        return _linear(path, 128 * _log(rng, 2 * hidden // 128, 11008 // 128), hidden, rng.choice([1, 1, 2, 4]), dtype,
                       bits, group, bias, True, rng.choice([hidden, hidden // 4]))
    if path == "load":
        return _linear(path, _log(rng, 512, 11008), 128 * _log(rng, 4, 32), _log(rng, 1, 64), rng.choice(["float16", "bfloat16"]), 4, group, bias)
    n, k = _log(rng, 512, 14336), 128 * _log(rng, 4, 86)
    if path == "packed" and rng.random() < 0.15:
        k += 8 * rng.randint(1, 15)           # rows that end inside a scale group, as the reference lays them out
    m = (rng.randint(1, 8) if path == "eoq" else rng.randint(1, 32)) if kind == path else _log(rng, 16, 2048)
    return _linear(path, n, k, m, dtype, bits, group, bias)


def _shapes(case):
    """(out, in) of the case's layers."""
    n, k = case["n"], case["k"]
    if not case["block"]:
        return [(n, k)]
    return [(k, k), (case["kv"], k), (case["kv"], k), (k, k), (n, k), (n, k), (k, n)]


def _wire_codes(case, gen):
    w = torch.randn(case["n"], generator=gen, device="cuda") * 0.02
    q = quantize_absmax(w, case["bits"], 128)
    return q.data, q.scale


def _layer(case, n, k, gen):
    """One layer of the case's path with Gaussian weights of deviation 0.02."""
    path, bits, group = case["path"], case["bits"], case["group"]
    w = torch.randn(n, k, generator=gen, device="cuda") * 0.02
    bias = torch.randn(n, generator=gen, device="cuda") * 0.1 if case["bias"] else None
    if path == "polar":
        res = polar_quantize(w, bits, group, use_qjl=False)
        return PolarLinear.from_polar_quant(res.codes, res.norms, _ensure_centroids(bits), (n, k), bits, group, bias=bias).cuda()
    q = quantize_absmax(w, bits, group)
    qmax = (1 << (bits - 1)) - 1
    if path == "eoq":
        return EOQLinear(EOQWeight.from_device_symbols((q.data + qmax).to(torch.uint8), q.scale.half(), group=group), bias, bits, group)
    layer = QuantizedLinear(k, n, bias=bias is not None, bits=bits, block_size=group).cuda()
    if bits == 8:
        layer.packed_weight.copy_(q.data)
    else:
        pack = QuantizedLinear.pack_4bit if bits == 4 else QuantizedLinear.pack_2bit
        layer.packed_weight.copy_(pack(q.data).view(n, -1))
    layer.scales.copy_(q.scale)
    if bias is not None:
        layer.bias_param.copy_(bias)
    return layer


@torch.no_grad()
def prepare(case, seed):
    """What a program has in hand before the call: the layers and their activations, or the host's bytes."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    path = case["path"]
    if path in ("wire_decode", "wire_encode"):
        codes, scales = _wire_codes(case, gen)
        codes, scales, bits, n = codes.to(torch.int8).cpu(), scales.cpu(), case["bits"], case["n"]
        qmax = (1 << (bits - 1)) - 1
        if case["api"] == "blocked":
            codes = codes.numpy().astype(np.int64) + qmax
        state = {"case": case, "codes": codes, "scales": scales}
        if path == "wire_decode":
            state["bytes"] = _encode(state)
        else:                     # the slot of the model file that the tensor's bytes go to, as long as they can get
            blocks = n // case["block_size"] + 1
            state["slot"] = np.zeros(32 + 4 * (1 << bits) + 10 * blocks + n * (2 * bits + 1) // 16, np.uint8)
        return state
    state = {"case": case, "x": [torch.randn(case["m"], k, generator=gen, device="cuda").to(DTYPES[case["dtype"]]) for _, k in _shapes(case)]}
    if path == "load":
        n, k = case["n"], case["k"]
        q = quantize_absmax(torch.randn(n, k, generator=gen, device="cuda") * 0.02, case["bits"], case["group"])
        rec = compress_tensor_rans("w", q.data, q.scale, case["bits"], case["group"], (n, k))
        state["record"] = EOQTensorRecord("w", (n, k), "float32", rec.bits, rec.block_size, rec.scales_bytes, rec.rans_bytes, rec.n_elements)
        state["bias"] = torch.randn(n, generator=gen, device="cuda") * 0.1 if case["bias"] else None
    else:
        state["layers"] = [_layer(case, n, k, gen) for n, k in _shapes(case)]
    return state


def _encode(state):
    case = state["case"]
    if case["api"] == "tensor":
        return compress_tensor_rans("w", state["codes"], state["scales"], case["bits"], 128, (case["n"],))
    enc = BlockedRANSEncoder(block_size=case["block_size"], precision_bits=case["precision"])
    return serialize_blocked_rans(enc.encode(state["codes"], 2 ** case["bits"] - 1))


@torch.no_grad()
def run(state):
    path = state["case"]["path"]
    if path == "wire_encode":
        got = _encode(state)
        whole = got.rans_bytes if isinstance(got, CompressedTensorData) else got
        slot = state["slot"]
        slot[:len(whole)] = np.frombuffer(whole, np.uint8)
        slot[len(whole):] = 0
        return [slot, np.frombuffer(got.scales_bytes, np.float16)] if isinstance(got, CompressedTensorData) else slot
    if path == "wire_decode":
        data = state["bytes"]
        if isinstance(data, CompressedTensorData):
            return decompress_tensor_rans(data)
        return BlockedRANSDecoder().decode_all(deserialize_blocked_rans(data))
    if path == "load":
        return EOQLinear.from_record(state["record"], state["bias"])(state["x"][0])
    return [layer(x) for layer, x in zip(state["layers"], state["x"])]


def work(case):
    """Bytes and operations of one pass that no implementation can do without: compressed weights and scales, inputs,
    outputs; two operations per weight and row."""
    if case["path"].startswith("wire"):
        n, wide = case["n"], 8 if case["api"] == "blocked" else 1
        scales = (4 + 2) * n / 128 if case["api"] == "tensor" else 0
        return {"bytes": n * ENTROPY[case["bits"]] / 8 + n * wide + scales, "flops": 0}
    m, e, bits = case["m"], BYTES[case["dtype"]], case["bits"]
    out_e = 2 if case["path"] == "polar" else e
    stored = ENTROPY[bits] if case["path"] in ("eoq", "load") else 8 if case["path"] == "polar" else bits
    total = flops = 0
    for n, k in _shapes(case):
        total += n * k * stored / 8 + 2 * n * k / case["group"] + m * k * e + m * n * out_e + (4 * n if case["bias"] else 0)
        flops += 2 * m * n * k
    return {"bytes": total, "flops": flops}


def tolerance(case):
    if case["path"].startswith("wire"):
        return "exact"
    if case["path"] == "polar":           # float16 results whatever the activations
        return {"rel": 1e-3, "max": 1e-2}
    if case["dtype"] == "bfloat16":
        return {"rel": 1e-2, "max": 6e-2}
    return {"rel": 1e-3, "max": 1e-2} if case["dtype"] == "float16" else {"rel": 1e-5, "max": 1e-4}
