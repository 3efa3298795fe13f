"""Host-visible behaviour of the bounded waits.  The fused all-gather's waiting half: a wait for words nobody sends runs out after the
limit set on the host, the kernel returns, the status call reports the failure once and the object stays usable.
Nothing here faults or hangs: the wait is bounded by design and the limit is set to a few milliseconds."""
import ctypes as C

import numpy as np
import pytest
import torch

from eoq_quantization_b200 import _lib as L

pytestmark = pytest.mark.gpu


def test_wait_for_a_peer_that_never_sends_expires_and_reports():
    lib = L.lib()
    torch.cuda.set_device(0)
    handle = (C.c_ubyte * 64)()
    g = C.c_void_p()
    L.check(lib.eoq_b200_gather_create(2, 0, 2, 2 * 96 * 2, C.byref(g), handle), "eoq_b200_gather_create")
    try:
        assert lib.eoq_b200_gather_set_timeout_ms(g, 0) == L.EOQ_ERR_UNSUPPORTED
        L.check(lib.eoq_b200_gather_set_timeout_ms(g, 5), "eoq_b200_gather_set_timeout_ms")
        assert lib.eoq_b200_gather_status(g, None) == 0
        # rank 1 does not exist: its 32 words of slot 0 never arrive
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        t0.record()
        L.check(lib.eoq_b200_gather_wait(g, 0, 96, 1, L.F16, 3, torch.cuda.current_stream().cuda_stream), "eoq_b200_gather_wait")
        t1.record()
        torch.cuda.synchronize()
        assert 1.0 < t0.elapsed_time(t1) < 500.0            # gave up after about the limit, far below the default second
        assert lib.eoq_b200_gather_status(g, None) == L.EOQ_ERR_CUDA
        assert lib.eoq_b200_gather_status(g, None) == 0      # reported once; the context and the object are still usable
        assert lib.eoq_b200_gather_wait(g, 7, 96, 1, L.F16, 3, None) == L.EOQ_ERR_UNSUPPORTED
        assert lib.eoq_b200_gather_wait(g, 0, 1 << 20, 1, L.F16, 3, None) == L.EOQ_ERR_BUFFER_TOO_SMALL
        y = torch.ones(8, device="cuda") * 2                 # ordinary work still runs on the device
        assert float(y.sum()) == 16.0
    finally:
        lib.eoq_b200_gather_destroy(g)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_weight_used_with_another_device_current_is_refused_before_any_launch():
    from eoq_quantization_b200.fused import EOQWeight
    lib = L.lib()
    rng = np.random.default_rng(0)
    sym = rng.integers(0, 15, (96, 128), dtype=np.uint8)
    sc = np.ones(96, np.float16)
    with torch.cuda.device(0):
        w = EOQWeight.from_symbols(sym, sc)
        x0 = torch.zeros(1, 128, device="cuda:0", dtype=torch.float16)
    with torch.cuda.device(1):
        x1 = torch.zeros(1, 128, device="cuda:1", dtype=torch.float16)
        y1 = torch.full((1, 96), 3.0, device="cuda:1", dtype=torch.float16)
        n0 = lib.eoq_b200_launch_count()
        rc = lib.eoq_b200_gemv(w._h, x1.data_ptr(), L.F16, 1, y1.data_ptr(), L.F16, None, None)
        assert rc == L.EOQ_ERR_UNSUPPORTED and lib.eoq_b200_launch_count() == n0
        assert lib.eoq_b200_gemm(w._h, x1.data_ptr(), L.F16, 16, y1.data_ptr(), L.F16, None, None) == L.EOQ_ERR_UNSUPPORTED
        assert lib.eoq_b200_gemv_static_scratch(w._h, x1.data_ptr(), L.F16, 1, y1.data_ptr(), L.F16, None, None) == L.EOQ_ERR_UNSUPPORTED
        assert lib.eoq_b200_launch_count() == n0
        torch.cuda.synchronize()
        assert float(y1.float().min()) == 3.0
        with pytest.raises(RuntimeError):
            w.gemv(x1)                                        # the Python wrapper refuses activations on another device
        assert w.gemv(x0).shape == (1, 96)                    # and makes the weight's device current for its own


def _gather(lib, milliseconds):
    handle, g = (C.c_ubyte * 64)(), C.c_void_p()
    L.check(lib.eoq_b200_gather_create(2, 0, 2, 2 * 96 * 2, C.byref(g), handle), "eoq_b200_gather_create")
    L.check(lib.eoq_b200_gather_set_timeout_ms(g, milliseconds), "eoq_b200_gather_set_timeout_ms")
    return g


def _products():
    """(name, launch, result, expected result, weight) of every form of the product kernel: scale groups folded or applied to
    the codes, byte codes either way, fp32 rows, several CTAs a tile, and the codes a decoder leaves."""
    from eoq_quantization_b200.core.polar_quant import hadamard_matrix
    from eoq_quantization_b200.fused import EOQWeight
    lib, st = L.lib(), torch.cuda.current_stream().cuda_stream
    torch.manual_seed(0)
    n, k = 300, 1024
    c = torch.randint(-7, 8, (n, k), device="cuda")
    s = (torch.rand(n, k // 128, device="cuda") * 0.01 + 1e-3).half()
    dense = (c.double().view(n, -1, 128) * s.double()[:, :, None]).view(n, k)
    u = (c + 7).to(torch.uint8)
    packed = (u[:, 0::2] | (u[:, 1::2] << 4)).contiguous()
    centroids = torch.sort(torch.randn(256, device="cuda"))[0]
    norms, bytes_ = (torch.rand(n * k // 64, device="cuda") + 0.1).half(), torch.randint(0, 256, (n, k), device="cuda").to(torch.uint8)
    polar = ((centroids.double()[bytes_.long()].view(-1, 64) / 8.0) @ hadamard_matrix(64).cuda().double() * norms.double()[:, None]).view(n, k)
    weight = EOQWeight.from_device_symbols(u, s.flatten())
    for name, rows, dt in (("fold", 16, torch.float16), ("fold", 100, torch.bfloat16), ("fold", 40, torch.float32), ("scaled", 300, torch.float16),
                           ("polar", 16, torch.float16), ("polar, many rows", 200, torch.float32), ("decoded", 300, torch.float16)):
        x = torch.randn(rows, k, device="cuda").to(dt)
        y, scratch = torch.empty(rows, n, device="cuda"), torch.empty(rows * (k + 1) + n * k, device="cuda")
        code = {torch.float16: L.F16, torch.bfloat16: L.BF16, torch.float32: L.F32}[dt]
        if name.startswith("polar"):
            call = lambda x=x, y=y, m=rows, code=code, scratch=scratch: lib.eoq_b200_linear_polar_codes(
                bytes_.data_ptr(), norms.data_ptr(), centroids.data_ptr(), n, k, 8, 64, x.data_ptr(), code, m, scratch.data_ptr(), y.data_ptr(), L.F32,
                None, L.F32, st)
        elif name == "decoded":
            call = lambda x=x, y=y, m=rows, code=code, scratch=scratch: lib.eoq_b200_weight_linear(
                weight._h, x.data_ptr(), code, m, scratch.data_ptr(), y.data_ptr(), L.F32, None, st)
        else:
            call = lambda x=x, y=y, m=rows, code=code, scratch=scratch: lib.eoq_b200_linear_packed(
                packed.data_ptr(), s.data_ptr(), n, k, 4, 128, x.data_ptr(), code, m, scratch.data_ptr(), y.data_ptr(), L.F32, None, st)
        yield name, call, y, x.double() @ (polar if name.startswith("polar") else dense).T, weight


def _right(y, want):
    return bool(torch.isfinite(y).all()) and ((y.double() - want).norm() / want.norm()).item() < 4e-4       # code x scale in fp16: 2^-11 at most


def test_product_behind_a_kernel_that_takes_longer_than_its_waits_may():
    """The kernel before a product may run on for longer than the product's waits are allowed: that time does not count."""
    lib = L.lib()
    g = _gather(lib, 200)
    assert lib.eoq_b200_tune(b"qmm_wait_us", 20000) == 0
    try:
        for name, call, y, want, weight in _products():
            torch.cuda.synchronize()
            L.check(lib.eoq_b200_gather_wait(g, 0, 96, 1, L.F16, 3, torch.cuda.current_stream().cuda_stream), "eoq_b200_gather_wait")
            L.check(call(), name)
            assert _right(y, want), name
            assert lib.eoq_b200_linear_status() == 0 and weight.status() == 0, name
            assert lib.eoq_b200_gather_status(g, None) == L.EOQ_ERR_CUDA
    finally:
        lib.eoq_b200_tune(b"qmm_wait_us", 2000000)
        lib.eoq_b200_gather_destroy(g)


def test_product_whose_waits_run_out_says_so_and_leaves_the_next_one_alone():
    """A wait that runs out (no patience for the kernel in front, which waits for a peer that never sends) gives NaN and a
    status, at the weight where there is one; the calls after it are right, whether or not anybody has read the status."""
    lib = L.lib()
    g = _gather(lib, 100)
    try:
        for name, call, y, want, weight in _products():
            if name == "polar, many rows":         # the kernel that rotates its rows fills the device: the product cannot start beside it
                continue
            for _ in range(2):
                torch.cuda.synchronize()
                assert lib.eoq_b200_tune(b"qmm_wait_us", 0) == 0
                L.check(lib.eoq_b200_gather_wait(g, 0, 96, 1, L.F16, 3, torch.cuda.current_stream().cuda_stream), "eoq_b200_gather_wait")
                L.check(call(), name)
                torch.cuda.synchronize()
                assert torch.isnan(y).any(), name
                assert lib.eoq_b200_tune(b"qmm_wait_us", 2000000) == 0
                L.check(call(), name)
                assert _right(y, want), name
            if name == "decoded":
                assert weight.status() == L.EOQ_ERR_CUDA and lib.eoq_b200_linear_status() == 0
            else:
                assert lib.eoq_b200_linear_status() == 1 and lib.eoq_b200_linear_status() == 0 and weight.status() == 0
    finally:
        lib.eoq_b200_tune(b"qmm_wait_us", 2000000)
        lib.eoq_b200_gather_destroy(g)
