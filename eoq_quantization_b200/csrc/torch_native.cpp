// The modules' forward calls without the interpreter in between: one C function per route takes the module's tensors,
// checks them, allocates the output and calls the library's C ABI.
//
// What a small call costs is the host, not the kernel: through ctypes, with tensor views and device guards made in
// Python, EOQLinear took 25 us of host time around a 12 us kernel (4096 x 4096, one row) and the seven packed linears
// of a 7B-shape block 160 us around 49 us of kernels.
//
// Activations that are strided or misaligned are copied first, and the activations' device is made current.  Every function
// returns None where anything else is out of the ordinary (a subclass, gradients, autocast or a transform of the call asked
// for, a shape or type the route does not take, no rows): the caller then runs its Python path, which handles those cases and raises their errors.
// An error of a call that was made is raised here.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/add.h>
#include <ATen/ops/constant_pad_nd.h>
#include <ATen/ops/linear.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>
#include <optional>
#include <vector>

#include "../../include/eoq_b200.h"

extern "C" int eoq_b200_linear_packed_preferred(const uint8_t *d_packed, uint32_t rows, uint32_t cols, uint32_t bits, uint32_t group,
                                                const void *x, int x_dtype, uint32_t batch);
struct eoq_b200_symbols;
extern "C" int eoq_b200_symbols_preferred(size_t n, uint64_t block);
extern "C" eoq_b200_symbols *eoq_b200_symbols_stage(const void *symbols, int elem, size_t n, int64_t shift, int clamp, uint32_t alphabet);
extern "C" eoq_error_t eoq_b200_symbols_count(eoq_b200_symbols *s, uint64_t *counts);
extern "C" eoq_error_t eoq_b200_symbols_encode(eoq_b200_symbols *s, const uint32_t *freq, uint32_t alphabet, uint32_t p, uint32_t block, size_t *bytes);
extern "C" eoq_error_t eoq_b200_symbols_fetch(eoq_b200_symbols *s, uint8_t *data, uint32_t *offsets);
extern "C" void eoq_b200_symbols_free(eoq_b200_symbols *s);
extern "C" size_t eoq_b200_symbols_size(const eoq_b200_symbols *s);
extern "C" int eoq_b200_ordered_launches(int on);
extern "C" int eoq_b200_gemv_packed_preferred(uint32_t rows, uint32_t cols, uint32_t bits, uint32_t group);
extern "C" int eoq_b200_weight_linear_preferred(const eoq_b200_weight_t *w, const void *x, int x_dtype, uint32_t batch);

namespace {

using at::Tensor;

// A single row against a large PolarLinear is the CUDA-core kernel's.  GEMV / product in us, blocks of 64 and of 128 columns:
// 1024 x 4096 11.5 / 8.9, 11.2 / 8.6; 4096 x 4096 13.0 / 12.9, 13.0 / 12.0; 3072 x 8192 21.1 / 18.4, 20.9 / 17.5; 5120 x 5120
// 18.5 / 17.9, 18.6 / 17.3; 11008 x 4096 23.4 / 31.3, 23.6 / 28.8; 4096 x 11008 27.1 / 27.8, 26.9 / 26.5; 14336 x 4096
// 30.3 / 34.1, 30.3 / 30.1; 8192 x 8192 34.4 / 36.4, 34.3 / 32.9; 28672 x 8192 100.9 / 139.8, 101.2 / 128.4.  The line costs
// four per cent at worst (8192 x 8192 in blocks of 128).  Two rows take the GEMV twice as long.
constexpr int64_t kPolarSingleRowWeights = 32 << 20;

// Two, and three or four, rows against an entropy-coded weight: the fused GEMV above these many weights, below them the
// decode and the tcgen05 product, whose time is the decoder's and hardly depends on the rows.  Device time, GEMV / product,
// fp16: two rows 1001 x 2048 11.2 / 8.6 us, 2048 x 2048 11.0 / 9.7, 4096 x 4096 14.9 / 17.1; four rows 1001 x 2048
// 24.1 / 8.7, 4096 x 4096 24.1 / 17.2, 11008 x 4096 31.0 / 37.4.  One row: 2048 x 2048 8.3 / 9.6, always the GEMV.
constexpr int64_t kTwoRowWeights = 7 << 20, kFourRowWeights = 28 << 20;

int dtype_code(at::ScalarType t)
{
    return t == at::kHalf ? EOQ_B200_F16 : t == at::kBFloat16 ? EOQ_B200_BF16 : t == at::kFloat ? EOQ_B200_F32 : -1;
}

const Tensor *tensor_of(PyObject *o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

// What torch is to make of a call besides running it: nothing; gradients with respect to one of its tensors; or something that
// only its own operations know how to do (vmap and the other function transforms, forward-mode tangents, tracing, dispatch
// modes, tensors that stand for others).
enum CallKind { kPlain = 0, kGradient = 1, kWatched = 2 };

CallKind kind_of(const Tensor &t)
{
    // a dense CUDA tensor's keys, and nothing else
    static const uint64_t dense = (c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
                                   c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) | c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA)).raw_repr();
    if ((t.key_set().raw_repr() & ~dense) || t._fw_grad(0).defined()) return kWatched;
    return t.requires_grad() && c10::GradMode::is_enabled() ? kGradient : kPlain;
}

bool thread_is_watched()
{
    static const uint64_t always = (c10::DispatchKeySet(c10::DispatchKey::BackendSelect) | c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView)).raw_repr();
    return (c10::impl::tls_local_dispatch_key_set().included_.raw_repr() & ~always) || c10::impl::TorchDispatchModeTLS::any_modes_set();
}

// call_kind(tensor or None, ...): the kind of a call on these tensors, the strongest of all.  (A tensor that is not on a CUDA
// device, or a subclass, says nothing.)
PyObject *call_kind(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    int kind = thread_is_watched() ? kWatched : kPlain;
    for (Py_ssize_t i = 0; i < n; i++)
        if (const Tensor *t = tensor_of(a[i]); t && t->is_cuda()) kind = std::max(kind, (int)kind_of(*t));
    return PyLong_FromLong(kind);
}

// Nothing is going to watch or rewrite this call: the thread's state is the ordinary one, no autocast, x stands for itself.
bool plain_call(const Tensor &x) { return !thread_is_watched() && !at::autocast::is_autocast_enabled(at::kCUDA) && kind_of(x) == kPlain; }

// The activations of one call as the kernels take them: [..., K] of a type they know, contiguous and 16-byte aligned, their
// device current for as long as this lives.
struct Activations {
    const Tensor *x = nullptr;
    int code = -1;
    int64_t rows = 0;
    bool open(PyObject *o, int64_t K)
    {
        const Tensor *t = tensor_of(o);
        if (!t || !t->is_cuda() || t->layout() != at::kStrided || t->dim() < 1 || t->size(-1) != K || K <= 0 || !plain_call(*t)) return false;
        code = dtype_code(t->scalar_type());
        rows = t->numel() / K;
        if (code < 0 || rows < 1 || rows > 0x7fffffff) return false;
        if (t->get_device() != c10::cuda::current_device()) guard.emplace(t->device());
        x = t;
        if (!t->is_contiguous() || (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15u)) {
            at::AutoDispatchBelowADInplaceOrView below;
            held = t->clone(at::MemoryFormat::Contiguous);
            x = &held;
        }
        return true;
    }

  private:
    Tensor held;
    std::optional<c10::cuda::CUDAGuard> guard;
};

bool resident(const Tensor *t, const Tensor &x, at::ScalarType type)
{
    return t && t->is_cuda() && t->get_device() == x.get_device() && t->scalar_type() == type && t->is_contiguous();
}

// A parameter of the module beside x in the type that the kernels read, converted for this call where a cast of the module
// (half(), to(bfloat16), float(), double()) left it in another one: for this call only, since nothing that a copy could be
// kept by says that the parameter has not been written since.
struct Parameter {
    const Tensor *t = nullptr;
    bool converted = false;
    bool open(PyObject *o, const Tensor &x, at::ScalarType type)
    {
        t = tensor_of(o);
        if (!t || !t->is_cuda() || t->get_device() != x.get_device() || t->layout() != at::kStrided || !t->is_floating_point() || kind_of(*t) == kWatched)
            return false;
        if (t->scalar_type() == type && t->is_contiguous()) return true;
        at::AutoDispatchBelowADInplaceOrView below;
        held = t->to(type).contiguous();
        t = &held;
        converted = true;
        return true;
    }

  private:
    Tensor held;
};

// `bias` (None or a vector of N values beside x) as the kernels take it, fp32; false if it is anything else.
struct Bias {
    const float *p = nullptr;
    bool open(PyObject *o, const Tensor &x, int64_t N)
    {
        if (o == Py_None) return true;
        if (!tensor_of(o) || kind_of(*tensor_of(o)) != kPlain || !value.open(o, x, at::kFloat) || value.t->numel() != N) return false;
        p = static_cast<const float *>(value.t->data_ptr());
        return true;
    }

  private:
    Parameter value;
};

// While this lives the library launches its kernels one behind the other: they read scales before the kernel in front of them
// has ended, which may be the one that is writing the converted copy.
struct Ordered {
    explicit Ordered(bool on) : was(on ? eoq_b200_ordered_launches(1) : -1) {}
    ~Ordered() { if (was >= 0) eoq_b200_ordered_launches(was); }
    Ordered(const Ordered &) = delete;
    Ordered &operator=(const Ordered &) = delete;

  private:
    int was;
};

Tensor result(const Tensor &x, int64_t N, at::ScalarType type)
{
    auto sizes = x.sizes();
    if (sizes.size() == 2) return at::detail::empty_cuda({sizes[0], N}, type, x.device(), std::nullopt);
    c10::SmallVector<int64_t, 6> s(sizes.begin(), sizes.end());
    s.back() = N;
    return at::detail::empty_cuda(s, type, x.device(), std::nullopt);
}

void *stream_of(const Tensor &x) { return c10::cuda::getCurrentCUDAStream(x.get_device()).stream(); }

// An error of the library as the exception that the Python path raises for it.  Only "not supported" is the caller's to
// try another route for: a launch that failed would otherwise come back as a slower call, or as garbage later.
PyObject *failed(eoq_error_t rc, const char *where)
{
    if (rc == EOQ_ERR_UNSUPPORTED) Py_RETURN_NONE;
    PyObject *lib = PyImport_ImportModule("eoq_quantization_b200._lib");
    PyObject *r = lib ? PyObject_CallMethod(lib, "check", "is", (int)rc, where) : nullptr;
    Py_XDECREF(lib);
    if (r) {
        Py_DECREF(r);
        PyErr_SetString(PyExc_RuntimeError, where);
    }
    return nullptr;
}

PyObject *done(eoq_error_t rc, Tensor &&y, const char *where)
{
    return rc == EOQ_OK ? THPVariable_Wrap(std::move(y)) : failed(rc, where);
}

// x @ W.T (+ bias) by the library, W written by `fill` into a dense matrix of x's type.  Where rows of a 16-bit y would not
// be 16-byte multiples the matrix gets rows for them to be (whatever those hold ends in columns that are cut off): the
// library's kernels for other widths are three to nine times slower.  fp16, as it is / padded and cut: 4595 x 2056, 26 rows
// 25.5 / 11.5 us, 2048 rows 290 / 46; 1043 x 8888, 64 rows 67.6 / 18.8; 11007 x 4104, one row 36.7 / 19.5.  Not below 2048
// columns of y and 33 rows (1573 x 1336, 8 rows 9.1 / 10.2), nor for fp32 (55 / 60).
template <class Fill>
PyObject *dense_linear(const Tensor &x, int64_t N, int64_t K, int64_t rows, PyObject *bias, Fill &&fill)
{
    const bool pad = x.scalar_type() != at::kFloat && N % 8 && K % 8 == 0 && (rows > 32 || N >= 2048);
    const int64_t wide = pad ? (N + 7) & ~(int64_t)7 : N;
    Tensor dense = at::detail::empty_cuda({wide, K}, x.scalar_type(), x.device(), std::nullopt);
    if (const eoq_error_t rc = fill(dense.data_ptr()); rc != EOQ_OK) return failed(rc, "dequantised copy");
    at::AutoDispatchBelowADInplaceOrView guard;
    std::optional<Tensor> b;
    if (bias != Py_None) b = THPVariable_Unpack(bias).to(x.scalar_type());
    if (!pad) return THPVariable_Wrap(at::linear(x, dense, b));
    if (b) b = at::constant_pad_nd(*b, {0, wide - N});
    return THPVariable_Wrap(at::linear(x, dense, b).narrow(-1, 0, N).contiguous());
}

#define GUARD_BEGIN try {
#define GUARD_END                                                        \
    } catch (const std::exception &e) {                                  \
        PyErr_SetString(PyExc_RuntimeError, e.what());                   \
        return nullptr;                                                  \
    }

// weight_linear(handle, device, N, K, rows16, rows32, x, bias): EOQWeight.linear.  One row, a few against a
// large weight, and up to rows16 (rows32 for fp32) against layouts without a product kernel, by the fused decode + GEMV; more
// by decoding the codes for the tcgen05 product kernel where it takes the layout and is the quicker, else by one decode to a
// dense matrix and a library GEMM.
PyObject *weight_linear(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 8) { PyErr_SetString(PyExc_TypeError, "weight_linear takes 8 arguments"); return nullptr; }
    GUARD_BEGIN
    const int64_t dev = PyLong_AsLongLong(a[1]), N = PyLong_AsLongLong(a[2]), K = PyLong_AsLongLong(a[3]);
    Activations act;
    Bias bias;
    if (!act.open(a[6], K) || act.x->get_device() != dev || !bias.open(a[7], *act.x, N)) Py_RETURN_NONE;
    const Tensor *x = act.x;
    const float *b = bias.p;
    const int code = act.code;
    const int64_t rows = act.rows;
    eoq_b200_weight_t *w = static_cast<eoq_b200_weight_t *>(PyLong_AsVoidPtr(a[0]));
    void *st = stream_of(*x);
    const bool product = rows > 1 && eoq_b200_weight_linear_preferred(w, x->data_ptr(), code, (uint32_t)rows);
    const bool few = product ? rows <= 4 && N * K > (rows == 2 ? kTwoRowWeights : kFourRowWeights)
                             : rows <= PyLong_AsLongLong(a[code == EOQ_B200_F32 ? 5 : 4]);
    if (few) {
        if (rows > 8) Py_RETURN_NONE;
        Tensor y = result(*x, N, x->scalar_type());
        return done(eoq_b200_gemv(w, x->data_ptr(), code, (uint32_t)rows, y.data_ptr(), code, b, st), std::move(y), "eoq_b200_gemv");
    }
    if (product) {
        Tensor y = result(*x, N, x->scalar_type());
        Tensor scratch = at::detail::empty_cuda({(int64_t)eoq_b200_weight_linear_scratch(w, (uint32_t)rows, code)}, at::kByte, x->device(), std::nullopt);
        return done(eoq_b200_weight_linear(w, x->data_ptr(), code, (uint32_t)rows, scratch.data_ptr(), y.data_ptr(), code, b, st), std::move(y), "eoq_b200_weight_linear");
    }
    return dense_linear(*x, N, K, rows, a[7], [&](void *dense) { return eoq_b200_weight_decode(w, nullptr, 0, dense, code, st); });
    GUARD_END
}

// packed_linear(packed, scales, N, K, bits, group, x, bias): QuantizedLinear.forward.  Up to eight rows of 16-bit
// activations against rows of whole 128-column spans by the warp-level tensor-core GEMV where it is quicker than the tcgen05
// kernel, otherwise by that where it takes the shape and is the quicker one, else by a dequantised copy and a library GEMM.
PyObject *packed_linear(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 8) { PyErr_SetString(PyExc_TypeError, "packed_linear takes 8 arguments"); return nullptr; }
    GUARD_BEGIN
    const Tensor *pk = tensor_of(a[0]);
    const int64_t N = PyLong_AsLongLong(a[2]), K = PyLong_AsLongLong(a[3]), bits = PyLong_AsLongLong(a[4]), group = PyLong_AsLongLong(a[5]);
    Activations act;
    Bias bias;
    Parameter sc;
    if (group <= 0 || !act.open(a[6], K) || !bias.open(a[7], *act.x, N) || !sc.open(a[1], *act.x, at::kHalf)) Py_RETURN_NONE;
    const Tensor *x = act.x;
    const float *b = bias.p;
    const Ordered ordered(sc.converted);
    const int code = act.code;
    const int64_t rows = act.rows;
    const at::ScalarType pt = bits == 4 || bits == 2 ? at::kByte : at::kChar;
    const int64_t row_bytes = bits == 4 ? (K + 1) / 2 : bits == 2 ? (K + 3) / 4 : K;
    if (!resident(pk, *x, pt) || pk->numel() != N * row_bytes || sc.t->numel() < (N * K + group - 1) / group)
        Py_RETURN_NONE;
    // two-bit codes in groups below 128 columns against a few fp32 rows stay with the entropy-coded GEMV
    if (bits == 2 && code == EOQ_B200_F32 && rows <= 8 && group % 128 && group % 16 == 0 && K % group == 0) Py_RETURN_NONE;
    void *st = stream_of(*x);
    const uint8_t *codes = static_cast<const uint8_t *>(pk->data_ptr());
    const uint16_t *scales = static_cast<const uint16_t *>(sc.t->data_ptr());
    const bool f32 = code == EOQ_B200_F32, aligned = (reinterpret_cast<uintptr_t>(codes) & 15u) == 0;
    if (rows <= 8 && !f32 && aligned && K % group == 0 && eoq_b200_gemv_packed_preferred((uint32_t)N, (uint32_t)K, (uint32_t)bits, (uint32_t)group)) {
        Tensor y = result(*x, N, x->scalar_type());
        return done(eoq_b200_gemv_packed(codes, scales, (uint32_t)N, (uint32_t)K, (uint32_t)bits, (uint32_t)group, x->data_ptr(), code,
                                         (uint32_t)rows, nullptr, y.data_ptr(), code, b, st),
                    std::move(y), "eoq_b200_gemv_packed");
    }
    if (eoq_b200_linear_packed_preferred(codes, (uint32_t)N, (uint32_t)K, (uint32_t)bits, (uint32_t)group, x->data_ptr(), code, (uint32_t)rows)) {
        Tensor y = result(*x, N, x->scalar_type()), scratch;
        // fp32 activations: room for their two fp16 halves and a factor per row
        if (f32) scratch = at::detail::empty_cuda({rows, K + 1}, at::kFloat, x->device(), std::nullopt);
        return done(eoq_b200_linear_packed(codes, scales, (uint32_t)N, (uint32_t)K, (uint32_t)bits, (uint32_t)group, x->data_ptr(), code,
                                           (uint32_t)rows, f32 ? scratch.data_ptr() : nullptr, y.data_ptr(), code, b, st),
                    std::move(y), "eoq_b200_linear_packed");
    }
    // a few rows against whole groups per row: the entropy-coded form may take them
    if (rows <= 8 && K % 16 == 0 && group % 16 == 0 && K % group == 0) Py_RETURN_NONE;
    return dense_linear(*x, N, K, rows, a[7], [&](void *dense) {
        return eoq_b200_dequant_packed(codes, scales, (uint32_t)N, (uint32_t)K, (uint32_t)bits, (uint32_t)group, 0, (uint32_t)N, dense, code, st);
    });
    GUARD_END
}

// polar_linear(codes, norms, centroids, N, K, bits, block, x, bias): PolarLinear.forward, fp16 results, from the byte codes.
// By the tcgen05 kernel where blocks have 64, 128 or 256 columns, but for a single row against a large weight: that, and few
// rows of other blocks, by the GEMV on the CUDA cores.
PyObject *polar_linear(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 9) { PyErr_SetString(PyExc_TypeError, "polar_linear takes 9 arguments"); return nullptr; }
    GUARD_BEGIN
    const Tensor *cd = tensor_of(a[0]);
    const int64_t N = PyLong_AsLongLong(a[3]), K = PyLong_AsLongLong(a[4]), bits = PyLong_AsLongLong(a[5]), block = PyLong_AsLongLong(a[6]);
    Activations act;
    if (block < 16 || (block & (block - 1)) || K % block || bits < 1 || bits > 8 || !act.open(a[7], K)) Py_RETURN_NONE;
    const Tensor *x = act.x;
    const int code = act.code;
    const int64_t rows = act.rows;
    Parameter nr, ct;
    if (!resident(cd, *x, at::kChar) || !nr.open(a[1], *x, at::kHalf) || !ct.open(a[2], *x, at::kFloat) || cd->numel() < N * K ||
        nr.t->numel() < N * K / block || ct.t->numel() < (1 << bits))
        Py_RETURN_NONE;
    if (kind_of(*tensor_of(a[1])) != kPlain || kind_of(*tensor_of(a[2])) != kPlain) Py_RETURN_NONE;
    // what the kernels read is what the module holds: wider types are rounded for the few rows that always took this route
    if (rows > 32 && (tensor_of(a[1])->element_size() > 2 || tensor_of(a[2])->element_size() > 4)) Py_RETURN_NONE;
    const Ordered ordered(nr.converted || ct.converted);
    // a bias of another type than the result's is added to it, in the type that the two come to
    const Tensor *bias = a[8] == Py_None ? nullptr : tensor_of(a[8]), *after = nullptr;
    if (a[8] != Py_None) {
        if (!bias || !bias->is_cuda() || bias->get_device() != x->get_device() || bias->numel() != N || kind_of(*bias) != kPlain)
            Py_RETURN_NONE;
        if (!resident(bias, *x, at::kHalf)) std::swap(bias, after);
    }
    auto finish = [&](Tensor &&y) {
        if (!after) return THPVariable_Wrap(std::move(y));
        at::AutoDispatchBelowADInplaceOrView below;
        return THPVariable_Wrap(y.add(*after));
    };
    const uint8_t *codes = static_cast<const uint8_t *>(cd->data_ptr());
    const uint16_t *norms = static_cast<const uint16_t *>(nr.t->data_ptr());
    const float *cent = static_cast<const float *>(ct.t->data_ptr());
    Tensor y = result(*x, N, at::kHalf), scratch = at::detail::empty_cuda({rows, K + 1}, at::kFloat, x->device(), std::nullopt);
    if (rows > 1 || N * K < kPolarSingleRowWeights) {
        eoq_error_t rc = eoq_b200_linear_polar_codes(codes, norms, cent, (uint32_t)N, (uint32_t)K, (uint32_t)bits, (uint32_t)block, x->data_ptr(), code,
                                                     (uint32_t)rows, scratch.data_ptr(), y.data_ptr(), EOQ_B200_F16,
                                                     bias ? bias->data_ptr() : nullptr, EOQ_B200_F16, stream_of(*x));
        if (rc == EOQ_OK) return finish(std::move(y));
        if (rc != EOQ_ERR_UNSUPPORTED) return failed(rc, "eoq_b200_linear_polar_codes");
    }
    if (rows > (block >= 64 ? 32 : 8)) Py_RETURN_NONE;
    const eoq_error_t rc = eoq_b200_gemv_polar_codes(codes, norms, cent, (uint32_t)N, (uint32_t)K, (uint32_t)bits, (uint32_t)block, x->data_ptr(), code,
                                                     (uint32_t)rows, scratch.data_ptr(), y.data_ptr(), EOQ_B200_F16, nullptr, -1, stream_of(*x));
    if (rc != EOQ_OK) return failed(rc, "eoq_b200_gemv_polar_codes");
    if (bias) {
        at::AutoDispatchBelowADInplaceOrView below;
        y.add_(*bias);
    }
    return finish(std::move(y));
    GUARD_END
}

// -- codec ---------------------------------------------------------------------

// A C-contiguous buffer for as long as it is in scope.
struct Buffer {
    Py_buffer v;
    bool ok;
    explicit Buffer(PyObject *o, bool writable = false) : ok(PyObject_GetBuffer(o, &v, writable ? PyBUF_CONTIG : PyBUF_CONTIG_RO) == 0) {}
    Buffer(const Buffer &) = delete;
    Buffer &operator=(const Buffer &) = delete;
    ~Buffer() { if (ok) PyBuffer_Release(&v); }
};

PyObject *codec_error(eoq_error_t rc) { return PyLong_FromLong((long)rc); }      // the caller raises EOQError of it

// count_symbols(array, type, shift, clamp, alphabet) -> ([counts], least, greatest) or an error code
PyObject *count_symbols(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 5) { PyErr_SetString(PyExc_TypeError, "count_symbols takes 5 arguments"); return nullptr; }
    GUARD_BEGIN
    Buffer sym(a[0]);
    if (!sym.ok) return nullptr;
    const int type = (int)PyLong_AsLong(a[1]), clamp = (int)PyLong_AsLong(a[3]);
    const int64_t shift = PyLong_AsLongLong(a[2]), alphabet = PyLong_AsLongLong(a[4]);
    if (PyErr_Occurred()) return nullptr;
    if (alphabet < 1 || alphabet > (1 << 20)) return codec_error(EOQ_ERR_UNSUPPORTED);
    std::vector<uint64_t> counts((size_t)alphabet);
    int64_t range[2];
    eoq_error_t rc;
    Py_BEGIN_ALLOW_THREADS
    rc = eoq_b200_count_symbols(sym.v.buf, type, (size_t)(sym.v.len / sym.v.itemsize), shift, clamp, (uint32_t)alphabet, counts.data(), range);
    Py_END_ALLOW_THREADS
    if (rc != EOQ_OK) return codec_error(rc);
    PyObject *list = PyList_New((Py_ssize_t)alphabet);
    if (!list) return nullptr;
    for (int64_t s = 0; s < alphabet; s++) PyList_SET_ITEM(list, s, PyLong_FromUnsignedLongLong(counts[(size_t)s]));
    return Py_BuildValue("NLL", list, (long long)range[0], (long long)range[1]);
    GUARD_END
}

constexpr const char *kStaged = "eoq_b200.symbols";

void free_staged(PyObject *c)
{
    eoq_b200_symbols *s = static_cast<eoq_b200_symbols *>(PyCapsule_GetPointer(c, kStaged));
    Py_BEGIN_ALLOW_THREADS             // may wait for the device
    eoq_b200_symbols_free(s);
    Py_END_ALLOW_THREADS
}

// stage_symbols(array, type, shift, clamp, alphabet, block size or 0) -> (staged, [counts]): the array on the device, for one
// encode_symbols call in front of which it is counted there; or None: count_symbols and encode_symbols take the array.
PyObject *stage_symbols(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 6) { PyErr_SetString(PyExc_TypeError, "stage_symbols takes 6 arguments"); return nullptr; }
    GUARD_BEGIN
    Buffer sym(a[0]);
    if (!sym.ok) return nullptr;
    const int type = (int)PyLong_AsLong(a[1]), clamp = (int)PyLong_AsLong(a[3]);
    const int64_t shift = PyLong_AsLongLong(a[2]), alphabet = PyLong_AsLongLong(a[4]), block = PyLong_AsLongLong(a[5]);
    if (PyErr_Occurred()) return nullptr;
    const size_t count = (size_t)(sym.v.len / sym.v.itemsize);
    if (alphabet < 1 || alphabet > 4096 || block < 0 || (block && !eoq_b200_symbols_preferred(count, (uint64_t)block))) Py_RETURN_NONE;
    eoq_b200_symbols *s = nullptr;
    std::vector<uint64_t> counts((size_t)alphabet);
    eoq_error_t rc = EOQ_OK;
    Py_BEGIN_ALLOW_THREADS
    s = eoq_b200_symbols_stage(sym.v.buf, type, count, shift, clamp, (uint32_t)alphabet);
    if (s) rc = eoq_b200_symbols_count(s, counts.data());
    if (s && rc != EOQ_OK) { eoq_b200_symbols_free(s); s = nullptr; }
    Py_END_ALLOW_THREADS
    if (!s) Py_RETURN_NONE;
    PyObject *staged = PyCapsule_New(s, kStaged, free_staged);
    if (!staged) { eoq_b200_symbols_free(s); return nullptr; }
    PyObject *list = PyList_New((Py_ssize_t)alphabet);
    if (!list) { Py_DECREF(staged); return nullptr; }
    for (int64_t i = 0; i < alphabet; i++) PyList_SET_ITEM(list, i, PyLong_FromUnsignedLongLong(counts[(size_t)i]));
    return Py_BuildValue("NN", staged, list);
    GUARD_END
}

// What encode_symbols encoded, on the host or (staged) on the device, until it has been fetched.
struct Encoded {
    eoq_b200_wire_t *wire = nullptr;
    eoq_b200_symbols *staged = nullptr;
    size_t bytes = 0;
    Encoded() = default;
    Encoded(const Encoded &) = delete;
    Encoded &operator=(const Encoded &) = delete;
    ~Encoded() { if (wire) eoq_b200_wire_take(wire, nullptr, nullptr); }
    eoq_error_t fetch(uint8_t *data, uint32_t *offsets)
    {
        if (staged) return eoq_b200_symbols_fetch(staged, data, offsets);
        eoq_b200_wire_take(wire, data, offsets);
        wire = nullptr;
        return EOQ_OK;
    }
};

// encode_symbols(array, type, shift, clamp, freq, precision, block_size, head, table, staged): with head None (bytes, [offsets]), else the
// container in one piece: head, u32 data size, table, u32 offsets, data; or an error code.
PyObject *encode_symbols(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 10) { PyErr_SetString(PyExc_TypeError, "encode_symbols takes 10 arguments"); return nullptr; }
    GUARD_BEGIN
    Buffer sym(a[0]);
    if (!sym.ok) return nullptr;
    Buffer freq(a[4]);
    if (!freq.ok) return nullptr;
    const int type = (int)PyLong_AsLong(a[1]), clamp = (int)PyLong_AsLong(a[3]);
    const int64_t shift = PyLong_AsLongLong(a[2]), p = PyLong_AsLongLong(a[5]), block = PyLong_AsLongLong(a[6]);
    if (PyErr_Occurred()) return nullptr;
    const int64_t count = sym.v.len / sym.v.itemsize, alphabet = freq.v.len / 4;
    if (count < 1 || count > 0xFFFFFFFFll || block < 1 || block > 0xFFFFFFFFll || p < 1 || p > 16) return codec_error(EOQ_ERR_UNSUPPORTED);
    Encoded w;
    if (a[9] != Py_None) {
        w.staged = static_cast<eoq_b200_symbols *>(PyCapsule_GetPointer(a[9], kStaged));
        if (!w.staged) return nullptr;
        if (eoq_b200_symbols_size(w.staged) != (size_t)count) w.staged = nullptr;      // another array's: as many offsets as that one has blocks
    }
    const int64_t nb = (count + block - 1) / block;
    std::optional<Buffer> head, table;
    size_t at_table = 0, at_offs = 0, at_data = 0;
    if (a[7] != Py_None) {
        head.emplace(a[7]);
        table.emplace(a[8]);
        if (!head->ok || !table->ok) return nullptr;
        at_table = (size_t)head->v.len + 4; at_offs = at_table + (size_t)table->v.len; at_data = at_offs + 4 * (size_t)nb;
    }
    std::vector<uint32_t> offs((size_t)nb);
    // on the device where the symbols are staged, and whatever goes wrong there, on the host, which has all that it takes
    for (;;) {
        eoq_error_t rc;
        Py_BEGIN_ALLOW_THREADS
        rc = w.staged ? eoq_b200_symbols_encode(w.staged, static_cast<const uint32_t *>(freq.v.buf), (uint32_t)alphabet, (uint32_t)p, (uint32_t)block, &w.bytes)
                      : eoq_b200_wire_encode(sym.v.buf, type, (uint32_t)count, shift, clamp, static_cast<const uint32_t *>(freq.v.buf), (uint32_t)alphabet,
                                             (uint32_t)p, (uint32_t)block, &w.wire, &w.bytes);
        Py_END_ALLOW_THREADS
        PyObject *whole = nullptr;                     // the container, or the blocks' bytes alone
        if (rc == EOQ_OK) {
            whole = PyBytes_FromStringAndSize(nullptr, (Py_ssize_t)(at_data + w.bytes));
            if (!whole) return nullptr;
            uint8_t *to = reinterpret_cast<uint8_t *>(PyBytes_AS_STRING(whole));
            Py_BEGIN_ALLOW_THREADS
            rc = w.fetch(to + at_data, offs.data());
            Py_END_ALLOW_THREADS
        }
        if (rc != EOQ_OK) {
            Py_XDECREF(whole);
            if (!w.staged) return codec_error(rc);
            w.staged = nullptr;
            continue;
        }
        if (!head) {
            PyObject *list = PyList_New((Py_ssize_t)nb);
            if (!list) { Py_DECREF(whole); return nullptr; }
            for (int64_t b = 0; b < nb; b++) PyList_SET_ITEM(list, b, PyLong_FromUnsignedLong(offs[(size_t)b]));
            return Py_BuildValue("NN", whole, list);
        }
        // head, data size, table, offsets, data
        uint8_t *to = reinterpret_cast<uint8_t *>(PyBytes_AS_STRING(whole));
        const uint32_t size32 = (uint32_t)w.bytes;
        std::memcpy(to, head->v.buf, (size_t)head->v.len);
        std::memcpy(to + head->v.len, &size32, 4);
        std::memcpy(to + at_table, table->v.buf, (size_t)table->v.len);
        std::memcpy(to + at_offs, offs.data(), 4 * (size_t)nb);
        return whole;
    }
    GUARD_END
}

// decode_symbols(freq, precision, data, offsets (list or u32 buffer), block_size, out, out_type, shift) -> None or an error code
PyObject *decode_symbols(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 8) { PyErr_SetString(PyExc_TypeError, "decode_symbols takes 8 arguments"); return nullptr; }
    GUARD_BEGIN
    Buffer freq(a[0]);
    if (!freq.ok) return nullptr;
    Buffer data(a[2]);
    if (!data.ok) return nullptr;
    Buffer out(a[5], true);
    if (!out.ok) return nullptr;
    const int64_t p = PyLong_AsLongLong(a[1]), block = PyLong_AsLongLong(a[4]), shift = PyLong_AsLongLong(a[7]);
    const int type = (int)PyLong_AsLong(a[6]);
    if (PyErr_Occurred()) return nullptr;
    std::vector<uint32_t> offs;
    if (PyList_CheckExact(a[3])) {
        const Py_ssize_t nb = PyList_GET_SIZE(a[3]);
        offs.resize((size_t)nb);
        for (Py_ssize_t b = 0; b < nb; b++) {
            const int64_t v = PyLong_AsLongLong(PyList_GET_ITEM(a[3], b));
            if (v == -1 && PyErr_Occurred()) return nullptr;
            if (v < 0 || v > 0xFFFFFFFFll) { PyErr_SetString(PyExc_OverflowError, "block offset out of bounds for a 32-bit number"); return nullptr; }
            offs[(size_t)b] = (uint32_t)v;
        }
    } else {
        Buffer o(a[3]);
        if (!o.ok) return nullptr;
        offs.assign(static_cast<const uint32_t *>(o.v.buf), static_cast<const uint32_t *>(o.v.buf) + o.v.len / 4);
    }
    const int64_t count = out.v.len / out.v.itemsize;
    if (count > 0xFFFFFFFFll || block < 1 || block > 0xFFFFFFFFll || p < 1 || p > 16) return codec_error(EOQ_ERR_UNSUPPORTED);
    eoq_error_t rc;
    Py_BEGIN_ALLOW_THREADS
    rc = eoq_b200_decode_blocked_as(static_cast<const uint32_t *>(freq.v.buf), (uint32_t)(freq.v.len / 4), (uint32_t)p,
                                    static_cast<const uint8_t *>(data.v.buf), (size_t)data.v.len, offs.data(), (uint32_t)offs.size(),
                                    (uint32_t)block, (uint32_t)count, out.v.buf, type, shift, nullptr);
    Py_END_ALLOW_THREADS
    if (rc != EOQ_OK) return codec_error(rc);
    Py_RETURN_NONE;
    GUARD_END
}

PyMethodDef methods[] = {
    {"call_kind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_kind)), METH_FASTCALL, nullptr},
    {"count_symbols", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(count_symbols)), METH_FASTCALL, nullptr},
    {"stage_symbols", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(stage_symbols)), METH_FASTCALL, nullptr},
    {"encode_symbols", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(encode_symbols)), METH_FASTCALL, nullptr},
    {"decode_symbols", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(decode_symbols)), METH_FASTCALL, nullptr},
    {"weight_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(weight_linear)), METH_FASTCALL, nullptr},
    {"packed_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(packed_linear)), METH_FASTCALL, nullptr},
    {"polar_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(polar_linear)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
