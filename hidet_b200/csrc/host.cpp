// The host side of one call, natively: checks, output allocation, stream and scratch lookup, launch.
//
// At decode sizes a kernel of this library takes 3 to 10 us while the same steps in Python (tensor attribute reads, a
// device context manager, a stream object, two or three ctypes calls) take about 15 us, so an eager program is bound by
// them; here they take about 4 us.  Every function answers None for whatever is not the plain case -- CPU tensors,
// wrong types or shapes, tensors that need a copy first, an active dispatch mode, another current device, scratch that does not exist yet, a
// call that failed -- and the Python function that called it then takes its general path, which checks, copies,
// allocates and reports errors.  So this file decides nothing: it only makes the plain case short.
//
// The library's entry points are given as addresses by bind() (the ctypes binding looks them up), so that one loaded
// copy of the library serves both paths.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <unordered_map>
#include <utility>

#include "../../include/hidet_b200q.h"

namespace {

struct Library {
    decltype(&b200q_symmetric_quantize) quantize = nullptr;
    decltype(&b200q_symmetric_dequantize) dequantize = nullptr;
    decltype(&b200q_embedding_dequantize) take = nullptr;
    decltype(&b200q_qlinear_workspace_bytes) workspace_bytes = nullptr;
    decltype(&b200q_qlinear_f16_i8) linear = nullptr;
    decltype(&b200q_qlinear_f16_i8_fused) linear_fused = nullptr;
    decltype(&b200q_qlinear_f16_u4_workspace_bytes) w4_workspace_bytes = nullptr;
    decltype(&b200q_qlinear_f16_u4) w4 = nullptr;
} lib;

// Scratch buffers that the Python side owns and has told us about, by stream and device.
struct Scratch {
    void *ptr;
    size_t bytes;
};
struct KeyHash {
    size_t operator()(const std::pair<uintptr_t, int> &k) const { return std::hash<uintptr_t>()(k.first) * 31 + (size_t)k.second; }
};
std::unordered_map<std::pair<uintptr_t, int>, Scratch, KeyHash> scratch;  // guarded by the GIL

#define PLAIN_OR_NONE(cond) \
    do {                    \
        if (!(cond)) Py_RETURN_NONE; \
    } while (0)

// A dispatch mode (fake tensors, tracing, counting) wants to see the operators the Python path runs.
inline bool watched() { return c10::impl::TorchDispatchModeTLS::any_modes_set(); }
// A strided CUDA tensor with memory of its own (a vmap or grad wrapper has none) and no Python-level overrides,
// contiguous: what a kernel can be given.
inline bool plain(const at::Tensor &t) {
    return t.is_cuda() && t.layout() == at::kStrided && t.has_storage() && !t.unsafeGetTensorImpl()->is_python_dispatch() &&
           t.is_contiguous() && !t.is_neg();
}
inline const at::Tensor *plain_tensor(PyObject *o) {
    if (!THPVariable_Check(o)) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    return plain(t) ? &t : nullptr;
}

struct Where {
    int device;
    cudaStream_t stream;
};
// The current stream of the tensor's device, if that device is the current one.
inline bool where_is(const at::Tensor &t, Where &w) {
    w.device = t.get_device();
    if (c10::cuda::current_device() != w.device) return false;
    w.stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)w.device).stream();
    return true;
}
inline bool find_scratch(const Where &w, size_t need, void *&ptr, size_t &bytes) {
    ptr = nullptr;
    bytes = 0;
    if (need == 0) return true;
    const auto it = scratch.find({reinterpret_cast<uintptr_t>(w.stream), w.device});
    if (it == scratch.end() || it->second.bytes < need) return false;
    ptr = it->second.ptr;
    bytes = it->second.bytes;
    return true;
}
inline at::Tensor empty(at::IntArrayRef shape, at::ScalarType type, int device) {
    return at::detail::empty_cuda(shape, type, c10::Device(c10::kCUDA, (c10::DeviceIndex)device), c10::nullopt);
}
inline int float_code(at::ScalarType t) { return t == at::kHalf ? B200Q_F16 : t == at::kBFloat16 ? B200Q_BF16 : t == at::kFloat ? B200Q_F32 : -1; }
inline int quant_code(at::ScalarType t) { return t == at::kChar ? B200Q_I8 : t == at::kShort ? B200Q_I16 : -1; }
inline bool is_text(PyObject *o, const char *text) { return PyUnicode_Check(o) && PyUnicode_CompareWithASCIIString(o, text) == 0; }

// dims of a 2-D tensor -> reduce_dim, or -1
inline int reduce_dim_of(PyObject *o) {
    if (!PyLong_CheckExact(o)) return -1;
    const long d = PyLong_AsLong(o);
    return d == 0 || d == -2 ? 0 : d == 1 || d == -1 ? 1 : -1;
}

#define WITHOUT_GIL(status, call) \
    do {                          \
        Py_BEGIN_ALLOW_THREADS status = (call); \
        Py_END_ALLOW_THREADS      \
    } while (0)

// linear(a, weight, scale, weight_layout, out, bias, residual, activation)
PyObject *linear(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    PLAIN_OR_NONE(n_args == 8 && lib.linear != nullptr && !watched());
    const at::Tensor *a = plain_tensor(args[0]), *weight = plain_tensor(args[1]), *scale = plain_tensor(args[2]);
    PLAIN_OR_NONE(a && weight && scale);
    const bool nk = is_text(args[3], "NK");
    PLAIN_OR_NONE(nk || is_text(args[3], "KN"));
    PLAIN_OR_NONE(a->dim() >= 2 && weight->dim() == 2 && scale->dim() == 1);
    PLAIN_OR_NONE(a->scalar_type() == at::kHalf && weight->scalar_type() == at::kChar && scale->scalar_type() == at::kHalf);
    const int64_t k = a->size(-1), m = [&] {
        int64_t p = 1;
        for (int64_t d = 0; d + 1 < a->dim(); ++d) p *= a->size(d);
        return p;
    }();
    const int64_t n = weight->size(nk ? 0 : 1);
    PLAIN_OR_NONE(k == weight->size(nk ? 1 : 0) && n == scale->size(0) && k % 2 == 0 && weight->size(1) % 2 == 0 && m > 0 && n > 0 && k > 0);
    const bool pairs = is_text(args[7], "silu_mul");
    PLAIN_OR_NONE(pairs || args[7] == Py_None);
    const bool fused = pairs || args[5] != Py_None || args[6] != Py_None;
    PLAIN_OR_NONE(!(fused && nk));
    Where w;
    PLAIN_OR_NONE(where_is(*a, w) && weight->get_device() == w.device && scale->get_device() == w.device);
    const int64_t n_out = pairs ? n / 2 : n;
    auto of_result_shape = [&](const at::Tensor *t) {
        if (!t || t->scalar_type() != at::kHalf || t->get_device() != w.device || t->dim() != a->dim() || t->size(-1) != n_out) return false;
        for (int64_t d = 0; d + 1 < a->dim(); ++d)
            if (t->size(d) != a->size(d)) return false;
        return true;
    };
    b200q_epilogue ep = {};
    if (args[5] != Py_None) {
        const at::Tensor *bias = plain_tensor(args[5]);
        PLAIN_OR_NONE(bias && bias->scalar_type() == at::kHalf && bias->get_device() == w.device && bias->dim() == 1 && bias->size(0) == n);
        ep.bias = bias->const_data_ptr();
    }
    if (args[6] != Py_None) {
        const at::Tensor *residual = plain_tensor(args[6]);
        PLAIN_OR_NONE(of_result_shape(residual));
        ep.residual = residual->const_data_ptr();
    }
    ep.ldr = n_out;
    ep.activation = pairs ? B200Q_ACT_SILU_MUL : B200Q_ACT_NONE;
    const int layout = nk ? B200Q_LAYOUT_NK : B200Q_LAYOUT_KN;
    void *ws;
    size_t ws_bytes;
    PLAIN_OR_NONE(find_scratch(w, lib.workspace_bytes(m, n, k, layout), ws, ws_bytes));
    at::Tensor made;
    void *c;
    if (args[4] != Py_None) {
        const at::Tensor *out = plain_tensor(args[4]);
        PLAIN_OR_NONE(of_result_shape(out));
        c = out->data_ptr();
    } else {
        at::DimVector shape(a->sizes());
        shape.back() = n_out;
        made = empty(shape, at::kHalf, w.device);
        c = made.data_ptr();
    }
    int status;
    const void *ap = a->const_data_ptr(), *wp = weight->const_data_ptr(), *sp = scale->const_data_ptr();
    WITHOUT_GIL(status, fused ? lib.linear_fused(ap, wp, sp, c, m, n, k, layout, &ep, ws, ws_bytes, w.stream)
                              : lib.linear(ap, wp, sp, c, m, n, k, layout, ws, ws_bytes, w.stream));
    PLAIN_OR_NONE(status == B200Q_OK);
    if (!made.defined()) return Py_NewRef(args[4]);
    return THPVariable_Wrap(std::move(made));
    END_HANDLE_TH_ERRORS
}

// quantize(w, quant_type, dims) -> (wq, scale)
PyObject *quantize(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    PLAIN_OR_NONE(n_args == 3 && lib.quantize != nullptr && !watched());
    const at::Tensor *x = plain_tensor(args[0]);
    PLAIN_OR_NONE(x && x->dim() == 2 && float_code(x->scalar_type()) >= 0);
    at::ScalarType q;
    if (is_text(args[1], "int8")) q = at::kChar;
    else if (is_text(args[1], "int16")) q = at::kShort;
    else if (THPDtype_Check(args[1])) q = reinterpret_cast<THPDtype *>(args[1])->scalar_type;
    else Py_RETURN_NONE;
    const int reduce = reduce_dim_of(args[2]);
    Where w;
    PLAIN_OR_NONE(quant_code(q) >= 0 && reduce >= 0 && x->numel() > 0 && where_is(*x, w));
    at::Tensor wq = empty(x->sizes(), q, w.device), scale = empty({x->size(reduce == 0 ? 1 : 0)}, x->scalar_type(), w.device);
    int status;
    const void *src = x->const_data_ptr();
    void *codes = wq.data_ptr(), *scales = scale.data_ptr();
    WITHOUT_GIL(status, lib.quantize(src, codes, scales, x->size(0), x->size(1), float_code(x->scalar_type()), quant_code(q), reduce, w.stream));
    PLAIN_OR_NONE(status == B200Q_OK);
    PyObject *first = THPVariable_Wrap(std::move(wq));
    PyObject *second = first ? THPVariable_Wrap(std::move(scale)) : nullptr;
    PyObject *pair = second ? PyTuple_Pack(2, first, second) : nullptr;
    Py_XDECREF(first);
    Py_XDECREF(second);
    return pair;
    END_HANDLE_TH_ERRORS
}

// dequantize(wq, scale, dims)
PyObject *dequantize(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    PLAIN_OR_NONE(n_args == 3 && lib.dequantize != nullptr && !watched());
    const at::Tensor *q = plain_tensor(args[0]), *scale = plain_tensor(args[1]);
    PLAIN_OR_NONE(q && scale && q->dim() == 2 && scale->dim() == 1 && q->numel() > 0);
    const int reduce = reduce_dim_of(args[2]);
    const int fc = float_code(scale->scalar_type()), qc = quant_code(q->scalar_type());
    Where w;
    PLAIN_OR_NONE(reduce >= 0 && fc >= 0 && qc >= 0 && scale->size(0) == q->size(reduce == 0 ? 1 : 0) && where_is(*q, w) && scale->get_device() == w.device);
    at::Tensor out = empty(q->sizes(), scale->scalar_type(), w.device);
    int status;
    const void *codes = q->const_data_ptr(), *scales = scale->const_data_ptr();
    void *dst = out.data_ptr();
    WITHOUT_GIL(status, lib.dequantize(codes, scales, dst, q->size(0), q->size(1), fc, qc, reduce, w.stream));
    PLAIN_OR_NONE(status == B200Q_OK);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// take(wq, scale, indices)
PyObject *take(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    PLAIN_OR_NONE(n_args == 3 && lib.take != nullptr && !watched());
    const at::Tensor *q = plain_tensor(args[0]), *scale = plain_tensor(args[1]), *idx = plain_tensor(args[2]);
    PLAIN_OR_NONE(q && scale && idx && q->dim() == 2 && scale->dim() == 1 && scale->size(0) == q->size(0));
    const int fc = float_code(scale->scalar_type()), qc = quant_code(q->scalar_type());
    const bool wide = idx->scalar_type() == at::kLong;
    Where w;
    PLAIN_OR_NONE(fc >= 0 && qc >= 0 && (wide || idx->scalar_type() == at::kInt) && q->numel() > 0 && idx->numel() > 0 && where_is(*q, w) &&
                  scale->get_device() == w.device && idx->get_device() == w.device);
    at::DimVector shape(idx->sizes());
    shape.push_back(q->size(1));
    at::Tensor out = empty(shape, scale->scalar_type(), w.device);
    int status;
    const void *table = q->const_data_ptr(), *scales = scale->const_data_ptr(), *which = idx->const_data_ptr();
    void *dst = out.data_ptr();
    WITHOUT_GIL(status, lib.take(table, scales, which, dst, q->size(0), q->size(1), idx->numel(), fc, qc, wide ? 8 : 4, w.stream));
    PLAIN_OR_NONE(status == B200Q_OK);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// w4(a, codes, scale, zeros or None, k, n, group_size)
PyObject *w4(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    PLAIN_OR_NONE(n_args == 7 && lib.w4 != nullptr && !watched());
    const at::Tensor *a = plain_tensor(args[0]), *q = plain_tensor(args[1]), *scale = plain_tensor(args[2]);
    PLAIN_OR_NONE(a && q && scale && PyLong_CheckExact(args[4]) && PyLong_CheckExact(args[5]) && PyLong_CheckExact(args[6]));
    const int64_t k = PyLong_AsLongLong(args[4]), n = PyLong_AsLongLong(args[5]), group = PyLong_AsLongLong(args[6]);
    PLAIN_OR_NONE(k > 0 && n > 0 && group > 0);
    PLAIN_OR_NONE(a->dim() == 2 && a->scalar_type() == at::kHalf && a->size(1) == k && a->size(0) > 0);
    PLAIN_OR_NONE(q->dim() == 2 && q->size(0) == k && q->size(1) * (int64_t)q->element_size() * 2 == n);
    auto grouped = [&](const at::Tensor *t) { return t && t->scalar_type() == at::kHalf && t->dim() == 2 && t->size(0) == k / group && t->size(1) == n; };
    Where w;
    PLAIN_OR_NONE(grouped(scale) && where_is(*a, w) && q->get_device() == w.device && scale->get_device() == w.device);
    const void *zp = nullptr;
    if (args[3] != Py_None) {
        const at::Tensor *zeros = plain_tensor(args[3]);
        PLAIN_OR_NONE(grouped(zeros) && zeros->get_device() == w.device);
        zp = zeros->const_data_ptr();
    }
    const int64_t m = a->size(0);
    PLAIN_OR_NONE(group % 16 != 0 || (reinterpret_cast<uintptr_t>(a->const_data_ptr()) & 15u) == 0);  // else the general path aligns it
    void *ws;
    size_t ws_bytes;
    PLAIN_OR_NONE(find_scratch(w, lib.w4_workspace_bytes(m, n, k, group), ws, ws_bytes));
    at::Tensor out = empty({m, n}, at::kHalf, w.device);
    int status;
    const void *ap = a->const_data_ptr(), *codes = q->const_data_ptr(), *sp = scale->const_data_ptr();
    void *dst = out.data_ptr();
    WITHOUT_GIL(status, lib.w4(ap, codes, sp, zp, dst, m, n, k, group, ws, ws_bytes, w.stream));
    PLAIN_OR_NONE(status == B200Q_OK);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// bind(quantize, dequantize, take, workspace_bytes, linear, linear_fused, w4_workspace_bytes, w4): addresses
PyObject *bind(PyObject *, PyObject *args) {
    unsigned long long p[8];
    if (!PyArg_ParseTuple(args, "KKKKKKKK", &p[0], &p[1], &p[2], &p[3], &p[4], &p[5], &p[6], &p[7])) return nullptr;
    lib.quantize = reinterpret_cast<decltype(lib.quantize)>(p[0]);
    lib.dequantize = reinterpret_cast<decltype(lib.dequantize)>(p[1]);
    lib.take = reinterpret_cast<decltype(lib.take)>(p[2]);
    lib.workspace_bytes = reinterpret_cast<decltype(lib.workspace_bytes)>(p[3]);
    lib.linear = reinterpret_cast<decltype(lib.linear)>(p[4]);
    lib.linear_fused = reinterpret_cast<decltype(lib.linear_fused)>(p[5]);
    lib.w4_workspace_bytes = reinterpret_cast<decltype(lib.w4_workspace_bytes)>(p[6]);
    lib.w4 = reinterpret_cast<decltype(lib.w4)>(p[7]);
    Py_RETURN_NONE;
}

// set_scratch(device, stream, address, bytes): the buffer of that stream from now on; 0 bytes: it has none
PyObject *set_scratch(PyObject *, PyObject *args) {
    HANDLE_TH_ERRORS
    int device;
    unsigned long long stream, ptr, bytes;
    if (!PyArg_ParseTuple(args, "iKKK", &device, &stream, &ptr, &bytes)) return nullptr;
    const std::pair<uintptr_t, int> key((uintptr_t)stream, device);
    if (bytes == 0) scratch.erase(key);
    else scratch[key] = {reinterpret_cast<void *>((uintptr_t)ptr), (size_t)bytes};
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

PyObject *clear_scratch(PyObject *, PyObject *) {
    scratch.clear();
    Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(linear),
                         FAST(quantize),
                         FAST(dequantize),
                         FAST(take),
                         FAST(w4),
                         {"bind", bind, METH_VARARGS, nullptr},
                         {"set_scratch", set_scratch, METH_VARARGS, nullptr},
                         {"clear_scratch", clear_scratch, METH_NOARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "hidet_b200_host", "the host side of one call, natively", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_hidet_b200_host() { return PyModule_Create(&module); }
