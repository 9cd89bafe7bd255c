// The per-call host path of the Python mirror as a CPython extension (shrew_b200._host).
//
// A small forward or quantize call is a few microseconds of GPU work, so what a caller in a Python loop waits for is the
// host: argument checks, the output allocation, torch's current stream and the call into libshrewq.  Done in
// Python over ctypes that was 11-17 us a call (4096 x 4096, one token; the kernel itself takes 5-6 us); here it is one
// C function per entry point, with the same checks, messages and error class.
//
// Nothing is computed here.  Tensors come from torch's caching allocator on torch's current stream, the library is
// called through addresses that the Python side hands over (bind), so the binding follows whichever build of the
// library ctypes loaded.  The GIL is released around every library call.
//
// The CPU tests build this file with SHREWQ_CPU_EMU: tensors, allocations and device checks are those of the CPU device then.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <ATen/cuda/PeerToPeerAccess.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>
#include <vector>

#include "../../include/shrewq.h"

namespace {

// the library's entry points, by address (bind)
struct Library {
    decltype(&shrewq_ctx_set_stream) set_stream = nullptr;
    decltype(&shrewq_last_error) last_error = nullptr;
    decltype(&shrewq_quantize_f32) quantize_f32 = nullptr;
    decltype(&shrewq_quantize_f32_ex) quantize_f32_ex = nullptr;
    decltype(&shrewq_quantize_any) quantize_any = nullptr;
    decltype(&shrewq_quantize_f32_batch) quantize_f32_batch = nullptr;
    decltype(&shrewq_dequantize_ex) dequantize_ex = nullptr;
    decltype(&shrewq_linear_forward) linear_forward = nullptr;
    decltype(&shrewq_linear_forward_gate_up_silu) gate_up_silu = nullptr;
} L;

PyObject *g_error = nullptr;       // ShrewError(code, message)
PyObject *g_get_context = nullptr; // device index -> context address (creates the context on first use)
constexpr int kMaxDevices = 64;
shrewq_ctx *g_ctx[kMaxDevices] = {nullptr};

struct PythonError {};  // thrown when a Python exception is already set

[[noreturn]] void fail(int code, const std::string &msg) {
    PyObject *e = PyObject_CallFunction(g_error, "is", code, msg.c_str());
    if (e) {
        PyErr_SetObject(g_error, e);
        Py_DECREF(e);
    }
    throw PythonError{};
}

void check(int rc, shrewq_ctx *ctx) {
    if (rc == SHREWQ_OK) return;
    const char *m = L.last_error(ctx);
    fail(rc, m ? m : "");
}

shrewq_ctx *context_of(int device) {
    if (device >= 0 && device < kMaxDevices && g_ctx[device]) return g_ctx[device];
    PyObject *r = PyObject_CallFunction(g_get_context, "i", device);
    if (!r) throw PythonError{};
    void *p = PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    if (!p && PyErr_Occurred()) throw PythonError{};
    if (device >= 0 && device < kMaxDevices) g_ctx[device] = static_cast<shrewq_ctx *>(p);
    return static_cast<shrewq_ctx *>(p);
}

#ifdef SHREWQ_CPU_EMU
bool on_device(const at::Tensor &t) { return t.device().is_cpu(); }
int device_index(const at::Tensor &) { return 0; }
bool peer_access(int, int) { return false; }
void *current_stream(int) { return nullptr; }
at::Tensor empty(at::IntArrayRef shape, at::ScalarType t, int) { return at::empty(shape, at::TensorOptions().dtype(t)); }
#else
bool on_device(const at::Tensor &t) { return t.is_cuda(); }
int device_index(const at::Tensor &t) { return (int)t.get_device(); }
bool peer_access(int from, int to) { return at::cuda::get_p2p_access((c10::DeviceIndex)from, (c10::DeviceIndex)to); }
void *current_stream(int device) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }
at::Tensor empty(at::IntArrayRef shape, at::ScalarType t, int device) {
    return at::Tensor(at::detail::empty_cuda(shape, t, c10::Device(c10::kCUDA, (c10::DeviceIndex)device), std::nullopt));
}
#endif

void bind_stream(shrewq_ctx *ctx, int device) { check(L.set_stream(ctx, current_stream(device)), ctx); }

// forward activations and outputs
int act_code(at::ScalarType t) { return t == at::kFloat ? SHREWQ_F32 : t == at::kBFloat16 ? SHREWQ_BF16 : -1; }
// storage types of quantize / dequantize
int storage_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return SHREWQ_F32;
        case at::kBFloat16: return SHREWQ_BF16;
        case at::kHalf: return SHREWQ_F16;
        case at::kDouble: return SHREWQ_F64;
        default: return -1;
    }
}

std::string dtype_name(at::ScalarType t) {
    PyObject *s = PyObject_Str(reinterpret_cast<PyObject *>(torch::getTHPDtype(t)));
    std::string r = s ? PyUnicode_AsUTF8(s) : "?";
    Py_XDECREF(s);
    return r;
}

std::string shape_text(const at::Tensor &t) {
    std::string r = "[";
    for (int64_t i = 0; i < t.dim(); ++i) r += (i ? ", " : "") + std::to_string(t.size(i));
    return r + "]";
}

const at::Tensor &tensor_arg(PyObject *o, const char *who) {
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s: expected a tensor, got %s", who, Py_TYPE(o)->tp_name);
        throw PythonError{};
    }
    return THPVariable_Unpack(o);
}

PyObject *wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

// every entry point: C++ exceptions (an out-of-memory from torch among them) become Python ones
template <typename F>
PyObject *guarded(F &&f) {
    try {
        return f();
    } catch (const PythonError &) {
        return nullptr;
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
    }
    return nullptr;
}

// ---- a quantized Linear -----------------------------------------------------------------------------------
struct Layer {
    PyObject_HEAD
    shrewq_ctx *ctx;
    shrewq_linear *h;   // owned by the Python QuantizedLinear, which outlives this object's calls
    int device;
    int64_t in_features, out_features;
};

int layer_init(PyObject *self, PyObject *args, PyObject *) {
    Layer *l = reinterpret_cast<Layer *>(self);
    unsigned long long ctx, h;
    long long in, out;
    if (!PyArg_ParseTuple(args, "KKiLL", &ctx, &h, &l->device, &in, &out)) return -1;
    l->ctx = reinterpret_cast<shrewq_ctx *>(ctx);
    l->h = reinterpret_cast<shrewq_linear *>(h);
    l->in_features = in;
    l->out_features = out;
    return 0;
}

extern PyTypeObject LayerType;

// x as the library reads it: contiguous, on the layer's device, of a type it takes.  any_rank: [M, ..., in_features] of
// M * in_features elements will do ([M, 1, in_features], say)
at::Tensor checked_input(const Layer *l, PyObject *o, const char *who, bool any_rank = false) {
    const at::Tensor &x = tensor_arg(o, who);
    if (any_rank && x.dim() > 2 ? x.numel() != x.size(0) * l->in_features : x.dim() != 2 || x.size(1) != l->in_features)
        fail(SHREWQ_ERR_INVALID_ARG, std::string(who) + ": expected x of shape [M," + std::to_string(l->in_features) + "], got " + shape_text(x));
    if (act_code(x.scalar_type()) < 0)
        fail(SHREWQ_ERR_UNSUPPORTED, std::string(who) + ": activation dtype " + dtype_name(x.scalar_type()) + " not supported");
    if (!on_device(x) || device_index(x) != l->device) fail(SHREWQ_ERR_INVALID_ARG, std::string(who) + ": x is not on the layer's device");
    return x.is_contiguous() ? x : x.contiguous();
}

// the caller's output buffer, checked, or a new one; its row stride in ldy
at::Tensor checked_output(const Layer *l, PyObject *out, int64_t M, at::ScalarType type, const char *who, size_t *ldy, bool any_rank = false) {
    if (!out || out == Py_None) {
        *ldy = (size_t)l->out_features;
        if (act_code(type) < 0) fail(SHREWQ_ERR_UNSUPPORTED, std::string(who) + ": output dtype " + dtype_name(type) + " not supported");
        const int64_t shape[2] = {M, l->out_features};
        return empty(shape, type, l->device);
    }
    const at::Tensor &y = tensor_arg(out, who);
    // (another GPU's memory may be written where the two have peer access)
    if (y.numel() > 0 && (!on_device(y) || (device_index(y) != l->device && !peer_access(l->device, device_index(y)))))
        fail(SHREWQ_ERR_INVALID_ARG, std::string(who) + ": the output buffer is not on the layer's device");
    if (any_rank && y.dim() > 2 && y.size(0) == M && y.numel() == M * l->out_features && y.is_contiguous() && act_code(y.scalar_type()) >= 0) {
        *ldy = (size_t)l->out_features;
        return y;
    }
    if (y.dim() != 2 || y.size(0) != M || y.size(1) != l->out_features || (M > 0 && y.stride(1) != 1) || act_code(y.scalar_type()) < 0)
        fail(SHREWQ_ERR_INVALID_ARG, std::string(who) + ": bad output buffer");
    *ldy = (size_t)(M > 1 ? y.stride(0) : std::max(y.stride(0), l->out_features));
    return y;
}

at::ScalarType dtype_arg(PyObject *o, at::ScalarType otherwise, const char *what) {
    if (!o || o == Py_None) return otherwise;
    if (!THPDtype_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s is a torch.dtype, got %s", what, Py_TYPE(o)->tp_name);
        throw PythonError{};
    }
    return reinterpret_cast<THPDtype *>(o)->scalar_type;
}

// forward(x, epilogue, out, out_dtype)
PyObject *layer_forward(PyObject *self, PyObject *const *args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        Layer *l = reinterpret_cast<Layer *>(self);
        if (n != 4) {
            PyErr_SetString(PyExc_TypeError, "forward(x, epilogue, out, out_dtype)");
            throw PythonError{};
        }
        const at::Tensor x = checked_input(l, args[0], "forward");
        const long epilogue = PyLong_AsLong(args[1]);
        if (epilogue == -1 && PyErr_Occurred()) throw PythonError{};
        const int64_t M = x.size(0);
        size_t ldy = 0;
        at::Tensor y = checked_output(l, args[2], M, dtype_arg(args[3], x.scalar_type(), "forward: out_dtype"), "forward", &ldy);
        bind_stream(l->ctx, l->device);
        const int xt = act_code(x.scalar_type()), yt = act_code(y.scalar_type());
        const void *xp = x.data_ptr();
        void *yp = y.data_ptr();
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = L.linear_forward(l->h, xp, xt, (size_t)M, yp, yt, ldy, (int)epilogue);
        Py_END_ALLOW_THREADS
        check(rc, l->ctx);
        if (args[2] != Py_None) {
            Py_INCREF(args[2]);
            return args[2];
        }
        return wrap(std::move(y));
    });
}

// gate_up_silu(up, x, out)
PyObject *layer_gate_up_silu(PyObject *self, PyObject *const *args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        Layer *l = reinterpret_cast<Layer *>(self);
        if (n != 3 || !PyObject_TypeCheck(args[0], &LayerType)) {
            PyErr_SetString(PyExc_TypeError, "gate_up_silu(up, x, out)");
            throw PythonError{};
        }
        const Layer *up = reinterpret_cast<Layer *>(args[0]);
        const at::Tensor x = checked_input(l, args[1], "gate_up_silu", true);
        const int64_t M = x.size(0);
        size_t ldh = 0;
        at::Tensor y = checked_output(l, args[2], M, x.scalar_type(), "gate_up_silu", &ldh, true);
        bind_stream(l->ctx, l->device);
        const int xt = act_code(x.scalar_type()), yt = act_code(y.scalar_type());
        const void *xp = x.data_ptr();
        void *yp = y.data_ptr();
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = L.gate_up_silu(l->h, up->h, xp, xt, (size_t)M, yp, yt, ldh);
        Py_END_ALLOW_THREADS
        check(rc, l->ctx);
        if (args[2] != Py_None) {
            Py_INCREF(args[2]);
            return args[2];
        }
        return wrap(std::move(y));
    });
}

PyMethodDef kLayerMethods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(layer_forward)), METH_FASTCALL, nullptr},
    {"gate_up_silu", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(layer_gate_up_silu)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyTypeObject LayerType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- quantize / dequantize ----------------------------------------------------------------------------------
struct Rows {
    int64_t rows, cols;
};
// rows = shape[0], cols = product(shape[1..]); rank 0 is one element (quantize.rs:276-281)
Rows rows_cols(at::IntArrayRef shape) {
    if (shape.empty()) return {1, 1};
    int64_t cols = 1;
    for (size_t i = 1; i < shape.size(); ++i) cols *= shape[i];
    return {shape[0], cols};
}

PyObject *shape_list(at::IntArrayRef shape) {
    PyObject *l = PyList_New((Py_ssize_t)shape.size());
    for (size_t i = 0; l && i < shape.size(); ++i) PyList_SET_ITEM(l, (Py_ssize_t)i, PyLong_FromLongLong(shape[i]));
    return l;
}

// quantize(tensor, per_channel, bits, asymmetric) -> (codes, scales, zero points or None, shape)
PyObject *quantize(PyObject *, PyObject *const *args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        if (n != 4) {
            PyErr_SetString(PyExc_TypeError, "quantize(tensor, per_channel, bits, asymmetric)");
            throw PythonError{};
        }
        const at::Tensor &t = tensor_arg(args[0], "quantize_tensor");
        const int wt = storage_code(t.scalar_type());
        if (wt < 0) fail(SHREWQ_ERR_UNSUPPORTED, "quantize_tensor: dtype " + dtype_name(t.scalar_type()) + " is not a float storage type");
        const int device = device_index(t);
        shrewq_ctx *ctx = context_of(device);
        const at::Tensor w = t.is_contiguous() ? t : t.contiguous();
        const Rows rc_ = rows_cols(w.sizes());
        const int gran = (args[1] == Py_True && w.dim() > 0) ? SHREWQ_PER_CHANNEL : SHREWQ_PER_TENSOR;
        const long bits = PyLong_AsLong(args[2]);
        const int mode = args[3] == Py_True ? SHREWQ_ASYMMETRIC : SHREWQ_SYMMETRIC;
        const int64_t groups = gran == SHREWQ_PER_CHANNEL ? rc_.rows : 1, total = w.numel();
        at::Tensor q = empty(total, at::kChar, device), scales = empty(groups, at::kDouble, device), zps;
        const bool tuned = wt == SHREWQ_F32 && bits == 8 && mode == SHREWQ_SYMMETRIC;
        if (!tuned) zps = empty(groups, at::kDouble, device);
        bind_stream(ctx, device);
        const void *wp = w.data_ptr();
        int8_t *qp = static_cast<int8_t *>(q.data_ptr());
        double *sp = static_cast<double *>(scales.data_ptr()), *zp = tuned ? nullptr : static_cast<double *>(zps.data_ptr());
        const size_t R = (size_t)rc_.rows, C = (size_t)rc_.cols;
        int rc;
        Py_BEGIN_ALLOW_THREADS
        if (tuned) rc = L.quantize_f32(ctx, static_cast<const float *>(wp), R, C, gran, qp, sp);
        else if (wt == SHREWQ_F32) rc = L.quantize_f32_ex(ctx, static_cast<const float *>(wp), R, C, gran, (int)bits, mode, qp, sp, zp);
        else rc = L.quantize_any(ctx, wp, wt, R, C, gran, (int)bits, mode, qp, sp, zp);
        Py_END_ALLOW_THREADS
        check(rc, ctx);
        PyObject *zo = Py_None;
        if (mode == SHREWQ_ASYMMETRIC) zo = wrap(std::move(zps));
        else Py_INCREF(zo);
        return Py_BuildValue("NNNN", wrap(std::move(q)), wrap(std::move(scales)), zo, shape_list(w.sizes()));
    });
}

// quantize_batch(tensors, per_channel) -> [(codes, scales, shape)]; rank-0 tensors are per-tensor (quantize.rs:276-278)
PyObject *quantize_batch(PyObject *, PyObject *const *args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        if (n != 2) {
            PyErr_SetString(PyExc_TypeError, "quantize_batch(tensors, per_channel)");
            throw PythonError{};
        }
        PyObject *seq = PySequence_Fast(args[0], "quantize_tensors: a sequence of tensors");
        if (!seq) throw PythonError{};
        struct Release {
            PyObject *o;
            ~Release() { Py_DECREF(o); }
        } release{seq};
        const Py_ssize_t count = PySequence_Fast_GET_SIZE(seq);
        const bool per_channel = args[1] == Py_True;
        std::vector<at::Tensor> w, q, s;
        w.reserve(count);
        q.reserve(count);
        s.reserve(count);
        std::vector<shrewq_quant_item> main, single;
        main.reserve(count);
        int device = -1;
        for (Py_ssize_t i = 0; i < count; ++i) {
            const at::Tensor &t = tensor_arg(PySequence_Fast_GET_ITEM(seq, i), "quantize_tensors");
            if (i == 0) device = device_index(t);
            if (t.scalar_type() != at::kFloat || !on_device(t) || device_index(t) != device)
                fail(SHREWQ_ERR_UNSUPPORTED, "quantize_tensors: f32 tensors on one CUDA device");
            w.push_back(t.is_contiguous() ? t : t.contiguous());
            const at::Tensor &c = w.back();
            const Rows rc_ = rows_cols(c.sizes());
            const bool rows_scaled = per_channel && c.dim() > 0;
            q.push_back(empty(c.numel(), at::kChar, device));
            s.push_back(empty(rows_scaled ? rc_.rows : 1, at::kDouble, device));
            (rows_scaled == per_channel ? main : single)
                .push_back({static_cast<const float *>(c.data_ptr()), (size_t)rc_.rows, (size_t)rc_.cols,
                            static_cast<int8_t *>(q.back().data_ptr()), static_cast<double *>(s.back().data_ptr())});
        }
        shrewq_ctx *ctx = context_of(device);
        bind_stream(ctx, device);
        int rc = SHREWQ_OK;
        Py_BEGIN_ALLOW_THREADS
        if (!main.empty()) rc = L.quantize_f32_batch(ctx, main.data(), main.size(), per_channel ? SHREWQ_PER_CHANNEL : SHREWQ_PER_TENSOR);
        if (rc == SHREWQ_OK && !single.empty()) rc = L.quantize_f32_batch(ctx, single.data(), single.size(), SHREWQ_PER_TENSOR);
        Py_END_ALLOW_THREADS
        check(rc, ctx);
        PyObject *out = PyList_New(count);
        if (!out) throw PythonError{};
        for (Py_ssize_t i = 0; i < count; ++i) {
            PyObject *item = Py_BuildValue("NNN", wrap(std::move(q[i])), wrap(std::move(s[i])), shape_list(w[i].sizes()));
            if (!item) {
                Py_DECREF(out);
                throw PythonError{};
            }
            PyList_SET_ITEM(out, i, item);
        }
        return out;
    });
}

// scales or zero points of a dequantize: f64, on the codes' device, one per group
at::Tensor group_values(PyObject *o, int device, int64_t groups, const char *what) {
    const at::Tensor &t = tensor_arg(o, "dequantize_tensor");
    if (groups > 0 && (!on_device(t) || device_index(t) != device || t.scalar_type() != at::kDouble || t.numel() < groups))
        fail(SHREWQ_ERR_INVALID_ARG, std::string("dequantize_tensor: needs ") + std::to_string(groups) + " float64 " + what + " on the codes' device");
    return t.is_contiguous() ? t : t.contiguous();
}

// dequantize(codes, scales, zero points or None, shape, per_channel, dtype) -> tensor
PyObject *dequantize(PyObject *, PyObject *const *args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        if (n != 6) {
            PyErr_SetString(PyExc_TypeError, "dequantize(codes, scales, zero_points, shape, per_channel, dtype)");
            throw PythonError{};
        }
        const at::Tensor &codes = tensor_arg(args[0], "dequantize_tensor");
        const at::ScalarType type = dtype_arg(args[5], at::kFloat, "dequantize_tensor: the target dtype");
        const int ot = storage_code(type);
        if (ot < 0) fail(SHREWQ_ERR_UNSUPPORTED, "dequantize_tensor: target dtype " + dtype_name(type) + " not supported");
        const int device = device_index(codes);
        shrewq_ctx *ctx = context_of(device);
        PyObject *seq = PySequence_Fast(args[3], "dequantize_tensor: shape is a list of sizes");
        if (!seq) throw PythonError{};
        c10::SmallVector<int64_t, 8> shape;
        for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) shape.push_back(PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq, i)));
        Py_DECREF(seq);
        if (PyErr_Occurred()) throw PythonError{};
        const Rows rc_ = rows_cols(shape);
        const int gran = (args[4] == Py_True && !shape.empty()) ? SHREWQ_PER_CHANNEL : SHREWQ_PER_TENSOR;
        const int64_t groups = gran == SHREWQ_PER_CHANNEL ? rc_.rows : 1;
        // every pointer that a kernel follows, before anything is launched
        if (!on_device(codes) || codes.element_size() != 1 || codes.numel() < rc_.rows * rc_.cols)
            fail(SHREWQ_ERR_INVALID_ARG, "dequantize_tensor: needs an i8 code for every element of the shape on a CUDA device");
        const at::Tensor q = codes.is_contiguous() ? codes : codes.contiguous();
        const at::Tensor s = group_values(args[1], device, rc_.rows * rc_.cols > 0 ? groups : 0, "scales");
        const at::Tensor z = args[2] == Py_None ? at::Tensor() : group_values(args[2], device, rc_.rows * rc_.cols > 0 ? groups : 0, "zero points");
        at::Tensor out = empty(shape, type, device);
        bind_stream(ctx, device);
        const int8_t *qp = static_cast<const int8_t *>(q.data_ptr());
        const double *sp = static_cast<const double *>(s.data_ptr());
        const double *zp = z.defined() ? static_cast<const double *>(z.data_ptr()) : nullptr;
        void *op = out.data_ptr();
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = L.dequantize_ex(ctx, qp, sp, zp, (size_t)rc_.rows, (size_t)rc_.cols, gran, ot, op);
        Py_END_ALLOW_THREADS
        check(rc, ctx);
        return wrap(std::move(out));
    });
}

// bind(addresses by name, error class, device index -> context address)
PyObject *bind(PyObject *, PyObject *args) {
    PyObject *table, *error, *get;
    if (!PyArg_ParseTuple(args, "O!OO", &PyDict_Type, &table, &error, &get)) return nullptr;
    struct {
        const char *name;
        void **slot;
    } entries[] = {{"shrewq_ctx_set_stream", reinterpret_cast<void **>(&L.set_stream)},
                   {"shrewq_last_error", reinterpret_cast<void **>(&L.last_error)},
                   {"shrewq_quantize_f32", reinterpret_cast<void **>(&L.quantize_f32)},
                   {"shrewq_quantize_f32_ex", reinterpret_cast<void **>(&L.quantize_f32_ex)},
                   {"shrewq_quantize_any", reinterpret_cast<void **>(&L.quantize_any)},
                   {"shrewq_quantize_f32_batch", reinterpret_cast<void **>(&L.quantize_f32_batch)},
                   {"shrewq_dequantize_ex", reinterpret_cast<void **>(&L.dequantize_ex)},
                   {"shrewq_linear_forward", reinterpret_cast<void **>(&L.linear_forward)},
                   {"shrewq_linear_forward_gate_up_silu", reinterpret_cast<void **>(&L.gate_up_silu)}};
    for (auto &e : entries) {
        PyObject *v = PyDict_GetItemString(table, e.name);
        if (!v) {
            PyErr_Format(PyExc_KeyError, "bind: no address for %s", e.name);
            return nullptr;
        }
        *e.slot = PyLong_AsVoidPtr(v);
        if (!*e.slot) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "bind: %s is NULL", e.name);
    }
    Py_XDECREF(g_error);
    Py_XDECREF(g_get_context);
    Py_INCREF(error);
    Py_INCREF(get);
    g_error = error;
    g_get_context = get;
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"quantize", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(quantize)), METH_FASTCALL, nullptr},
    {"quantize_batch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(quantize_batch)), METH_FASTCALL, nullptr},
    {"dequantize", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(dequantize)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
    LayerType.tp_name = "shrew_b200._host.Layer";
    LayerType.tp_basicsize = sizeof(Layer);
    LayerType.tp_flags = Py_TPFLAGS_DEFAULT;
    LayerType.tp_methods = kLayerMethods;
    LayerType.tp_init = layer_init;
    LayerType.tp_new = PyType_GenericNew;
    if (PyType_Ready(&LayerType) < 0) return nullptr;
    PyObject *m = PyModule_Create(&kModule);
    if (!m) return nullptr;
    Py_INCREF(&LayerType);
    PyModule_AddObject(m, "Layer", reinterpret_cast<PyObject *>(&LayerType));
    return m;
}
