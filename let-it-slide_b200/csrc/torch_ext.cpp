// The layers' forward passes as the interpreter calls them.  The library itself (librptc_b200.so) knows no tensors; what lies
// between a module's `forward` and its entry points -- reading the module's attributes, checks, the result and the
// workspace, device and stream -- cost 12 us of Python and ctypes per call, as much as the kernels of a one-token pass.
// Functions return the result, or the rptc_status of the entry point as an int (the caller raises).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>
#include <optional>
#include <string>
#include <vector>

#include "../../include/rptc_b200.h"

namespace {

// Entry points of the library that the Python side has loaded.
struct {
    decltype(&rptc_linear_workspace_bytes) linear_workspace_bytes;
    decltype(&rptc_linear_forward) linear_forward;
    decltype(&rptc_packed_workspace_bytes) packed_workspace_bytes;
    decltype(&rptc_packed_forward) packed_forward;
    decltype(&rptc_gemv_timed) gemv_timed;
    decltype(&rptc_dequantize) dequantize;
    decltype(&rptc_decompress) decompress;
} g_lib;

#define RPTC_NAMES(X) X(in_features) X(out_features) X(block_in) X(block_out) X(scale) X(fmt) X(_buffers) X(codes) X(lut) X(carry_in) \
    X(signs_in) X(signs_out) X(num_banks) X(bank_blocks) X(L) X(alphabets) X(biases_out) X(biases_in) X(scales_out) X(scales_in) X(bias)
struct Names {
#define RPTC_FIELD(n) PyObject *n;
    RPTC_NAMES(RPTC_FIELD)
} g_names;

struct PyError : std::exception {};      // the interpreter's error is set
[[noreturn]] void fail(const char *what) {
    PyErr_SetString(PyExc_RuntimeError, what);
    throw PyError();
}

// A module's instance attributes and buffers, where they usually lie without the module's __getattr__; what lies elsewhere (a buffer
// that was replaced by a parameter, a property of a subclass) is asked of the module.
class Attributes {
public:
    explicit Attributes(PyObject *module) : module_(module), dict_(PyObject_GenericGetDict(module, nullptr)) {
        if (!dict_) throw PyError();
        buffers_ = get(dict_, g_names._buffers);
    }
    Attributes(const Attributes &) = delete;
    ~Attributes() {
        for (PyObject *o : owned_) Py_DECREF(o);
        Py_XDECREF(dict_);
    }
    PyObject *object(PyObject *name) { return get(dict_, name); }
    int64_t integer(PyObject *name) {
        const long long v = PyLong_AsLongLong(get(dict_, name));
        if (v == -1 && PyErr_Occurred()) throw PyError();
        return v;
    }
    double number(PyObject *name) {
        const double v = PyFloat_AsDouble(get(dict_, name));
        if (v == -1.0 && PyErr_Occurred()) throw PyError();
        return v;
    }
    // A buffer as a kernel reads it: `count` values of `type`, contiguous, and (device_with) on one GPU with the others; null for
    // None where the layer may do without.  (`.half()` and the like change buffers of a module, `.to()` may have been missed.)
    const void *pointer(PyObject *name, at::ScalarType type, int64_t count, bool optional = false) {
        PyObject *o = get(buffers_, name);
        if (o == Py_None && optional) return nullptr;
        if (!THPVariable_Check(o)) refuse(name, "must be a tensor");
        const at::Tensor &t = THPVariable_Unpack(o);
        if (t.scalar_type() != type) refuse(name, (std::string("must have dtype ") + c10::toString(type) + ", got " + c10::toString(t.scalar_type())).c_str());
        if (t.numel() != count) refuse(name, ("must have " + std::to_string(count) + " elements, got " + std::to_string(t.numel())).c_str());
        if (!t.is_contiguous()) refuse(name, "must be contiguous");
        if (held_n_ == sizeof(held_) / sizeof(held_[0])) fail("too many buffers");
        held_[held_n_++] = t;
        if (!device_) device_ = t.device();
        if (!elsewhere_ && (!t.is_cuda() || *device_ != t.device())) elsewhere_ = name;
        return t.data_ptr();
    }
    // The device of all buffers asked for; x has to be there too.
    c10::Device device_with(const at::Tensor &x) const {
        if (elsewhere_) refuse(elsewhere_, "must be a CUDA tensor on the GPU of the layer's other buffers");
        if (!x.is_cuda()) fail("x must be a CUDA tensor");
        if (x.device() != *device_) fail("x is on another GPU than the layer");
        return *device_;
    }

private:
    PyObject *get(PyObject *dict, PyObject *name) {
        PyObject *o = PyDict_GetItemWithError(dict, name);
        if (o) return o;
        if (!PyErr_Occurred()) o = PyObject_GetAttr(module_, name);
        if (!o) throw PyError();
        owned_.push_back(o);
        return o;
    }
    [[noreturn]] static void refuse(PyObject *name, const char *what) {
        const char *n = PyUnicode_AsUTF8(name);
        fail((std::string(n ? n : "a buffer") + " " + what).c_str());
    }
    PyObject *module_, *dict_, *buffers_ = nullptr, *elsewhere_ = nullptr;
    std::vector<PyObject *> owned_;
    at::Tensor held_[7];      // a launch lets other threads run, and they may give the module new buffers
    size_t held_n_ = 0;
    std::optional<c10::Device> device_;
};

const at::Tensor &unpack(PyObject *o, const char *what) {
    if (!THPVariable_Check(o)) fail(what);
    return THPVariable_Unpack(o);
}

rptc_format format_of(PyObject *structure) {      // the ctypes mirror of rptc_format
    rptc_format f;
    Py_buffer view;
    if (PyObject_GetBuffer(structure, &view, PyBUF_SIMPLE)) throw PyError();
    const bool fits = view.len == (Py_ssize_t)sizeof(f);
    if (fits) memcpy(&f, view.buf, sizeof(f));
    PyBuffer_Release(&view);
    if (!fits) fail("fmt is not a Format");
    return f;
}

// The activations as the kernels read them: contiguous, 16-byte aligned.
at::Tensor ready(const at::Tensor &x) {
    at::Tensor t = x.contiguous();
    if (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) t = t.clone(at::MemoryFormat::Contiguous);
    return t;
}

at::Tensor result_like(const at::Tensor &x, int64_t columns) {
    at::DimVector shape(x.sizes());
    shape.back() = columns;
    return at::empty(shape, x.options().requires_grad(false));
}

template <typename F>
PyObject *guarded(F &&f) {
    try {
        return f();
    } catch (const PyError &) {
    } catch (...) {      // torch's own classes: out of memory is torch.OutOfMemoryError here too
        torch::translate_exception_to_python(std::current_exception());
    }
    return nullptr;
}

cudaStream_t current_stream(const at::Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// linear_forward(module, x)
PyObject *linear_forward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 2) fail("linear_forward(module, x)");
        Attributes a(args[0]);
        const at::Tensor &x_in = unpack(args[1], "x must be a tensor");
        rptc_linear l;
        l.m = a.integer(g_names.out_features);
        l.n = a.integer(g_names.in_features);
        l.fmt = format_of(a.object(g_names.fmt));
        if (x_in.dim() < 1 || x_in.size(-1) != l.n || x_in.numel() == 0) fail("x must have in_features columns and at least one row");
        if (l.fmt.L < 1 || l.fmt.L > 16 || l.fmt.S < 0 || l.fmt.S > 16) fail("fmt has no such code");
        l.codes = a.pointer(g_names.codes, at::kInt, l.m * l.n * l.fmt.K / 32);
        l.lut = a.pointer(g_names.lut, at::kHalf, l.fmt.code == RPTC_CODE_LUT ? int64_t(1) << l.fmt.L : int64_t(2) << l.fmt.S);
        l.carry_in = static_cast<const uint32_t *>(a.pointer(g_names.carry_in, at::kInt, l.m, true));
        l.signs_in = a.pointer(g_names.signs_in, at::kHalf, l.n, true);
        l.signs_out = a.pointer(g_names.signs_out, at::kHalf, l.m, true);
        l.block_in = (int32_t)a.integer(g_names.block_in);
        l.block_out = (int32_t)a.integer(g_names.block_out);
        l.scale = (float)a.number(g_names.scale);
        const c10::cuda::OptionalCUDAGuard guard(a.device_with(x_in));
        const at::Tensor x = ready(x_in.scalar_type() == at::kHalf ? x_in : x_in.to(at::kHalf));
        const int64_t rows = x.numel() / l.n;
        at::Tensor y = result_like(x, l.m);
        const int64_t need = g_lib.linear_workspace_bytes(&l, rows);
        at::Tensor ws = at::empty({need > 0 ? need : 1}, x.options().dtype(at::kByte));
        const cudaStream_t s = current_stream(x);
        int status;
        Py_BEGIN_ALLOW_THREADS                                        // a launch waits where the stream's queue is full
        status = g_lib.linear_forward(&l, x.data_ptr(), y.data_ptr(), rows, ws.data_ptr(), need, s);
        Py_END_ALLOW_THREADS
        if (status != RPTC_OK) return PyLong_FromLong(status);
        // beyond 64 rows the product of a layer without transforms leaves the scale to be applied
        if (!l.signs_in && rows > 64 && l.scale != 1.f) y = y * a.number(g_names.scale);
        return THPVariable_Wrap(std::move(y));
    });
}

// packed_forward(module, x)
PyObject *packed_forward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 2) fail("packed_forward(module, x)");
        Attributes a(args[0]);
        const at::Tensor &x_in = unpack(args[1], "x must be a tensor");
        rptc_packed l;
        l.m = a.integer(g_names.out_features);
        l.n = a.integer(g_names.in_features);
        l.banks = (int32_t)a.integer(g_names.num_banks);
        l.bank_blocks = (int32_t)a.integer(g_names.bank_blocks);
        l.L = (int32_t)a.integer(g_names.L);
        if (x_in.dim() < 1 || x_in.size(-1) != l.n) fail("x must have in_features columns");
        if (l.L < 1 || l.L > 16) fail("L must be 1 to 16");
        l.codes = a.pointer(g_names.codes, at::kInt, (int64_t)l.banks * l.bank_blocks * 32 * l.n / 16);
        l.alphabets = a.pointer(g_names.alphabets, at::kHalf, (int64_t)l.banks << l.L);
        l.biases_out = static_cast<const float *>(a.pointer(g_names.biases_out, at::kFloat, l.m));
        l.biases_in = static_cast<const float *>(a.pointer(g_names.biases_in, at::kFloat, l.n));
        l.scales_out = static_cast<const float *>(a.pointer(g_names.scales_out, at::kFloat, l.m));
        l.scales_in = static_cast<const float *>(a.pointer(g_names.scales_in, at::kFloat, l.n));
        l.bias = static_cast<const float *>(a.pointer(g_names.bias, at::kFloat, l.m, true));
        const at::ScalarType type = x_in.scalar_type();
        const int dtype = type == at::kHalf ? 0 : type == at::kBFloat16 ? 1 : 2;
        const c10::cuda::OptionalCUDAGuard guard(a.device_with(x_in));
        const at::Tensor x = ready(dtype == 2 && type != at::kFloat ? x_in.to(at::kFloat) : x_in);
        at::Tensor y = result_like(x, l.m);
        const int64_t tokens = x.numel() / l.n;
        if (tokens > 0) {
            const int64_t most = tokens < 65535 ? tokens : 65535;      // tokens per native call
            const int64_t need = g_lib.packed_workspace_bytes(&l, most);
            if (need < 0) return PyLong_FromLong(RPTC_ERR_SHAPE);
            at::Tensor ws = at::empty({need}, x.options().dtype(at::kByte));
            const char *xp = static_cast<const char *>(x.data_ptr());
            char *yp = static_cast<char *>(y.data_ptr());
            const int64_t width = x.element_size();
            const cudaStream_t s = current_stream(x);
            int status = RPTC_OK;
            Py_BEGIN_ALLOW_THREADS
            for (int64_t t = 0; t < tokens && status == RPTC_OK; t += most)
                status = g_lib.packed_forward(&l, xp + t * l.n * width, dtype, yp + t * l.m * width, most < tokens - t ? most : tokens - t, ws.data_ptr(), need, s);
            Py_END_ALLOW_THREADS
            if (status != RPTC_OK) return PyLong_FromLong(status);
        }
        if (y.scalar_type() != type) y = y.to(type);
        return THPVariable_Wrap(std::move(y));
    });
}

// gemv_timed(codes, lut, x, acc, y, m, n, x_order, accumulate, fmt): milliseconds, or the status
PyObject *gemv_timed(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 10) fail("gemv_timed(codes, lut, x, acc, y, m, n, x_order, accumulate, fmt)");
        const at::Tensor *t[5];
        for (int i = 0; i < 5; ++i) t[i] = &unpack(args[i], "expected a tensor");
        long long v[4];
        for (int i = 0; i < 4; ++i) {
            v[i] = PyLong_AsLongLong(args[5 + i]);
            if (v[i] == -1 && PyErr_Occurred()) throw PyError();
        }
        const rptc_format fmt = format_of(args[9]);
        const c10::cuda::OptionalCUDAGuard guard(t[4]->device());
        const cudaStream_t s = current_stream(*t[4]);
        float ms = 0.f;
        int status;
        Py_BEGIN_ALLOW_THREADS                                        // waits for the result
        status = g_lib.gemv_timed(t[0]->data_ptr(), t[1]->data_ptr(), t[2]->data_ptr(), static_cast<float *>(t[3]->data_ptr()), t[4]->data_ptr(),
                                  v[0], v[1], (int)v[2], (int)v[3], &fmt, &ms, s);
        Py_END_ALLOW_THREADS
        return status == RPTC_OK ? PyFloat_FromDouble(ms) : PyLong_FromLong(status);
    });
}

bool plain(const at::Tensor &t, at::ScalarType type) { return t.is_cuda() && t.scalar_type() == type && t.is_contiguous(); }

// dequantize(alphabet, symbols): symbols to weights, or None for what is not as the kernel reads it (the caller converts it, or refuses it)
PyObject *dequantize(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 2) fail("dequantize(alphabet, symbols)");
        if (!THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) Py_RETURN_NONE;
        const at::Tensor &alphabet = THPVariable_Unpack(args[0]), &symbols = THPVariable_Unpack(args[1]);
        const bool f32 = alphabet.scalar_type() == at::kFloat;
        const int64_t entries = alphabet.numel(), dims = symbols.dim();
        if (!plain(alphabet, f32 ? at::kFloat : at::kHalf) || !plain(symbols, at::kInt) || alphabet.device() != symbols.device() || alphabet.dim() != 1 ||
            entries < 8 || entries > 65536 || (entries & (entries - 1)) || dims < 1 || dims > 2 || symbols.numel() == 0)
            Py_RETURN_NONE;
        const c10::cuda::OptionalCUDAGuard guard(symbols.device());
        at::Tensor out = at::empty(symbols.sizes(), alphabet.options().requires_grad(false));
        int L = 0;
        while ((int64_t(1) << L) < entries) ++L;
        const cudaStream_t s = current_stream(symbols);
        int status;
        Py_BEGIN_ALLOW_THREADS
        status = g_lib.dequantize(alphabet.data_ptr(), static_cast<const int32_t *>(symbols.data_ptr()), out.data_ptr(), f32, dims == 2 ? symbols.size(0) : 1,
                                  symbols.size(-1), L, s);
        Py_END_ALLOW_THREADS
        return status == RPTC_OK ? THPVariable_Wrap(std::move(out)) : PyLong_FromLong(status);
    });
}

// decompress(codes, lut, m, n, fmt, out): 0 when done, None for what is not as the kernel reads it (the caller refuses it)
PyObject *decompress(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 6) fail("decompress(codes, lut, m, n, fmt, out)");
        if (!THPVariable_Check(args[0]) || !THPVariable_Check(args[1]) || !THPVariable_Check(args[5])) Py_RETURN_NONE;
        const at::Tensor &codes = THPVariable_Unpack(args[0]), &lut = THPVariable_Unpack(args[1]), &out = THPVariable_Unpack(args[5]);
        const long long m = PyLong_AsLongLong(args[2]), n = PyLong_AsLongLong(args[3]);
        if (PyErr_Occurred()) throw PyError();
        const rptc_format fmt = format_of(args[4]);
        if (fmt.L < 1 || fmt.L > 16 || fmt.S < 0 || fmt.S > 16 || m <= 0 || n <= 0 || m > (1 << 30) || n > (1 << 30)) Py_RETURN_NONE;
        if (!plain(codes, at::kInt) || !plain(lut, at::kHalf) || codes.device() != lut.device() || codes.device() != out.device() ||
            lut.numel() != (fmt.code == RPTC_CODE_LUT ? int64_t(1) << fmt.L : int64_t(2) << fmt.S) || codes.numel() * 32 != m * n * fmt.K ||
            out.scalar_type() != at::kHalf || out.dim() != 2 || out.size(0) != m || out.size(1) != n || out.stride(1) != 1)
            Py_RETURN_NONE;
        const c10::cuda::OptionalCUDAGuard guard(codes.device());
        const cudaStream_t s = current_stream(codes);
        int status;
        Py_BEGIN_ALLOW_THREADS
        status = g_lib.decompress(codes.data_ptr(), lut.data_ptr(), nullptr, out.data_ptr(), out.stride(0), m, n, &fmt, s);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(status);
    });
}

// bind(linear_workspace_bytes, linear_forward, packed_workspace_bytes, packed_forward, gemv_timed, dequantize, decompress): addresses
PyObject *bind(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 7) fail("bind(seven addresses)");
        void *p[7];
        for (int i = 0; i < 7; ++i) {
            p[i] = PyLong_AsVoidPtr(args[i]);
            if (!p[i]) {
                if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "null address");
                throw PyError();
            }
        }
        g_lib.linear_workspace_bytes = reinterpret_cast<decltype(g_lib.linear_workspace_bytes)>(p[0]);
        g_lib.linear_forward = reinterpret_cast<decltype(g_lib.linear_forward)>(p[1]);
        g_lib.packed_workspace_bytes = reinterpret_cast<decltype(g_lib.packed_workspace_bytes)>(p[2]);
        g_lib.packed_forward = reinterpret_cast<decltype(g_lib.packed_forward)>(p[3]);
        g_lib.gemv_timed = reinterpret_cast<decltype(g_lib.gemv_timed)>(p[4]);
        g_lib.dequantize = reinterpret_cast<decltype(g_lib.dequantize)>(p[5]);
        g_lib.decompress = reinterpret_cast<decltype(g_lib.decompress)>(p[6]);
        Py_RETURN_NONE;
    });
}

#define RPTC_METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {RPTC_METHOD(bind), RPTC_METHOD(linear_forward), RPTC_METHOD(packed_forward), RPTC_METHOD(gemv_timed),
                           RPTC_METHOD(dequantize), RPTC_METHOD(decompress), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
#define RPTC_INTERN(n) \
    g_names.n = PyUnicode_InternFromString(#n); \
    if (!g_names.n) return nullptr;
    RPTC_NAMES(RPTC_INTERN)
    return PyModule_Create(&g_module);
}
