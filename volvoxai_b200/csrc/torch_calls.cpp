// The device-pointer entries as Python calls on torch tensors: the argument handling of w8a8.py's wrappers (row count,
// pointers, row pitches, the output's allocation) in native code.
//
// Why: a linear of a few rows is one or two launches of 2.3 us and 2 .. 6 us of GPU time, and the interpreted wrapper
// around them cost 4.4 us a call (torch.empty from Python 2.3, pointer, pitch and shape look-ups 0.9, the
// foreign-function call 0.7).  The calls are the same entries of libvxb200.so with the same arguments; a call that
// the library declines or fails comes back as its integer code, which w8a8.py turns into the exception.
//
// Nothing is kept between calls.  The GIL is released while the library runs, as ctypes does.  What torch throws (a
// tensor without storage, without a first dimension, an allocation that fails) becomes the Python exception that the
// same attribute or function raises.
#include <Python.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/vxb200_w8a8.h"

namespace {

// The Python and torch of the build, which build.py looks for in the file before the module is loaded.
__attribute__((used)) const char kBuiltFor[] = "built for " VXB_BUILT_FOR;

using at::Tensor;

// Arguments of one call, read left to right; `bad` is set (with a Python error) by the first that does not fit.
struct Args {
    PyObject* const* a;
    Py_ssize_t n, i = 0;
    bool bad = false;
    PyObject* next() {
        if (i >= n) { if (!bad) PyErr_SetString(PyExc_TypeError, "too few arguments"); bad = true; return Py_None; }
        return a[i++];
    }
    long long integer() {
        PyObject* o = next();
        if (bad) return 0;
        const long long v = PyLong_AsLongLong(o);
        if (v == -1 && PyErr_Occurred()) bad = true;
        return v;
    }
    template <typename T> T* handle() { return reinterpret_cast<T*>(static_cast<uintptr_t>(integer())); }
    double number() {
        PyObject* o = next();
        if (bad) return 0;
        const double v = PyFloat_AsDouble(o);
        if (v == -1.0 && PyErr_Occurred()) bad = true;
        return v;
    }
    // null for None where that is allowed
    const Tensor* tensor(bool optional = false) {
        PyObject* o = next();
        if (bad || (optional && o == Py_None)) return nullptr;
        if (!THPVariable_Check(o)) { PyErr_SetString(PyExc_TypeError, "expected a torch tensor"); bad = true; return nullptr; }
        return &THPVariable_Unpack(o);
    }
};

void* at_of(const Tensor* t) { return t ? t->data_ptr() : nullptr; }
uint32_t pitch(const Tensor* t) { return t ? (uint32_t)t->stride(0) : 0u; }

// Runs `call` without the GIL; the tensor on success, the library's code otherwise.
template <typename Make, typename Call> PyObject* result(const Tensor* out, const Make& make, const Call& call) {
    Tensor made;
    if (!out) { made = make(); out = &made; }
    void* y = out->data_ptr();
    const uint32_t ld = out->dim() ? (uint32_t)out->stride(0) : 0u;
    int code;
    Py_BEGIN_ALLOW_THREADS
    code = call(y, ld);
    Py_END_ALLOW_THREADS
    if (code != 1) return PyLong_FromLong(code);
    return THPVariable_Wrap(*out);
}

Tensor matrix(const Tensor& like, int64_t rows, int64_t columns, at::ScalarType type) {
    return at::empty({rows, columns}, like.options().dtype(type).requires_grad(false));
}
Tensor same_shape(const Tensor& like, at::ScalarType type) { return at::empty(like.sizes(), like.options().dtype(type).requires_grad(false)); }
uint32_t byte_type(const Tensor* t) { return t->scalar_type() == at::kByte ? VXB_DTYPE_U8 : VXB_DTYPE_I8; }

// linear_f32(ctx, weight, x, d_out, out | None, route)
PyObject* linear_f32(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a{args, n};
    auto* ctx = a.handle<VxbContext>(); auto* w = a.handle<VxbWeight>();
    const Tensor* x = a.tensor(); const long long d_out = a.integer(); const Tensor* out = a.tensor(true); const int route = (int)a.integer();
    if (a.bad) return nullptr;
    const int64_t rows = x->size(0);
    return result(out, [&] { return matrix(*x, rows, d_out, at::kFloat); },
                  [&, in = at_of(x)](void* y, uint32_t ld) { return vxb_linear_f32(ctx, w, (const float*)in, (uint32_t)rows, (float*)y, ld, route); });
    END_HANDLE_TH_ERRORS
}

// linear_f32_fused(ctx, weight, x, width, out | None, residual | None, silu)
PyObject* linear_f32_fused(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a{args, n};
    auto* ctx = a.handle<VxbContext>(); auto* w = a.handle<VxbWeight>();
    const Tensor* x = a.tensor(); const long long width = a.integer(); const Tensor* out = a.tensor(true);
    const Tensor* res = a.tensor(true); const int silu = (int)a.integer();
    if (a.bad) return nullptr;
    const int64_t rows = x->size(0);
    return result(out, [&] { return matrix(*x, rows, width, at::kFloat); }, [&, in = at_of(x), r = at_of(res), ldr = pitch(res)](void* y, uint32_t ld) {
        return vxb_linear_f32_fused(ctx, w, (const float*)in, (uint32_t)rows, (float*)y, ld, (const float*)r, ldr, silu);
    });
    END_HANDLE_TH_ERRORS
}

// rmsnorm_linear_f32_fused(ctx, weight, x, width, out | None, norm_weight, epsilon, norm_out | None, silu)
PyObject* rmsnorm_linear_f32_fused(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a{args, n};
    auto* ctx = a.handle<VxbContext>(); auto* w = a.handle<VxbWeight>();
    const Tensor* x = a.tensor(); const long long width = a.integer(); const Tensor* out = a.tensor(true);
    const Tensor* g = a.tensor(true); const double eps = a.number(); const Tensor* norm_out = a.tensor(true); const int silu = (int)a.integer();
    if (a.bad) return nullptr;
    const int64_t rows = x->size(0);
    return result(out, [&] { return matrix(*x, rows, width, at::kFloat); }, [&, in = at_of(x), gp = at_of(g), no = at_of(norm_out)](void* y, uint32_t ld) {
        return vxb_rmsnorm_linear_f32_fused(ctx, w, (const float*)in, (const float*)gp, (float)eps, (float*)no, (uint32_t)rows, (float*)y, ld, silu);
    });
    END_HANDLE_TH_ERRORS
}

// linear_i8(ctx, weight, x, d_out, out | None, out_scale, out_zero, route)
PyObject* linear_i8(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a{args, n};
    auto* ctx = a.handle<VxbContext>(); auto* w = a.handle<VxbWeight>();
    const Tensor* x = a.tensor(); const long long d_out = a.integer(); const Tensor* out = a.tensor(true);
    const double scale = a.number(); const long long zero = a.integer(); const int route = (int)a.integer();
    if (a.bad) return nullptr;
    const int64_t rows = x->size(0);
    return result(out, [&] { return matrix(*x, rows, d_out, at::kChar); }, [&, in = at_of(x)](void* y, uint32_t ld) {
        return vxb_linear_i8(ctx, w, (const float*)in, (uint32_t)rows, (float)scale, (int32_t)zero, (int8_t*)y, ld, route);
    });
    END_HANDLE_TH_ERRORS
}

// qlinear_device(ctx, weight, x, d_out, input_scale, input_zero, output_scale, output_zero, out_unsigned, route)
PyObject* qlinear_device(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a{args, n};
    auto* ctx = a.handle<VxbContext>(); auto* w = a.handle<VxbWeight>();
    const Tensor* x = a.tensor(); const long long d_out = a.integer();
    const double is = a.number(); const long long iz = a.integer(); const double os = a.number(); const long long oz = a.integer();
    const bool u8 = a.integer() != 0; const int route = (int)a.integer();
    if (a.bad) return nullptr;
    const int64_t rows = x->size(0);
    return result(nullptr, [&] { return matrix(*x, rows, d_out, u8 ? at::kByte : at::kChar); }, [&, in = at_of(x), dt = byte_type(x)](void* y, uint32_t ld) {
        return vxb_qlinear_device(ctx, w, in, (uint32_t)rows, (float)is, (int32_t)iz, (float)os, (int32_t)oz, dt, u8 ? VXB_DTYPE_U8 : VXB_DTYPE_I8, y, ld, route);
    });
    END_HANDLE_TH_ERRORS
}

// quantize_linear(ctx, x, scale, zero, unsigned)
PyObject* quantize_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a{args, n};
    auto* ctx = a.handle<VxbContext>();
    const Tensor* x = a.tensor(); const double scale = a.number(); const long long zero = a.integer(); const bool u8 = a.integer() != 0;
    if (a.bad) return nullptr;
    return result(nullptr, [&] { return same_shape(*x, u8 ? at::kByte : at::kChar); }, [&, in = at_of(x), count = (uint64_t)x->numel()](void* y, uint32_t) {
        return vxb_quantize_linear_device(ctx, (const float*)in, count, (float)scale, (int32_t)zero, u8 ? VXB_DTYPE_U8 : VXB_DTYPE_I8, y);
    });
    END_HANDLE_TH_ERRORS
}

// dequantize_linear(ctx, x, scale, zero)
PyObject* dequantize_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a{args, n};
    auto* ctx = a.handle<VxbContext>();
    const Tensor* x = a.tensor(); const double scale = a.number(); const long long zero = a.integer();
    if (a.bad) return nullptr;
    return result(nullptr, [&] { return same_shape(*x, at::kFloat); }, [&, in = at_of(x), count = (uint64_t)x->numel(), dt = byte_type(x)](void* y, uint32_t) {
        return vxb_dequantize_linear_device(ctx, in, count, (float)scale, (int32_t)zero, dt, (float*)y);
    });
    END_HANDLE_TH_ERRORS
}

// requantize_linear(ctx, x, input_scale, input_zero, output_scale, output_zero, unsigned)
PyObject* requantize_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a{args, n};
    auto* ctx = a.handle<VxbContext>();
    const Tensor* x = a.tensor();
    const double is = a.number(); const long long iz = a.integer(); const double os = a.number(); const long long oz = a.integer();
    const bool u8 = a.integer() != 0;
    if (a.bad) return nullptr;
    return result(nullptr, [&] { return same_shape(*x, u8 ? at::kByte : at::kChar); }, [&, in = at_of(x), count = (uint64_t)x->numel(), dt = byte_type(x)](void* y, uint32_t) {
        return vxb_requantize_linear_device(ctx, in, count, (float)is, (int32_t)iz, (float)os, (int32_t)oz, dt, u8 ? VXB_DTYPE_U8 : VXB_DTYPE_I8, y);
    });
    END_HANDLE_TH_ERRORS
}

#define VXB_CALL(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {VXB_CALL(linear_f32), VXB_CALL(linear_f32_fused), VXB_CALL(rmsnorm_linear_f32_fused), VXB_CALL(linear_i8),
                          VXB_CALL(qlinear_device), VXB_CALL(quantize_linear), VXB_CALL(dequantize_linear), VXB_CALL(requantize_linear),
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_calls", "Device entries of libvxb200 on torch tensors.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_calls(void) { return PyModule_Create(&kModule); }
