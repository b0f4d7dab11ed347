// The per-call work of nart_b200/ops.py: checks of the arguments, the output tensor, the current stream and the
// C-ABI call, without a Python statement or a ctypes conversion between them.  A small convolution runs in
// 5-8 us on the device; the same call through torch.empty (2.4 us), torch.cuda.current_stream (3.2 us), ctypes
// (1 us) and a dozen attribute look-ups took 11.8 us of host time, which bounded every small op.
// The CPython API is used directly; torch owns the memory and names the stream, as in ops.py.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "nart_b200.h"

namespace {

// Raises what nart_b200._lib.check raises for a failed call (its text is per thread, in the library).
PyObject *raise_status(int status)
{
    PyObject *mod = PyImport_ImportModule("nart_b200._lib");
    if (mod) {
        PyObject *r = PyObject_CallMethod(mod, "check", "i", status);
        Py_XDECREF(r);
        Py_DECREF(mod);
    }
    if (!PyErr_Occurred())
        PyErr_Format(PyExc_RuntimeError, "nart_b200 status %d", status);
    return nullptr;
}

// Positional arguments, converted as they are asked for; `ok` turns false (a Python error set) at the first bad one.
struct Args {
    PyObject *const *a;
    Py_ssize_t n, i = 0;
    bool ok = true;
    Args(PyObject *const *args, Py_ssize_t nargs, Py_ssize_t want) : a(args), n(nargs)
    {
        if (n != want) {
            PyErr_Format(PyExc_TypeError, "%zd arguments expected, %zd given", want, n);
            ok = false;
        }
    }
    long long integer()
    {
        if (!ok)
            return 0;
        const long long v = PyLong_AsLongLong(a[i++]);
        if (v == -1 && PyErr_Occurred())
            ok = false;
        return v;
    }
    float real()
    {
        if (!ok)
            return 0.f;
        const double v = PyFloat_AsDouble(a[i++]);
        if (v == -1.0 && PyErr_Occurred())
            ok = false;
        return (float)v;
    }
    bool flag()
    {
        if (!ok)
            return false;
        const int v = PyObject_IsTrue(a[i++]);
        if (v < 0)
            ok = false;
        return v > 0;
    }
    const at::Tensor *tensor(at::ScalarType type, int dims, const char *what)
    {
        if (!ok)
            return nullptr;
        return check_tensor(a[i++], type, dims, what);
    }
    const at::Tensor *check_tensor(PyObject *o, at::ScalarType type, int dims, const char *what)
    {
        if (!THPVariable_Check(o)) {
            PyErr_SetString(PyExc_TypeError, "expected a torch tensor");
            ok = false;
            return nullptr;
        }
        const at::Tensor &t = THPVariable_Unpack(o);
        if (!t.is_cuda() || t.scalar_type() != type || !t.is_contiguous() || (dims && t.dim() != dims)) {
            PyErr_Format(PyExc_ValueError, "expected a contiguous %s CUDA tensor", what);
            ok = false;
            return nullptr;
        }
        return &t;
    }
};

b200_stream_t current_stream() { return reinterpret_cast<b200_stream_t>(c10::cuda::getCurrentCUDAStream().stream()); }

uint8_t *u8(const at::Tensor &t) { return static_cast<uint8_t *>(t.data_ptr()); }

// Runs `call` (a C-ABI call that returns a status) without the GIL and hands `y` to Python.
template <typename F>
PyObject *finish(at::Tensor y, F call)
{
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = call();
    Py_END_ALLOW_THREADS
    return status == B200_OK ? THPVariable_Wrap(std::move(y)) : raise_status(status);
}

// torch reports a failed allocation and the like as C++ exceptions
#define B200_PY_TRY try {
#define B200_PY_CATCH                                             \
    }                                                             \
    catch (const std::exception &e)                               \
    {                                                             \
        PyErr_SetString(PyExc_RuntimeError, e.what());            \
        return nullptr;                                           \
    }

// conv_run(plan, x, signed, h, w, c, oh, ow, k)
PyObject *conv_run(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    B200_PY_TRY
    Args in(args, nargs, 9);
    b200_conv_t *plan = reinterpret_cast<b200_conv_t *>((intptr_t)in.integer());
    PyObject *xo = in.ok ? args[in.i++] : nullptr;
    const bool is_signed = in.flag();
    const at::Tensor *x = in.ok ? in.check_tensor(xo, is_signed ? at::kChar : at::kByte, 0, is_signed ? "int8" : "uint8") : nullptr;
    const int64_t h = in.integer(), w = in.integer(), c = in.integer(), oh = in.integer(), ow = in.integer(), k = in.integer();
    if (!in.ok)
        return nullptr;
    if (x->dim() != 4 || x->size(1) != h || x->size(2) != w || x->size(3) != c) {
        PyErr_SetString(PyExc_ValueError, "the input does not match the prepared plan");
        return nullptr;
    }
    const int64_t n = x->size(0);
    at::Tensor y = at::empty({ n, oh, ow, k }, x->options());
    const uint8_t *xp = u8(*x);
    uint8_t *yp = u8(y);
    b200_stream_t st = current_stream();
    return finish(std::move(y), [=] { return b200_conv2d_run(plan, xp, (int32_t)n, yp, st); });
    B200_PY_CATCH
}

// quantize(x, oalpha, ozp, obits, nhwc, signed)
PyObject *quantize(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    B200_PY_TRY
    Args in(args, nargs, 6);
    const at::Tensor *x = in.tensor(at::kFloat, 4, "float32 NCHW");
    const float oalpha = in.real();
    const uint8_t ozp = (uint8_t)in.integer(), obits = (uint8_t)in.integer();
    const bool nhwc = in.flag(), is_signed = in.flag();
    if (!in.ok)
        return nullptr;
    const int64_t n = x->size(0), c = x->size(1), h = x->size(2), w = x->size(3);
    const auto opt = x->options().dtype(is_signed ? at::kChar : at::kByte);
    at::Tensor y = nhwc ? at::empty({ n, h, w, c }, opt) : at::empty({ n, c, h, w }, opt);
    const float *xp = static_cast<const float *>(x->data_ptr());
    uint8_t *yp = u8(y);
    b200_stream_t st = current_stream();
    return finish(std::move(y), [=] {
        return is_signed ? b200_quantize_s8(xp, reinterpret_cast<int8_t *>(yp), (int32_t)n, (int32_t)c, (int32_t)h, (int32_t)w, oalpha, obits, nhwc, st)
                         : b200_quantize_u8(xp, yp, (int32_t)n, (int32_t)c, (int32_t)h, (int32_t)w, oalpha, ozp, obits, nhwc, st);
    });
    B200_PY_CATCH
}

// dequantize(x, ialpha, izp, nhwc, signed)
PyObject *dequantize(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    B200_PY_TRY
    Args in(args, nargs, 5);
    PyObject *xo = in.ok ? args[in.i++] : nullptr;
    const float ialpha = in.real();
    const uint8_t izp = (uint8_t)in.integer();
    const bool nhwc = in.flag(), is_signed = in.flag();
    const at::Tensor *x = in.ok ? in.check_tensor(xo, is_signed ? at::kChar : at::kByte, 4, is_signed ? "int8" : "uint8") : nullptr;
    if (!in.ok)
        return nullptr;
    const int64_t n = x->size(0), c = x->size(nhwc ? 3 : 1), h = x->size(nhwc ? 1 : 2), w = x->size(nhwc ? 2 : 3);
    at::Tensor y = at::empty({ n, c, h, w }, x->options().dtype(at::kFloat));
    const uint8_t *xp = u8(*x);
    float *yp = static_cast<float *>(y.data_ptr());
    b200_stream_t st = current_stream();
    return finish(std::move(y), [=] {
        return is_signed ? b200_dequantize_s8(reinterpret_cast<const int8_t *>(xp), yp, (int32_t)n, (int32_t)c, (int32_t)h, (int32_t)w, ialpha, nhwc, st)
                         : b200_dequantize_u8(xp, yp, (int32_t)n, (int32_t)c, (int32_t)h, (int32_t)w, ialpha, izp, nhwc, st);
    });
    B200_PY_CATCH
}

// float(o) and int(o), which take more than the plain conversions above: an integral float, a text
float as_float(PyObject *o)
{
    PyObject *f = PyNumber_Float(o);
    const double v = f ? PyFloat_AsDouble(f) : 0.0;
    Py_XDECREF(f);
    return (float)v;
}
uint8_t as_byte(PyObject *o)
{
    PyObject *i = PyNumber_Long(o);
    const unsigned long long v = i ? PyLong_AsUnsignedLongLongMask(i) : 0;
    Py_XDECREF(i);
    return (uint8_t)v;
}

// eltwise_sum(xs, ialpha, izp, coeff or None, oalpha, ozp, obits, relu); the first four are lists of one length (zero points
// that are not given are 0)
PyObject *eltwise_sum(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    B200_PY_TRY
    Args in(args, nargs, 8);
    if (!in.ok)
        return nullptr;
    constexpr Py_ssize_t kMost = 64;      // the library declines more than four with a message of its own
    PyObject *lists[4] = { args[0], args[1], args[2], args[3] };
    const bool has_coeff = lists[3] != Py_None;
    Py_ssize_t n = PyList_Check(lists[0]) ? PyList_GET_SIZE(lists[0]) : 0, n_zp = PyList_Check(lists[2]) ? PyList_GET_SIZE(lists[2]) : -1;
    for (int l = 0; l < (has_coeff ? 4 : 3); ++l)
        if (!PyList_Check(lists[l]) || (l != 2 && PyList_GET_SIZE(lists[l]) != n) || n_zp > n || n < 1 || n > kMost) {
            PyErr_SetString(PyExc_ValueError, "eltwise: inputs, scales, zero points and coefficients must have one length");
            return nullptr;
        }
    in.i = 4;
    const float oalpha = in.real();
    const uint8_t ozp = (uint8_t)in.integer(), obits = (uint8_t)in.integer();
    const bool relu = in.flag();
    const uint8_t *xs[kMost];
    float ia[kMost], cf[kMost];
    uint8_t iz[kMost];
    const at::Tensor *first = nullptr;
    for (Py_ssize_t i = 0; i < n && in.ok; ++i) {
        const at::Tensor *t = in.check_tensor(PyList_GET_ITEM(lists[0], i), at::kByte, 0, "uint8");
        if (!t)
            return nullptr;
        if (!first)
            first = t;
        // the kernel reads as many bytes of every input as the first one has
        if (t->numel() < first->numel() || t->device() != first->device()) {
            PyErr_SetString(PyExc_ValueError, "eltwise: an input is smaller than the first one, or on another device");
            return nullptr;
        }
        xs[i] = u8(*t);
        ia[i] = as_float(PyList_GET_ITEM(lists[1], i));
        iz[i] = i < n_zp ? as_byte(PyList_GET_ITEM(lists[2], i)) : 0;
        cf[i] = has_coeff ? as_float(PyList_GET_ITEM(lists[3], i)) : 1.0f;
        if (PyErr_Occurred())
            return nullptr;
    }
    if (!in.ok)
        return nullptr;
    at::Tensor y = at::empty(first->sizes(), first->options());
    uint8_t *yp = u8(y);
    const size_t count = (size_t)first->numel();
    b200_stream_t st = current_stream();
    return finish(std::move(y), [&, yp, count, st] {
        return b200_eltwise_sum_u8(xs, (int32_t)n, count, ia, iz, has_coeff ? cf : nullptr, oalpha, ozp, obits, relu, yp, st);
    });
    B200_PY_CATCH
}

// relu(x, ialpha, izp, oalpha, ozp, obits)
PyObject *relu(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    B200_PY_TRY
    Args in(args, nargs, 6);
    const at::Tensor *x = in.tensor(at::kByte, 0, "uint8");
    const float ialpha = in.real();
    const uint8_t izp = (uint8_t)in.integer();
    const float oalpha = in.real();
    const uint8_t ozp = (uint8_t)in.integer(), obits = (uint8_t)in.integer();
    if (!in.ok)
        return nullptr;
    at::Tensor y = at::empty(x->sizes(), x->options());
    const uint8_t *xp = u8(*x);
    uint8_t *yp = u8(y);
    const size_t count = (size_t)x->numel();
    b200_stream_t st = current_stream();
    return finish(std::move(y), [=] { return b200_relu_u8(xp, count, ialpha, izp, oalpha, ozp, obits, yp, st); });
    B200_PY_CATCH
}

// pool(x, method, kernel_h, kernel_w, pad_h, pad_w, stride_h, stride_w, ceil_mode, ialpha, izp, oalpha, ozp, obits)
PyObject *pool(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    B200_PY_TRY
    Args in(args, nargs, 14);
    const at::Tensor *x = in.tensor(at::kByte, 4, "uint8");
    int32_t v[8];
    for (int32_t &e : v)
        e = (int32_t)in.integer();
    const float ialpha = in.real();
    const uint8_t izp = (uint8_t)in.integer();
    const float oalpha = in.real();
    const uint8_t ozp = (uint8_t)in.integer(), obits = (uint8_t)in.integer();
    if (!in.ok)
        return nullptr;
    const int32_t n = (int32_t)x->size(0), h = (int32_t)x->size(1), w = (int32_t)x->size(2), c = (int32_t)x->size(3);
    int32_t oh = 0, ow = 0;
    const int rc = b200_pool_out_dims(h, w, v[1], v[2], v[3], v[4], v[5], v[6], v[7], &oh, &ow);
    if (rc != B200_OK)
        return raise_status(rc);
    if (oh < 0 || ow < 0) {
        PyErr_SetString(PyExc_RuntimeError, "pool: the window does not fit the input");
        return nullptr;
    }
    at::Tensor y = at::empty({ n, oh, ow, c }, x->options());
    const uint8_t *xp = u8(*x);
    uint8_t *yp = u8(y);
    b200_stream_t st = current_stream();
    return finish(std::move(y), [=] {
        return b200_pool_u8(xp, n, c, h, w, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], ialpha, izp, oalpha, ozp, obits, yp, st);
    });
    B200_PY_CATCH
}

#define B200_PY_METHOD(name) { #name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr }
PyMethodDef kMethods[] = { B200_PY_METHOD(conv_run), B200_PY_METHOD(quantize), B200_PY_METHOD(dequantize),
                           B200_PY_METHOD(eltwise_sum), B200_PY_METHOD(relu), B200_PY_METHOD(pool), { nullptr, nullptr, 0, nullptr } };
PyModuleDef kModule = { PyModuleDef_HEAD_INIT, "_py_ops", "Native call path of nart_b200.ops.", -1, kMethods, nullptr, nullptr, nullptr, nullptr };

}  // namespace

PyMODINIT_FUNC PyInit__py_ops(void) { return PyModule_Create(&kModule); }
