// The Python mirror's hot calls (hipgpt_b200/launchers.py) as a CPython extension: tensors are looked at and their addresses taken in C++.  Through
// attribute look-ups and ctypes a call of decode attention cost 3.4 us of the host beside the launch's own 2.6, more than the kernel takes
// (2.6 us at B=8 H=8 D=32 ctx=77): 6.2 -> 3.1 us per call, attention at B=2 H=8 S=64 D=32 5.6 -> 4.8 (the kernel 4.4).
// Every function returns the library's status; launchers.py raises.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "hipgpt_attn.h"

namespace {

// launchers._ptr and _ptr_bf16, for what is not exactly a tensor; _int, for what is not an int
PyObject *g_any_ptr = nullptr, *g_any_bf16 = nullptr, *g_any_int = nullptr;

// A contiguous CUDA tensor of `type` (for float32 also None or an address) -> its address; false with an exception set
bool address_of(PyObject *o, at::ScalarType type, void **out)
{
    if (o == Py_None && type == at::kFloat) { *out = nullptr; return true; }
    if (THPVariable_CheckExact(o)) {
        const at::Tensor &t = THPVariable_Unpack(o);
        if (!(t.is_cuda() && t.scalar_type() == type && t.is_contiguous())) {
            PyErr_Format(PyExc_ValueError, "expected a contiguous CUDA %s tensor", type == at::kFloat ? "float32" : "bfloat16");
            return false;
        }
        *out = t.data_ptr();
        return true;
    }
    PyObject *p = PyObject_CallOneArg(type == at::kFloat ? g_any_ptr : g_any_bf16, o);
    if (!p) return false;
    *out = reinterpret_cast<void *>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(p)));
    Py_DECREF(p);
    return !PyErr_Occurred();
}

bool ints(PyObject *const *args, int n, int *out)
{
    for (int i = 0; i < n; ++i) {
        if (PyLong_Check(args[i])) {
            out[i] = static_cast<int>(PyLong_AsUnsignedLongMask(args[i]));
            continue;
        }
        PyObject *x = PyObject_CallOneArg(g_any_int, args[i]);
        if (!x) return false;
        out[i] = static_cast<int>(PyLong_AsUnsignedLongMask(x));
        Py_DECREF(x);
    }
    return !PyErr_Occurred();
}

bool count(Py_ssize_t n, Py_ssize_t want)
{
    if (n != want) PyErr_Format(PyExc_TypeError, "%zd arguments expected, %zd given", want, n);
    return n == want;
}

// The call itself, without the interpreter's lock
template <typename F>
PyObject *status_of(F call)
{
    int rc;
    void *stream = c10::cuda::getCurrentCUDAStream().stream();
    Py_BEGIN_ALLOW_THREADS
    rc = call(stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

PyObject *attention(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    void *p[3];
    int i[5];
    if (!count(n, 8)) return nullptr;
    for (int x = 0; x < 3; ++x) if (!address_of(a[x], at::kFloat, &p[x])) return nullptr;
    if (!ints(a + 3, 5, i)) return nullptr;
    return status_of([&](void *st) {
        return hipgpt_mha_forward_planes(static_cast<const float *>(p[0]), static_cast<float *>(p[1]), static_cast<float *>(p[2]), i[0], i[1], i[2], i[3], i[4], st);
    });
    END_HANDLE_TH_ERRORS
}

PyObject *attention_bf16(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    void *p[2];
    int i[6];
    if (!count(n, 8)) return nullptr;
    for (int x = 0; x < 2; ++x) if (!address_of(a[x], at::kBFloat16, &p[x])) return nullptr;
    if (!ints(a + 2, 6, i)) return nullptr;
    const size_t plane = (size_t)i[0] * i[1] * i[2] * 2;         // bytes
    const char *q = static_cast<const char *>(p[0]);
    return status_of([&](void *st) { return hipgpt_mha_forward_bf16_ex(q, q + plane, q + 2 * plane, p[1], i[0], i[1], i[2], i[3], i[4], i[5], st); });
    END_HANDLE_TH_ERRORS
}

// q, key cache, value cache, out, scratch, bytes of scratch where it is not exactly a tensor, B, H, D, ctx, cap
PyObject *decode(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    void *p[5];
    int i[5];
    if (!count(n, 11)) return nullptr;
    for (int x = 0; x < 5; ++x) if (!address_of(a[x], at::kFloat, &p[x])) return nullptr;
    size_t bytes = 0;
    if (a[5] == Py_None) {
        if (THPVariable_CheckExact(a[4])) bytes = THPVariable_Unpack(a[4]).nbytes();
    } else {
        bytes = PyLong_AsSize_t(a[5]);
        if (PyErr_Occurred()) return nullptr;
    }
    if (!ints(a + 6, 5, i)) return nullptr;
    return status_of([&](void *st) {
        return hipgpt_mha_decode(static_cast<const float *>(p[0]), static_cast<const float *>(p[1]), static_cast<const float *>(p[2]), static_cast<float *>(p[3]),
                                 static_cast<float *>(p[4]), bytes, i[0], i[1], i[2], i[3], i[4], st);
    });
    END_HANDLE_TH_ERRORS
}

PyObject *bind(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (!count(n, 3)) return nullptr;
    Py_XSETREF(g_any_int, Py_NewRef(a[2]));
    Py_XSETREF(g_any_ptr, Py_NewRef(a[0]));
    Py_XSETREF(g_any_bf16, Py_NewRef(a[1]));
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(attention)), METH_FASTCALL, nullptr},
                         {"attention_bf16", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(attention_bf16)), METH_FASTCALL, nullptr},
                         {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(decode)), METH_FASTCALL, nullptr},
                         {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(bind)), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "hipgpt_launch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_hipgpt_launch() { return PyModule_Create(&module); }
