// CPython extension `_host`: the checks and the call of the two hot Python entry points, in native code.
//
// A small GEMM runs in 3.5 to 6.5 us, and the Python boundary around it took 6.5 to 7.3 us of host time, which bounded such
// calls when they follow one another: 1.7 us of attribute reads and comparisons, 1.8 us to convert ten arguments through
// ctypes, the rest interpreter.  This module reads the same attributes of the same objects, and where everything is as the
// hot path wants it, calls the library: 4.2 to 5.4 us, of which the launch is 2.  Where anything is not, it answers "not
// here", and the Python code that it stands in front of runs as ever, with its errors.  (It includes no torch header: it
// reads tensors through their Python attributes.)  The addresses of a MoE layer's expert weights are gathered the same way:
// 64 experts, 96 us of host time for a layer, now 70.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <vector>

namespace {

using RunFn = void (*)(void*, void*, void*, void*, void*, int, int, int, void*, void*);

RunFn g_run = nullptr;
PyObject *g_get_device = nullptr, *g_get_stream = nullptr;
PyObject *g_fp8 = nullptr, *g_f32 = nullptr, *g_bf16 = nullptr, *g_f16 = nullptr;
PyObject *s_is_cuda, *s_is_contiguous, *s_dtype, *s_shape, *s_data_ptr;

// 1 / 0 = the attribute is (is not) `want`; -1 = an exception is set
int attr_is(PyObject* o, PyObject* name, PyObject* want) {
    PyObject* v = PyObject_GetAttr(o, name);
    if (!v) return -1;
    const int r = v == want;
    Py_DECREF(v);
    return r;
}

int contiguous(PyObject* o) {
    PyObject* v = PyObject_CallMethodNoArgs(o, s_is_contiguous);
    if (!v) return -1;
    const int r = v == Py_True;
    Py_DECREF(v);
    return r;
}

// a contiguous CUDA tensor of this type
int hot_tensor(PyObject* o, PyObject* dtype) {
    int r = attr_is(o, s_is_cuda, Py_True);
    if (r == 1) r = attr_is(o, s_dtype, dtype);
    if (r == 1) r = contiguous(o);
    return r;
}

int shape2(PyObject* o, long long* rows, long long* cols) {
    PyObject* v = PyObject_GetAttr(o, s_shape);
    if (!v) return -1;
    int r = 0;
    if (PyTuple_Check(v) && PyTuple_GET_SIZE(v) == 2) {
        *rows = PyLong_AsLongLong(PyTuple_GET_ITEM(v, 0));
        *cols = PyLong_AsLongLong(PyTuple_GET_ITEM(v, 1));
        r = PyErr_Occurred() ? -1 : 1;
    }
    Py_DECREF(v);
    return r;
}

bool data_ptr(PyObject* o, uint64_t* p) {
    PyObject* v = PyObject_CallMethodNoArgs(o, s_data_ptr);
    if (!v) return false;
    *p = PyLong_AsUnsignedLongLong(v);
    Py_DECREF(v);
    return !PyErr_Occurred();
}

// setup(address of `run`, get_device, get_raw_stream, float8_e4m3fn, float32, bfloat16, float16)
PyObject* setup(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 7) {
        PyErr_SetString(PyExc_TypeError, "setup: seven arguments");
        return nullptr;
    }
    const unsigned long long run = PyLong_AsUnsignedLongLong(args[0]);
    if (PyErr_Occurred()) return nullptr;
    PyObject** slots[6] = {&g_get_device, &g_get_stream, &g_fp8, &g_f32, &g_bf16, &g_f16};
    for (int i = 0; i < 6; ++i) {
        Py_INCREF(args[1 + i]);
        Py_XSETREF(*slots[i], args[1 + i]);
    }
    g_run = reinterpret_cast<RunFn>(static_cast<uintptr_t>(run));
    Py_RETURN_NONE;
}

// gemm(a, b, a_scale, b_scale, c) -> True: launched; False: not the hot form, nothing done
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 5 || !g_run) Py_RETURN_FALSE;
    PyObject* const dtypes[5] = {g_fp8, g_fp8, g_f32, g_f32, g_bf16};
    long long rows[5], cols[5];
    for (int i = 0; i < 5; ++i) {
        int r = hot_tensor(args[i], dtypes[i]);
        if (r == 1) r = shape2(args[i], &rows[i], &cols[i]);
        if (r < 0) return nullptr;
        if (r == 0) Py_RETURN_FALSE;
    }
    const long long m = rows[0], k = cols[0], nn = rows[1], kb = k / 128;
    if (cols[1] != k || rows[4] != m || cols[4] != nn || rows[2] != m || cols[2] != kb || rows[3] != (nn + 127) / 128 ||
        cols[3] != kb || m > INT32_MAX || nn > INT32_MAX || k > INT32_MAX)
        Py_RETURN_FALSE;
    uint64_t p[5];
    for (int i = 0; i < 5; ++i)
        if (!data_ptr(args[i], &p[i])) return nullptr;
    PyObject* device = PyObject_CallNoArgs(g_get_device);
    if (!device) return nullptr;
    PyObject* stream = PyObject_CallOneArg(g_get_stream, device);
    Py_DECREF(device);
    if (!stream) return nullptr;
    const unsigned long long s = PyLong_AsUnsignedLongLong(stream);
    Py_DECREF(stream);
    if (PyErr_Occurred()) return nullptr;
    auto ptr = [](unsigned long long v) { return reinterpret_cast<void*>(static_cast<uintptr_t>(v)); };
    Py_BEGIN_ALLOW_THREADS
    g_run(ptr(p[0]), ptr(p[1]), ptr(p[2]), ptr(p[3]), ptr(p[4]), (int)m, (int)nn, (int)k, nullptr, ptr(s));
    Py_END_ALLOW_THREADS
    Py_RETURN_TRUE;
}

// fp16_addresses(weights, names) -> bytes: the 64-bit addresses of weights[name], all of them contiguous CUDA fp16
// tensors; None: not all are
PyObject* fp16_addresses(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2 || !g_run || !PyDict_CheckExact(args[0]) || !PyTuple_CheckExact(args[1])) Py_RETURN_NONE;
    const Py_ssize_t count = PyTuple_GET_SIZE(args[1]);
    std::vector<uint64_t> out((size_t)count);
    for (Py_ssize_t i = 0; i < count; ++i) {
        PyObject* t = PyDict_GetItemWithError(args[0], PyTuple_GET_ITEM(args[1], i));
        if (!t) {
            if (PyErr_Occurred()) return nullptr;
            Py_RETURN_NONE;
        }
        Py_INCREF(t);       // (attribute reads run Python code, which could take it out of the dict)
        const int r = hot_tensor(t, g_f16);
        const bool ok = r == 1 && data_ptr(t, &out[(size_t)i]);
        Py_DECREF(t);
        if (!ok) {
            if (PyErr_Occurred()) return nullptr;
            Py_RETURN_NONE;
        }
    }
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(out.data()), count * (Py_ssize_t)sizeof(uint64_t));
}

template <class F>
PyCFunction fast(F f) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }

PyMethodDef methods[] = {{"setup", fast(setup), METH_FASTCALL, nullptr},
                         {"gemm", fast(gemm), METH_FASTCALL, nullptr},
                         {"fp16_addresses", fast(fp16_addresses), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    s_is_cuda = PyUnicode_InternFromString("is_cuda");
    s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
    s_dtype = PyUnicode_InternFromString("dtype");
    s_shape = PyUnicode_InternFromString("shape");
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    if (!s_is_cuda || !s_is_contiguous || !s_dtype || !s_shape || !s_data_ptr) return nullptr;
    return PyModule_Create(&module);
}
