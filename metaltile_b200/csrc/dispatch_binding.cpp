// Python binding of the name-keyed call on host buffers (Context.dispatch_with_grid) over the C ABI of include/mtcuda.h.
//
// Inputs are read where they are (buffer protocol) and outputs are written in place: through ctypes every buffer was copied
// twice.  CPython and libmtcuda.so only - the call needs no PyTorch, which binding.cpp (the typed ops on tensors) does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <new>
#include <string>
#include <vector>

#include "../../include/mtcuda.h"

namespace {

struct PyErr {};                                // a Python exception is set

[[noreturn]] void raise(PyObject *type, const char *msg) {
    PyErr_SetString(type, msg);
    throw PyErr{};
}

PyObject *s_handle = nullptr, *s_check = nullptr;

mtc_ctx *handle_of(PyObject *ctx) {
    PyObject *v = PyObject_GetAttr(ctx, s_handle);
    if (!v) throw PyErr{};
    mtc_ctx *h = v == Py_None ? nullptr : static_cast<mtc_ctx *>(PyLong_AsVoidPtr(v));
    Py_DECREF(v);
    if (PyErr_Occurred()) throw PyErr{};
    return h;
}

void check(PyObject *ctx, int rc) {             // Context._check raises MetalTileError with the context's message
    if (rc == MTC_OK) return;
    PyObject *code = PyLong_FromLong(rc);
    PyObject *r = code ? PyObject_CallMethodOneArg(ctx, s_check, code) : nullptr;
    Py_XDECREF(code);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "mtcuda call failed");
    throw PyErr{};
}

using Args = PyObject *const *;

// dispatch(ctx, kernel, dtype, items, outputs, grid, tpg) -> ({name: bytes}, elapsed_us): mtc_dispatch on host buffers.
// Inputs are read where they are (buffer protocol); every output is a bytes object of its own that starts as a copy of the
// caller's buffer and that the library writes before anybody else can see it.
PyObject *dispatch(Args a, Py_ssize_t n) {
    if (n != 7) raise(PyExc_TypeError, "wrong number of arguments");
    const char *kernel = PyUnicode_AsUTF8(a[1]);
    if (!kernel) throw PyErr{};
    const long dt = PyLong_AsLong(a[2]);
    if (dt == -1 && PyErr_Occurred()) throw PyErr{};
    if (!PyDict_Check(a[3])) raise(PyExc_TypeError, "items must be a dict");
    struct State {
        std::vector<mtc_named_buf> bufs;
        std::vector<Py_buffer> views;
        std::vector<PyObject *> held;
        PyObject *outs = PyDict_New();
        ~State() {
            for (Py_buffer &v : views) PyBuffer_Release(&v);
            for (PyObject *o : held) Py_DECREF(o);
            Py_XDECREF(outs);
        }
    } st;
    if (!st.outs) throw PyErr{};
    const Py_ssize_t count = PyDict_Size(a[3]);
    st.bufs.reserve(count);
    st.views.reserve(count);
    PyObject *key, *val;
    Py_ssize_t pos = 0;
    while (PyDict_Next(a[3], &pos, &key, &val)) {
        mtc_named_buf b{};
        b.name = PyUnicode_AsUTF8(key);
        if (!b.name) throw PyErr{};
        const int is_out = PySequence_Contains(a[4], key);
        if (is_out < 0) throw PyErr{};
        // whatever bytes() takes: a contiguous buffer where it is, anything else (a strided array, a list) as a bytes object
        Py_buffer view;
        if (!PyObject_CheckBuffer(val) || PyObject_GetBuffer(val, &view, PyBUF_C_CONTIGUOUS) != 0) {
            PyErr_Clear();
            val = PyBytes_FromObject(val);
            if (!val) throw PyErr{};
            st.held.push_back(val);
            if (PyObject_GetBuffer(val, &view, PyBUF_SIMPLE) != 0) throw PyErr{};
        }
        st.views.push_back(view);
        b.data = view.buf;
        b.bytes = static_cast<size_t>(view.len);
        b.is_output = is_out;
        if (is_out) {
            PyObject *o = PyBytes_FromStringAndSize(static_cast<const char *>(view.buf), view.len);
            if (!o) throw PyErr{};
            b.data = PyBytes_AS_STRING(o);
            const int rc = PyDict_SetItem(st.outs, key, o);
            Py_DECREF(o);
            if (rc != 0) throw PyErr{};
        }
        st.bufs.push_back(b);
    }
    uint32_t dims[2][3];
    for (int i = 0; i < 2; ++i) {
        PyObject *seq = PySequence_Fast(a[5 + i], "grid_groups and threads_per_group are sequences");
        if (!seq) throw PyErr{};
        // three sizes that int() takes (fewer: the others are 0; they are ignored)
        const Py_ssize_t given = PySequence_Fast_GET_SIZE(seq);
        if (given > 3) PyErr_SetString(PyExc_IndexError, "invalid index");
        for (int j = 0; j < 3 && !PyErr_Occurred(); ++j) {
            PyObject *v = j < given ? PyNumber_Long(PySequence_Fast_GET_ITEM(seq, j)) : nullptr;
            dims[i][j] = v ? static_cast<uint32_t>(PyLong_AsUnsignedLongMask(v)) : 0u;
            Py_XDECREF(v);
        }
        Py_DECREF(seq);
        if (PyErr_Occurred()) throw PyErr{};
    }
    mtc_ctx *h = handle_of(a[0]);
    float us = 0.0f;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = mtc_dispatch(h, kernel, static_cast<int>(dt), st.bufs.data(), static_cast<int>(st.bufs.size()), dims[0], dims[1], &us);
    Py_END_ALLOW_THREADS
    check(a[0], rc);
    PyObject *r = Py_BuildValue("(Od)", st.outs, static_cast<double>(us));
    if (!r) throw PyErr{};
    return r;
}

PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    try {
        return dispatch(args, n);
    } catch (const PyErr &) {
        return nullptr;
    } catch (const std::bad_alloc &) {
        return PyErr_NoMemory();
    }
}

PyMethodDef methods[] = {
    {"dispatch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_dispatch", "the name-keyed call on host buffers over the C ABI of libmtcuda.so", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dispatch() {
    s_handle = PyUnicode_InternFromString("_handle");
    s_check = PyUnicode_InternFromString("_check");
    return s_handle && s_check ? PyModule_Create(&module) : nullptr;
}
