// The C ABI's per-step calls as functions of a CPython extension module (pulsatrix_b200._native).
//
// A decoding step's GPU work is of the order of ten microseconds, and a call of fourteen arguments through ctypes spends
// half of that on converting them.  Here a call is one vectorcall into C: integers become pointers and sizes, None is a
// null pointer, and where the entry point takes an array of numbers an array is its own address.  The functions return the
// psx_status; binding.py turns it into exceptions.  The library is the one that binding.py has loaded: load(path) looks
// the entry points up there, so that both see the same one.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <dlfcn.h>

#include <cstdint>
#include <tuple>
#include <type_traits>
#include <utility>

#include "psx_b200.h"

namespace {

// The address that a pointer argument stands for.  Handles, streams and settings (T is not a pointer to numbers or to
// psx_row_diag) are integers; a numpy scalar, which has a buffer of its own, is neither an integer nor an array here.
template <class T>
bool address_of(PyObject* o, void** out) {
    if (o == Py_None) {
        *out = nullptr;
        return true;
    }
    if (PyLong_Check(o)) {
        *out = PyLong_AsVoidPtr(o);
        return !PyErr_Occurred();
    }
    if constexpr (std::is_arithmetic_v<std::remove_pointer_t<T>> || std::is_same_v<T, psx_row_diag*>) {
        Py_buffer view;
        if (PyObject_GetBuffer(o, &view, PyBUF_STRIDES) != 0) return false;
        *out = view.buf;  // (the caller's frame keeps the object, and with it the memory, for the length of the call)
        const int dimensions = view.ndim;
        PyBuffer_Release(&view);
        if (dimensions > 0) return true;
    }
    PyErr_Format(PyExc_TypeError, "%s where an address is expected", Py_TYPE(o)->tp_name);
    return false;
}

template <class T>
bool convert(PyObject* o, T* out) {
    if constexpr (std::is_pointer_v<T>) {
        void* p = nullptr;
        if (!address_of<T>(o, &p)) return false;
        *out = reinterpret_cast<T>(p);
    } else if constexpr (std::is_floating_point_v<T>) {
        *out = static_cast<T>(PyFloat_AsDouble(o));
    } else {
        static_assert(std::is_integral_v<T>);
        *out = static_cast<T>(std::is_unsigned_v<T> ? (long long)PyLong_AsUnsignedLongLong(o) : PyLong_AsLongLong(o));
    }
    return !PyErr_Occurred();
}

template <class... A, size_t... I>
PyObject* invoke(psx_status (*fn)(A...), PyObject* const* args, Py_ssize_t count, std::index_sequence<I...>) {
    if (count != (Py_ssize_t)sizeof...(A)) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", (Py_ssize_t)sizeof...(A), count);
        return nullptr;
    }
    if (fn == nullptr) {
        PyErr_SetString(PyExc_RuntimeError, "load() has not been called");
        return nullptr;
    }
    std::tuple<A...> values;
    if (!(convert(args[I], &std::get<I>(values)) && ...)) return nullptr;
    psx_status status;
    Py_BEGIN_ALLOW_THREADS  // (as ctypes does: other threads run while this one enqueues or waits)
    status = fn(std::get<I>(values)...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong((long)status);
}

#define PSX_CALLS(X)                                                                                                     \
    X(sample_rows) X(sample_rows_static) X(sample_rows_host) X(process_logits_host) X(shard_scan) X(shard_merge_rows)   \
    X(exchange_sample) X(top_k_rows) X(lm_head_logits) X(lm_head_sample_rows) X(softmax_rows) X(logsumexp_rows)         \
    X(gather_rows) X(decode_attention)

#define PSX_DEFINE(name)                                                                                         \
    decltype(&psx_b200_##name) g_##name = nullptr;                                                               \
    template <class... A>                                                                                        \
    PyObject* run_##name(psx_status (*fn)(A...), PyObject* const* args, Py_ssize_t count) {                      \
        return invoke(fn, args, count, std::index_sequence_for<A...>{});                                         \
    }                                                                                                            \
    PyObject* call_##name(PyObject*, PyObject* const* args, Py_ssize_t count) { return run_##name(g_##name, args, count); }
PSX_CALLS(PSX_DEFINE)

PyObject* load(PyObject*, PyObject* path) {
    const char* name = PyUnicode_AsUTF8(path);
    if (name == nullptr) return nullptr;
    void* library = dlopen(name, RTLD_NOW | RTLD_LOCAL);  // (already loaded: the same one again)
    if (library == nullptr) {
        PyErr_SetString(PyExc_ImportError, dlerror());
        return nullptr;
    }
#define PSX_LOOK_UP(name) g_##name = reinterpret_cast<decltype(g_##name)>(dlsym(library, "psx_b200_" #name));
    PSX_CALLS(PSX_LOOK_UP)
    Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {
#define PSX_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&call_##name)), METH_FASTCALL, "psx_b200_" #name},
    PSX_CALLS(PSX_METHOD){"load", load, METH_O, "Looks the entry points up in the library at this path."},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "The per-step calls of include/psx_b200.h.", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&g_module); }
