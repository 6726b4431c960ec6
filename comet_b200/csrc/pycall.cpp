// Calls of the C ABI from Python without ctypes' per-argument objects.
//
// call(address, a0, a1, ...) calls the function at `address` with up to MAX_ARGS integer arguments (sizes, pointers,
// 32-bit options) and returns its 64-bit result (call_i32: its 32-bit result); the interpreter lock is released meanwhile, as ctypes does.  Every
// parameter of the C ABI is an integer or a pointer, and the System V calling convention passes those in 64-bit
// registers and stack slots, a 32-bit one in the lower half, so one template serves all entry points.
// A device call with twelve arguments costs 0.4 us here and 4 us through ctypes (argtypes, c_void_p objects), where the
// kernel it launches runs for 3.6 us (SpMV, 16384 rows of 16 entries).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#include <utility>

namespace {

constexpr int MAX_ARGS = 96;

template <size_t>
using word = int64_t;

template <size_t... I>
int64_t invoke(void *fn, const int64_t *a, std::index_sequence<I...>)
{
    return ((int64_t(*)(word<I>...))fn)(a[I]...);
}

using Invoker = int64_t (*)(void *, const int64_t *);

template <size_t N>
int64_t invoke_n(void *fn, const int64_t *a)
{
    return invoke(fn, a, std::make_index_sequence<N>());
}

template <size_t... N>
const Invoker *table(std::index_sequence<N...>)
{
    static const Invoker t[] = {&invoke_n<N>...};
    return t;
}

template <typename Result>
PyObject *call(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    static const Invoker *by_count = table(std::make_index_sequence<MAX_ARGS + 1>());
    if (n < 1 || n - 1 > MAX_ARGS) {
        PyErr_SetString(PyExc_TypeError, "call: an address and at most 96 integers");
        return nullptr;
    }
    void *fn = PyLong_AsVoidPtr(args[0]);
    if (!fn && PyErr_Occurred()) return nullptr;
    int64_t a[MAX_ARGS + 1];
    for (Py_ssize_t i = 1; i < n; i++) {
        a[i - 1] = PyLong_AsLongLong(args[i]);
        if (a[i - 1] == -1 && PyErr_Occurred()) return nullptr;
    }
    int64_t r;
    Py_BEGIN_ALLOW_THREADS
    r = by_count[n - 1](fn, a);
    Py_END_ALLOW_THREADS
    return PyLong_FromLongLong((Result)r);
}

PyMethodDef methods[] = {
    {"call", (PyCFunction)(void (*)(void))call<int64_t>, METH_FASTCALL, "call(address, *integers) -> 64-bit result"},
    {"call_i32", (PyCFunction)(void (*)(void))call<int32_t>, METH_FASTCALL, "call_i32(address, *integers) -> 32-bit result"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pycall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pycall(void) { return PyModule_Create(&module); }
