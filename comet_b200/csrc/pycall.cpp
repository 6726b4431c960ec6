// Calls of the C ABI from Python without ctypes' per-argument objects.
//
// call(address, a0, a1, ...) calls the function at `address` with up to MAX_ARGS integer arguments (sizes, pointers,
// 32-bit options) and returns its 64-bit result (call_i32: its 32-bit result); the interpreter lock is released meanwhile, as ctypes does.  Every
// parameter of the C ABI is an integer or a pointer, and the conventions of Linux hosts (System V on x86-64, AAPCS64 on Arm) pass
// those in 64-bit registers and stack slots, a 32-bit one in the lower half, so one template serves all entry points.
// A device call with twelve arguments costs 0.4 us here and 4 us through ctypes (argtypes, c_void_p objects), where the
// kernel it launches runs for 3.6 us (SpMV, 16384 rows of 16 entries).
//
// new_result(alloc, size, free, dtype, dims) makes a numpy array in a block of a memory pool that owns the block as any new
// array owns its memory (it can be resized in place, and gives the block back when it goes), through numpy's
// data-memory handlers; None where the pool has no block.  The pool is three functions, given by their addresses:
// void *alloc(int64_t bytes), int64_t size(void *) (0: not one of its blocks) and void free(void *).
#define PY_SSIZE_T_CLEAN
#define NPY_NO_DEPRECATED_API NPY_1_22_API_VERSION
#define NPY_TARGET_VERSION NPY_1_22_API_VERSION
#include <Python.h>
#include <numpy/arrayobject.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

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

struct Pool {
    void *(*alloc)(int64_t);
    int64_t (*size)(void *);
    void (*free)(void *);
    PyDataMem_Handler handler;
    PyObject *capsule;
    void *next;               // the block that the array being made gets
};

// With the interpreter lock held, as numpy calls them.
void *pool_malloc(void *ctx, size_t n)
{
    Pool *p = (Pool *)ctx;
    if (void *block = p->next) {
        p->next = nullptr;
        return block;
    }
    return malloc(n);
}
void *pool_calloc(void *, size_t n, size_t elsize) { return calloc(n, elsize); }
void pool_free(void *ctx, void *block, size_t)
{
    Pool *p = (Pool *)ctx;
    if (p->size(block)) p->free(block);
    else free(block);
}
void *pool_realloc(void *ctx, void *block, size_t n)
{
    Pool *p = (Pool *)ctx;
    const size_t have = block ? (size_t)p->size(block) : 0;
    if (!have) return realloc(block, n);
    if (n <= have) return block;
    void *q = malloc(n);
    if (!q) return nullptr;
    memcpy(q, block, have);
    p->free(block);
    return q;
}

// The pool with these functions.  Never freed: arrays keep their handler.
Pool *find_pool(void *alloc, void *size, void *free)
{
    static Pool *known[8];
    for (Pool *&p : known) {
        if (!p) {
            p = (Pool *)calloc(1, sizeof(Pool));
            if (!p) break;
            p->alloc = (void *(*)(int64_t))alloc;
            p->size = (int64_t(*)(void *))size;
            p->free = (void (*)(void *))free;
            strcpy(p->handler.name, "comet_b200_results");
            p->handler.version = 1;
            p->handler.allocator = {p, pool_malloc, pool_calloc, pool_realloc, pool_free};
            p->capsule = PyCapsule_New(&p->handler, "mem_handler", nullptr);
            if (!p->capsule) {
                ::free(p);
                p = nullptr;
                return nullptr;
            }
        }
        if ((void *)p->alloc == alloc && (void *)p->size == size && (void *)p->free == free) return p;
    }
    PyErr_SetString(PyExc_RuntimeError, "new_result: too many pools");
    return nullptr;
}

PyObject *new_result(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    if (n != 5) return PyErr_Format(PyExc_TypeError, "new_result(alloc, size, free, dtype, dims)");
    void *fn[3];
    for (int i = 0; i < 3; i++) {
        fn[i] = PyLong_AsVoidPtr(args[i]);
        if (!fn[i]) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "new_result: a null address");
    }
    PyArray_Descr *dtype = nullptr;
    if (!PyArray_DescrConverter(args[3], &dtype)) return nullptr;
    PyArray_Dims dims = {nullptr, 0};
    Pool *p = PyArray_IntpConverter(args[4], &dims) ? find_pool(fn[0], fn[1], fn[2]) : nullptr;
    PyObject *out = nullptr;
    if (p) {
        int64_t bytes = PyDataType_ELSIZE(dtype);
        for (int i = 0; i < dims.len; i++)
            if (dims.ptr[i] < 0 || __builtin_mul_overflow(bytes, (int64_t)dims.ptr[i], &bytes)) bytes = -1;
        void *block = bytes > 0 ? p->alloc(bytes) : nullptr;
        PyObject *old = block ? PyDataMem_SetHandler(p->capsule) : nullptr;
        if (old) {
            p->next = block;
            out = PyArray_NewFromDescr(&PyArray_Type, dtype, dims.len, dims.ptr, nullptr, nullptr, 0, nullptr);
            dtype = nullptr;                           // the call took the reference
            if (p->next) {                             // it failed before it asked for the memory
                p->next = nullptr;
                p->free(block);
            }
            PyObject *type, *value, *trace;
            PyErr_Fetch(&type, &value, &trace);
            PyObject *mine = PyDataMem_SetHandler(old);
            Py_XDECREF(mine);
            Py_DECREF(old);
            PyErr_Restore(type, value, trace);
        } else if (block) {
            p->free(block);
        } else {
            out = Py_NewRef(Py_None);
        }
    }
    PyDimMem_FREE(dims.ptr);
    Py_XDECREF(dtype);
    return out;
}

PyMethodDef methods[] = {
    {"call", (PyCFunction)(void (*)(void))call<int64_t>, METH_FASTCALL, "call(address, *integers) -> 64-bit result"},
    {"call_i32", (PyCFunction)(void (*)(void))call<int32_t>, METH_FASTCALL, "call_i32(address, *integers) -> 32-bit result"},
    {"new_result", (PyCFunction)(void (*)(void))new_result, METH_FASTCALL, "new_result(alloc, size, free, dtype, dims) -> array or None"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pycall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pycall(void)
{
    import_array();
    return PyModule_Create(&module);
}
