// Python's way into the launchers, as an extension module over the library of kernels, which does without Python and torch
// (build.py lists the launchers in entries.inc from the signatures in ops.py).  A layer launched kernel by kernel is a dozen calls with 8 to 30 arguments and
// three or four checked tensors each; a call through ctypes took 1.7 us where this one takes 0.12, a tensor's check 0.55
// us in Python and 0.08 here, a new tensor 2.6 by torch.empty with a type and a device and some 1.2 here.  A decoder layer of
// width 2,048 with 60 rows, nine launches: 161 -> 114 us, all of it the host's.
#include <Python.h>
#include <ATen/ops/empty.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <tuple>
#include <utility>

namespace {

template <class T> struct Argument;
template <class P> struct Argument<P*> {
    static P* from(PyObject* o) { return o == Py_None ? nullptr : (P*)PyLong_AsVoidPtr(o); }
};
template <> struct Argument<int> {
    static int from(PyObject* o) { return (int)PyLong_AsLong(o); }
};
template <> struct Argument<long long> {
    static long long from(PyObject* o) { return PyLong_AsLongLong(o); }
};
template <> struct Argument<float> {
    static float from(PyObject* o) { return (float)PyFloat_AsDouble(o); }
};

template <auto F> struct Entry;
template <class... A, int (*F)(A...)> struct Entry<F> {
    template <size_t... I> static PyObject* with(PyObject* const* args, std::index_sequence<I...>) {
        const std::tuple<A...> v{Argument<A>::from(args[I])...};
        if (PyErr_Occurred()) return nullptr;
        int code;
        Py_BEGIN_ALLOW_THREADS      // (a launch may have to wait for room in its stream's queue)
        code = F(std::get<I>(v)...);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(code);
    }
    static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
        if (n != (Py_ssize_t)sizeof...(A))
            return PyErr_Format(PyExc_TypeError, "the launcher takes %zd arguments, not %zd", (Py_ssize_t)sizeof...(A), n);
        return with(args, std::index_sequence_for<A...>());
    }
};

// ops._req(t, name, dtypes = None, shape = None): t where it is a contiguous CUDA tensor of one of the types and of the shape (a
// None in it stands for any size); everything else goes to the function in Python, which says what is wrong.
PyObject* say_why = nullptr;

bool fits(PyObject* const* args, Py_ssize_t n) {
    if (n < 2 || n > 4 || !THPVariable_Check(args[0])) return false;
    const at::Tensor& t = THPVariable_Unpack(args[0]);
    if (!t.is_cuda() || !t.is_contiguous()) return false;
    if (n > 2 && args[2] != Py_None) {
        if (!PyTuple_Check(args[2])) return false;
        bool one = false;
        for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[2]) && !one; ++i) {
            PyObject* d = PyTuple_GET_ITEM(args[2], i);
            if (!THPDtype_Check(d)) return false;
            one = ((THPDtype*)d)->scalar_type == t.scalar_type();
        }
        if (!one) return false;
    }
    if (n > 3 && args[3] != Py_None) {
        if (!PyTuple_Check(args[3]) || PyTuple_GET_SIZE(args[3]) != t.dim()) return false;
        for (Py_ssize_t i = 0; i < t.dim(); ++i) {
            PyObject* s = PyTuple_GET_ITEM(args[3], i);
            if (s == Py_None) continue;
            if (!PyLong_Check(s) || PyLong_AsLongLong(s) != t.size(i)) return false;
        }
    }
    return true;
}

PyObject* require(PyObject*, PyObject* const* args, Py_ssize_t n, PyObject* names) {
    if (!names) {
        try {
            if (fits(args, n)) {
                Py_INCREF(args[0]);
                return args[0];
            }
        } catch (...) {      // (a tensor without sizes, and the like: Python says why)
        }
        PyErr_Clear();
    }
    return PyObject_Vectorcall(say_why, args, (size_t)n, names);
}

// ops.empty(shape, dtype, device): torch.empty for a tuple of sizes or a number of elements; other forms go to torch itself.
PyObject* any_empty = nullptr;

PyObject* empty(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 3 || !(PyTuple_Check(args[0]) || PyLong_Check(args[0])) || !THPDtype_Check(args[1]) || !THPDevice_Check(args[2]))
        return PyObject_Vectorcall(any_empty, args, (size_t)n, nullptr);
    c10::SmallVector<int64_t, 5> sizes;
    if (PyLong_Check(args[0])) sizes.push_back(PyLong_AsLongLong(args[0]));
    else
        for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[0]); ++i) sizes.push_back(PyLong_AsLongLong(PyTuple_GET_ITEM(args[0], i)));
    if (PyErr_Occurred()) return nullptr;
    const auto options = at::TensorOptions().dtype(((THPDtype*)args[1])->scalar_type).device(((THPDevice*)args[2])->device);
    at::Tensor t;
    {
        pybind11::gil_scoped_release no_gil;
        t = at::empty(sizes, options);
    }
    return THPVariable_Wrap(std::move(t));
    END_HANDLE_TH_ERRORS
}

template <PyObject** F> PyObject* set(PyObject*, PyObject* f) {
    Py_XDECREF(*F);
    Py_INCREF(f);
    *F = f;
    Py_RETURN_NONE;
}

}  // namespace

#include "entries.inc"      // the launchers' prototypes, and AIR_ENTRIES: their places in the table of methods

namespace {

PyMethodDef methods[] = {
    AIR_ENTRIES
    {"require", (PyCFunction)(void (*)(void))require, METH_FASTCALL | METH_KEYWORDS, nullptr},
    {"empty", (PyCFunction)(void (*)(void))empty, METH_FASTCALL, nullptr},
    {"set_say_why", set<&say_why>, METH_O, nullptr},
    {"set_any_empty", set<&any_empty>, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "air_b200_entry", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_air_b200_entry() { return PyModule_Create(&module); }
