// Calls of the kernel library's entry points from Python, without ctypes: each entry point becomes a builtin function that
// takes torch tensors (their device addresses are passed on), numbers and None in the order of its C arguments.
//
//   bind(address, types, name)       the caller of one entry point; types: one letter an argument (csrc/signatures.py)
//   on_device(error, *tensors)       raises error unless every tensor (None is left out) lives on a CUDA device
//   strided(t, shape, strides, at)   a view of t's storage, as Tensor.as_strided gives it, for scratch that needs no autograd
//
// Through ctypes a call of 29 arguments takes 4.2 us (and 0.25 us more a tensor for its address), here 0.5 us; as_strided 2.3 us
// and strided 0.5 us.  A layer's step makes six to eleven calls and as many views.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <memory>
#include <string>
#include <vector>

namespace {

union Arg {
    void* p;
    long l;
    double d;
};

struct Signature {
    const char* types;
    int (*call)(void*, const Arg*);
};

// One caller per list of types, written out by build.py: {"PIF", [](void* f, const Arg* a) { return ((int (*)(void*, int, float))f)(...); }}
const Signature signatures[] = {
#include "signatures.inc"
};

constexpr Py_ssize_t kMostArgs = 64;

struct Entry {
    void* fn;
    int (*call)(void*, const Arg*);
    std::string types, name;
    PyMethodDef def;
};

bool convert(PyObject* o, char type, Arg* out) {
    if (type == 'P') {
        if (o == Py_None) {
            out->p = nullptr;
        } else if (PyLong_Check(o)) {
            out->p = reinterpret_cast<void*>(PyLong_AsUnsignedLongMask(o));
        } else if (THPVariable_Check(o)) {
            const at::Tensor& t = THPVariable_Unpack(o);
            if (!t.is_cuda()) {
                PyErr_SetString(PyExc_TypeError, "a kernel was handed a tensor that does not live on a CUDA device");
                return false;
            }
            out->p = t.data_ptr();
        } else {
            PyErr_Format(PyExc_TypeError, "a kernel takes an address, a tensor or None here, not %s", Py_TYPE(o)->tp_name);
            return false;
        }
    } else if (type == 'F' || type == 'D') {
        out->d = PyFloat_AsDouble(o);
    } else {
        if (PyFloat_Check(o)) {
            PyErr_SetString(PyExc_TypeError, "a kernel takes a whole number here, not float");
            return false;
        }
        out->l = static_cast<long>(PyLong_AsUnsignedLongMask(o));      // what does not fit int is cut, as ctypes does
    }
    return !PyErr_Occurred();
}

PyObject* call_entry(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    try {
        const Entry* e = static_cast<const Entry*>(PyCapsule_GetPointer(self, "aien.entry"));
        if (e == nullptr) return nullptr;
        if (n != static_cast<Py_ssize_t>(e->types.size())) {
            PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, not %zd", e->name.c_str(), static_cast<Py_ssize_t>(e->types.size()), n);
            return nullptr;
        }
        Arg a[kMostArgs];
        for (Py_ssize_t i = 0; i < n; ++i)
            if (!convert(args[i], e->types[i], &a[i])) return nullptr;
        int rc;
        Py_BEGIN_ALLOW_THREADS                                          // a full launch queue may make the call wait
        rc = e->call(e->fn, a);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(rc);
    } catch (const std::exception& x) {
        PyErr_SetString(PyExc_RuntimeError, x.what());
        return nullptr;
    }
}

void free_entry(PyObject* capsule) { delete static_cast<Entry*>(PyCapsule_GetPointer(capsule, "aien.entry")); }

PyObject* bind(PyObject*, PyObject* args) {
    unsigned long long address;
    const char *types, *name;
    if (!PyArg_ParseTuple(args, "Kss", &address, &types, &name)) return nullptr;
    const Signature* found = nullptr;
    for (const Signature& s : signatures)
        if (std::strcmp(s.types, types) == 0) found = &s;
    if (found == nullptr || std::strlen(types) > static_cast<size_t>(kMostArgs)) {
        PyErr_Format(PyExc_ValueError, "no caller was built for %s(%s)", name, types);
        return nullptr;
    }
    auto entry = std::make_unique<Entry>();
    entry->fn = reinterpret_cast<void*>(address);
    entry->call = found->call;
    entry->types = types;
    entry->name = name;
    entry->def = PyMethodDef{entry->name.c_str(), reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_entry)), METH_FASTCALL, nullptr};
    PyObject* capsule = PyCapsule_New(entry.get(), "aien.entry", free_entry);
    if (capsule == nullptr) return nullptr;
    PyMethodDef* def = &entry.release()->def;                           // the capsule owns the entry, the function the capsule
    PyObject* fn = PyCFunction_New(def, capsule);
    Py_DECREF(capsule);
    return fn;
}

PyObject* on_device(PyObject*, PyObject* const* args, Py_ssize_t n) {
    for (Py_ssize_t i = 1; i < n; ++i) {
        if (args[i] == Py_None) continue;
        if (!THPVariable_Check(args[i])) {
            PyErr_Format(PyExc_TypeError, "a tensor or None is wanted here, not %s", Py_TYPE(args[i])->tp_name);
            return nullptr;
        }
        if (!THPVariable_Unpack(args[i]).is_cuda()) {
            PyErr_SetString(args[0], "kernel arguments must live on the CUDA device (there is no CPU path)");
            return nullptr;
        }
    }
    Py_RETURN_NONE;
}

PyObject* strided(PyObject*, PyObject* const* args, Py_ssize_t n) {
    try {
        if (n != 4 || !THPVariable_Check(args[0]) || !PyTuple_Check(args[1]) || !PyTuple_Check(args[2]) || PyTuple_GET_SIZE(args[1]) != PyTuple_GET_SIZE(args[2])) {
            PyErr_SetString(PyExc_TypeError, "strided(tensor, shape, strides, offset)");
            return nullptr;
        }
        const at::Tensor& base = THPVariable_Unpack(args[0]);
        const Py_ssize_t dims = PyTuple_GET_SIZE(args[1]);
        c10::SmallVector<int64_t, 8> shape(dims), strides(dims);
        const int64_t at = PyLong_AsLongLong(args[3]);
        int64_t last = at;                                              // the last number that the view reaches
        bool empty = false;
        for (Py_ssize_t i = 0; i < dims; ++i) {
            shape[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(args[1], i));
            strides[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(args[2], i));
            if (shape[i] < 0 || strides[i] < 0) {
                if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "a view's sizes and strides are not negative");
                return nullptr;
            }
            empty |= shape[i] == 0;
            last += (shape[i] - 1) * strides[i];
        }
        if (PyErr_Occurred()) return nullptr;
        if (at < 0 || (!empty && static_cast<size_t>(last + 1) * base.itemsize() > base.storage().nbytes())) {
            PyErr_SetString(PyExc_ValueError, "a view reaches beyond its storage");
            return nullptr;
        }
        auto impl = c10::make_intrusive<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(base.storage()), base.key_set(), base.dtype());
        impl->set_sizes_and_strides(shape, strides, at);
        return THPVariable_Wrap(at::Tensor(std::move(impl)));
    } catch (const std::exception& x) {
        PyErr_SetString(PyExc_RuntimeError, x.what());
        return nullptr;
    }
}

template <typename F>
PyCFunction fast(F f) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }

PyMethodDef methods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"on_device", fast(on_device), METH_FASTCALL, nullptr},
    {"strided", fast(strided), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_aien_launch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__aien_launch() { return PyModule_Create(&module); }
