// The way from Python to the kernels' C entry points: ``bind(address, signature)`` makes a callable of an entry point,
// ``ptr(tensor, dtype, what)`` is a tensor's address after the checks that every launch makes.
//
// A step that runs eagerly is a few hundred launches, and its time is the host's where a prompt is short.  Through ctypes an
// entry point of 25 arguments took 2 us besides the launch itself (about 3 us), and the six pointers that a launch asks for on
// average 1.6 us.  Signatures are strings of one letter an argument, P pointer, i int, q long long, Q unsigned long long,
// f float; SIGNATURES (made from the list of entry points when this file is compiled) has a typed call for each that occurs.
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Dtype.h>

#include <cstring>
#include <utility>

namespace {
union Slot {
    void* p;
    long long i;
    float f;
};
template <typename T> T get(const Slot& s);
template <> inline void* get<void*>(const Slot& s) { return s.p; }
template <> inline int get<int>(const Slot& s) { return (int)s.i; }
template <> inline long long get<long long>(const Slot& s) { return s.i; }
template <> inline unsigned long long get<unsigned long long>(const Slot& s) { return (unsigned long long)s.i; }
template <> inline float get<float>(const Slot& s) { return s.f; }

template <typename... A, size_t... I>
int call_with(void* fn, const Slot* s, std::index_sequence<I...>) {
    return reinterpret_cast<int (*)(A...)>(fn)(get<A>(s[I])...);
}
template <typename... A> int call(void* fn, const Slot* s) { return call_with<A...>(fn, s, std::index_sequence_for<A...>{}); }

constexpr int MAX_ARGS = 64;
struct Signature {
    const char* letters;
    int (*call)(void*, const Slot*);
};
const Signature SIGNATURES[] = {
#include "entry_signatures.inc"
};

struct Entry {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    void* fn;
    const Signature* signature;
    int count;
};

PyObject* entry_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
    const Entry* e = reinterpret_cast<Entry*>(self);
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    if (n != e->count || (kwnames && PyTuple_GET_SIZE(kwnames))) {
        PyErr_Format(PyExc_TypeError, "this entry point takes %d arguments, %zd were given", e->count, n);
        return nullptr;
    }
    Slot slots[MAX_ARGS];
    for (int i = 0; i < e->count; i++) {
        PyObject* a = args[i];
        const char kind = e->signature->letters[i];
        if (kind == 'f') {
            const double v = PyFloat_AsDouble(a);
            if (v == -1.0 && PyErr_Occurred()) return nullptr;
            slots[i].f = (float)v;
        } else if (PyLong_Check(a)) {
            slots[i].i = (long long)PyLong_AsUnsignedLongLongMask(a);
        } else if (kind == 'P' && a == Py_None) {
            slots[i].p = nullptr;
        } else {
            PyErr_Format(PyExc_TypeError, "argument %d: expected %s, not %s", i + 1, kind == 'P' ? "an address or None" : "an int",
                         Py_TYPE(a)->tp_name);
            return nullptr;
        }
    }
    int code;
    Py_BEGIN_ALLOW_THREADS
    code = e->signature->call(e->fn, slots);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

PyTypeObject EntryType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2) {
        PyErr_SetString(PyExc_TypeError, "bind(address, signature)");
        return nullptr;
    }
    void* fn = PyLong_AsVoidPtr(args[0]);
    if (PyErr_Occurred()) return nullptr;
    const char* letters = PyUnicode_AsUTF8(args[1]);
    if (!letters) return nullptr;
    for (const Signature& s : SIGNATURES) {
        if (std::strcmp(s.letters, letters)) continue;
        Entry* e = PyObject_New(Entry, &EntryType);
        if (!e) return nullptr;
        e->vectorcall = entry_call;
        e->fn = fn;
        e->signature = &s;
        e->count = (int)std::strlen(letters);
        return reinterpret_cast<PyObject*>(e);
    }
    PyErr_Format(PyExc_ValueError, "no entry point of signature %s was compiled in", letters);
    return nullptr;
}

// Whatever is not in order goes to the function in Python, which says what is wrong.
PyObject* careful_ptr = nullptr;

bool is_dtype(PyObject* want, at::ScalarType have) {
    return THPDtype_Check(want) && reinterpret_cast<THPDtype*>(want)->scalar_type == have;
}

PyObject* ptr(PyObject*, PyObject* const* args, Py_ssize_t n, PyObject* kwnames) {
    if (!careful_ptr) {
        PyErr_SetString(PyExc_RuntimeError, "set_careful_ptr has not been called");
        return nullptr;
    }
    if (n >= 1 && !kwnames) {
        PyObject* t = args[0];
        if (t == Py_None) Py_RETURN_NONE;
        if (THPVariable_Check(t)) {
            try {
                const at::Tensor& v = THPVariable_Unpack(t);
                bool fits = v.is_cuda() && v.is_contiguous();
                if (fits && n >= 2 && args[1] != Py_None) {
                    const at::ScalarType have = v.scalar_type();
                    PyObject* want = args[1];
                    if (PyTuple_Check(want)) {
                        fits = false;
                        for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(want) && !fits; i++) fits = is_dtype(PyTuple_GET_ITEM(want, i), have);
                    } else {
                        fits = is_dtype(want, have);
                    }
                }
                if (fits) return PyLong_FromVoidPtr(v.data_ptr());
            } catch (const std::exception&) {                         // a tensor without one of these: as in Python
            }
        }
    }
    return PyObject_Vectorcall(careful_ptr, args, n, kwnames);
}

PyObject* set_careful_ptr(PyObject*, PyObject* fn) {
    Py_INCREF(fn);
    Py_XDECREF(careful_ptr);
    careful_ptr = fn;
    Py_RETURN_NONE;
}

PyMethodDef METHODS[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, "bind(address, signature): a callable"},
    {"ptr", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(ptr)), METH_FASTCALL | METH_KEYWORDS, "ptr(tensor, dtype, what): its address"},
    {"set_careful_ptr", set_careful_ptr, METH_O, "the function behind ptr for what is not in order"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef MODULE = {PyModuleDef_HEAD_INIT, "esp_b200_entry", nullptr, -1, METHODS};
}  // namespace

PyMODINIT_FUNC PyInit_esp_b200_entry() {
    EntryType.tp_name = "esp_b200_entry.Entry";
    EntryType.tp_basicsize = sizeof(Entry);
    EntryType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
    EntryType.tp_vectorcall_offset = offsetof(Entry, vectorcall);
    EntryType.tp_call = PyVectorcall_Call;
    if (PyType_Ready(&EntryType) < 0) return nullptr;
    return PyModule_Create(&MODULE);
}
