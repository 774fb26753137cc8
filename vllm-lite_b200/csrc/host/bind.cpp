// What Python does for every launch, as an extension module: checking a tensor argument, turning tensors into addresses, calling a
// library's entry point, asking for the current stream, and the library product.  A step of more than 64 tokens is a
// few hundred launches that nothing replays; with ctypes and Python checks a launch cost the host 15 us (a Puturax step of 24
// requests 3.8 ms for 2 ms on the GPU).
//
//   need(t, dtype, name, ndim=None)   a CUDA tensor of that dtype (None: any), contiguous, of ndim dimensions (None: any); otherwise the
//                                     first function given to `setup` is called with the same arguments and says what is wrong
//   pointer(t)                        t itself: an entry point takes tensors, addresses and None where it wants a pointer
//   Entry(address, signature)         an `extern "C" int` function: one letter an argument: p pointer, i int, l long long, f float
//   stream()                          the current stream of the current device
//   mm(a, w, out)                     out = a w^T by the library, as torch.mm(a, w.t(), out=out) does it; out in a's dtype or float32
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>
#include <cstring>
#include <ATen/core/Tensor.h>
#include <ATen/ops/mm.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/PythonTorchFunctionTLS.h>

namespace {
PyObject *g_slow_need = nullptr, *g_slow_mm = nullptr;

PyObject* setup(PyObject*, PyObject* args) {
    PyObject *need, *mm;
    if (!PyArg_ParseTuple(args, "OO", &need, &mm)) return nullptr;
    Py_INCREF(need);
    Py_XSETREF(g_slow_need, need);
    Py_INCREF(mm);
    Py_XSETREF(g_slow_mm, mm);
    Py_RETURN_NONE;
}

PyObject* need(PyObject*, PyObject* const* args, Py_ssize_t n, PyObject* kwnames) {
    const Py_ssize_t named = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
    if ((n == 3 || n == 4) && !named && THPVariable_Check(args[0])) {
        const at::Tensor& t = THPVariable_Unpack(args[0]);
        bool ok = t.is_cuda() && t.is_contiguous();
        if (ok && args[1] != Py_None) ok = THPDtype_Check(args[1]) && reinterpret_cast<THPDtype*>(args[1])->scalar_type == t.scalar_type();
        if (ok && n == 4 && args[3] != Py_None) {
            const long d = PyLong_AsLong(args[3]);
            if (d == -1 && PyErr_Occurred()) return nullptr;
            ok = t.dim() == d;
        }
        if (ok) Py_RETURN_NONE;
    }
    return PyObject_Vectorcall(g_slow_need, args, n, kwnames);
}

PyObject* pointer(PyObject*, PyObject* t) {
    Py_INCREF(t);
    return t;
}

PyObject* stream(PyObject*, PyObject*) {
    try {
        return PyLong_FromVoidPtr(c10::cuda::getCurrentCUDAStream().stream());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

PyObject* mm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 3 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1]) || !THPVariable_Check(args[2])) {
        PyErr_SetString(PyExc_TypeError, "mm(a, w, out) takes three tensors");
        return nullptr;
    }
    // Whoever watches torch's functions or brings a tensor type of their own is asked as `torch.mm` asks them.  What the dispatcher decides by
    // (gradients, modes, transforms) it decides here too: the call passes all of its keys.
    bool watched = at::impl::torch_function_mode_enabled();
    for (int i = 0; i < 3 && !watched; ++i) watched = !THPVariable_CheckTypeExact(Py_TYPE(args[i]));
    if (watched) return PyObject_Vectorcall(g_slow_mm, args, n, nullptr);
    HANDLE_TH_ERRORS
    {
        const at::Tensor a = THPVariable_Unpack(args[0]), w = THPVariable_Unpack(args[1]);
        at::Tensor out = THPVariable_Unpack(args[2]);
        pybind11::gil_scoped_release others_run;
        if (out.scalar_type() == a.scalar_type()) at::mm_out(out, a, w.t());
        else at::mm_out(out, a, w.t(), out.scalar_type());
    }
    Py_INCREF(args[2]);
    return args[2];
    END_HANDLE_TH_ERRORS
}

// ---- entry points --------------------------------------------------------------------------------------------------------
// In both calling conventions that this runs under (System V on x86-64, AAPCS64 on Linux) whole numbers and addresses fill their registers
// and then 8-byte slots of the stack, floats registers of their own, each in their order, whatever the other kind does
// between them; eight floats fit theirs.  So one prototype, whole numbers first, calls them all: what the callee does not take it does not read.
#if !(defined(__x86_64__) || defined(__aarch64__)) || !defined(__linux__)
#error "the calling convention of this machine is not one that bind.cpp knows"
#endif
constexpr int MOST_WORDS = 40, MOST_FLOATS = 8;
typedef unsigned long long u64;
#define W8(i) w[i], w[i + 1], w[i + 2], w[i + 3], w[i + 4], w[i + 5], w[i + 6], w[i + 7]
#define T8 u64, u64, u64, u64, u64, u64, u64, u64
#define F8 float, float, float, float, float, float, float, float
typedef int (*Fn)(T8, T8, T8, T8, T8, F8);

struct Entry {
    PyObject_HEAD
    vectorcallfunc call;
    void* fn;
    int count;
    char kinds[MOST_WORDS + MOST_FLOATS + 1];
};

PyObject* entry_call(PyObject* self, PyObject* const* args, size_t nf, PyObject* kwnames) {
    const Entry* e = reinterpret_cast<Entry*>(self);
    const Py_ssize_t n = PyVectorcall_NARGS(nf);
    if (n != e->count || (kwnames && PyTuple_GET_SIZE(kwnames))) {
        PyErr_Format(PyExc_TypeError, "the entry point takes %d arguments, got %zd", e->count, n);
        return nullptr;
    }
    u64 w[MOST_WORDS] = {};
    float f[MOST_FLOATS] = {};
    int nw = 0, nfl = 0;
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject* a = args[i];
        switch (e->kinds[i]) {
            case 'p':
                if (a == Py_None) w[nw++] = 0;
                else if (THPVariable_Check(a)) {
                    try {
                        w[nw++] = (u64)(uintptr_t)THPVariable_Unpack(a).data_ptr();
                    } catch (const std::exception& x) {
                        PyErr_SetString(PyExc_RuntimeError, x.what());
                        return nullptr;
                    }
                } else w[nw++] = (u64)PyLong_AsUnsignedLongLong(a);
                break;
            case 'f': f[nfl++] = (float)PyFloat_AsDouble(a); break;
            case 'i': w[nw++] = (u64)(long long)(int)PyLong_AsLongLong(a); break;
            default: w[nw++] = (u64)PyLong_AsLongLong(a);
        }
        if (PyErr_Occurred()) return nullptr;
    }
    int code;
    Py_BEGIN_ALLOW_THREADS
    code = reinterpret_cast<Fn>(e->fn)(W8(0), W8(8), W8(16), W8(24), W8(32), f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

PyObject* entry_new(PyTypeObject* type, PyObject* args, PyObject*) {
    unsigned long long address;
    const char* kinds;
    if (!PyArg_ParseTuple(args, "Ks", &address, &kinds)) return nullptr;
    const size_t n = strlen(kinds);
    int floats = 0;
    for (const char* k = kinds; *k; ++k) {
        floats += *k == 'f';
        if (!strchr("pilf", *k)) { PyErr_Format(PyExc_ValueError, "argument kind '%c' is not known", *k); return nullptr; }
    }
    if (!address || floats > MOST_FLOATS || (int)n - floats > MOST_WORDS) {
        PyErr_Format(PyExc_ValueError, "an entry point with %zu arguments, %d floats", n, floats);
        return nullptr;
    }
    Entry* e = reinterpret_cast<Entry*>(type->tp_alloc(type, 0));
    if (!e) return nullptr;
    e->call = entry_call;
    e->fn = reinterpret_cast<void*>(address);
    e->count = (int)n;
    memcpy(e->kinds, kinds, n + 1);
    return reinterpret_cast<PyObject*>(e);
}

PyMemberDef entry_members[] = {{"__vectorcalloffset__", T_PYSSIZET, offsetof(Entry, call), READONLY, nullptr}, {nullptr, 0, 0, 0, nullptr}};
PyType_Slot entry_slots[] = {{Py_tp_new, (void*)entry_new}, {Py_tp_call, (void*)PyVectorcall_Call}, {Py_tp_members, entry_members}, {0, nullptr}};
PyType_Spec entry_spec = {"bind.Entry", sizeof(Entry), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_IMMUTABLETYPE, entry_slots};

PyMethodDef methods[] = {{"setup", setup, METH_VARARGS, nullptr},
                         {"need", (PyCFunction)(void (*)(void))need, METH_FASTCALL | METH_KEYWORDS, nullptr},
                         {"pointer", pointer, METH_O, nullptr},
                         {"stream", stream, METH_NOARGS, nullptr},
                         {"mm", (PyCFunction)(void (*)(void))mm, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "bind", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
}  // namespace

PyMODINIT_FUNC PyInit_bind() {
    PyObject* m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    PyObject* type = PyType_FromSpec(&entry_spec);
    if (!type || PyModule_AddObject(m, "Entry", type) < 0) {
        Py_XDECREF(type);
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
