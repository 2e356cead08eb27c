// Calls of the kernel launchers from Python without ctypes: a launcher's entry point with the types of its parameters, called with
// Python numbers and tensors as they are.
//
// A layer of decoded tokens or a short portion is bound by the host, and a call of twenty-five parameters through ctypes - an object for
// every pointer, three questions to its tensor, a converter for every number - cost it about as much as the launch itself.  Layers
// launched from Python: 48 single tokens with window attention 66 -> 54 us (four launches, two library products), a routed
// feed-forward over one token 59 -> 37 us (eight launches).  The reference calls its kernels from C++ and has no such layer
// (apps/qwen_serve.cu).
//
// One function type serves all launchers.  By the System V x86-64 calling convention (and AAPCS64) numbers and pointers go into
// integer registers and then onto the stack, eight bytes each, in their own order; float parameters, of which no launcher has more than
// eight, go into vector registers in theirs.  So a call with the floats first and the others after them, padded with zeros,
// leaves every parameter where the launcher looks for it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <climits>
#include <cstdint>
#include <string>

#if !defined(__x86_64__) && !defined(__aarch64__)
#error "the calling convention this file relies on is that of 64-bit x86 or Arm"
#endif

namespace {

constexpr int MAX_FLOATS = 8, MAX_OTHERS = 40;
typedef int64_t W;
typedef int (*Launcher)(float, float, float, float, float, float, float, float, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W,
                        W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W);

PyObject* kernel_error = nullptr;          // the package's exception, given by `set_error`

struct Call {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    Launcher launcher;
    std::string* types;                    // one letter a parameter: p(ointer), i(nt), l(ong long), f(loat)
    Py_ssize_t required;                   // of so many; those after them are zero where they are left out
    PyObject* name;
};

// The address of a contiguous tensor on the device; false with an exception set.  Every question to the tensor may throw (a layout
// without strides, a subclass that answers in Python, a tensor without storage): the functions that Python calls catch that, by
// `translated` - torch's own frame, HANDLE_TH_ERRORS, also collects warnings, which cost a layer of four launches 3 us.
bool address_of(PyObject* obj, W& out) {
    const at::Tensor& t = THPVariable_Unpack(obj);
    if (!t.is_contiguous()) {
        PyErr_SetString(kernel_error ? kernel_error : PyExc_RuntimeError, "kernels take contiguous tensors");
        return false;
    }
    if (!t.is_cuda()) {
        PyErr_SetString(kernel_error ? kernel_error : PyExc_RuntimeError,
                        "kernels take tensors on the device; a host tensor's address means nothing there");
        return false;
    }
    out = reinterpret_cast<W>(t.data_ptr());
    return true;
}

PyObject* translated() {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
}

bool pointer_of(PyObject* obj, W& out) {
    if (obj == Py_None) { out = 0; return true; }
    if (PyLong_Check(obj)) {
        out = reinterpret_cast<W>(PyLong_AsVoidPtr(obj));
        return !(out == 0 && PyErr_Occurred());
    }
    if (THPVariable_Check(obj)) return address_of(obj, out);
    PyObject* value = PyObject_GetAttrString(obj, "value");        // ctypes.c_void_p
    if (!value) return false;
    const bool ok = value == Py_None || PyLong_Check(value);
    if (!ok) PyErr_SetString(PyExc_TypeError, "a pointer parameter takes None, an address, a tensor or ctypes.c_void_p");
    else out = value == Py_None ? 0 : reinterpret_cast<W>(PyLong_AsVoidPtr(value));
    Py_DECREF(value);
    return ok && !PyErr_Occurred();
}

PyObject* call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
    Call* c = reinterpret_cast<Call*>(self);
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    if (kwnames && PyTuple_GET_SIZE(kwnames)) return PyErr_Format(PyExc_TypeError, "%U takes no keyword arguments", c->name);
    if (n < c->required || n > (Py_ssize_t)c->types->size())
        return PyErr_Format(PyExc_TypeError, "%U takes %zd arguments, got %zd", c->name, (Py_ssize_t)c->types->size(), n);
    float f[MAX_FLOATS] = {};
    W w[MAX_OTHERS] = {};
    int nf = 0, nw = 0;
    try {
        for (Py_ssize_t i = 0; i < n; ++i) {
            switch ((*c->types)[i]) {
                case 'p':
                    if (!pointer_of(args[i], w[nw++])) return nullptr;
                    break;
                case 'f': {
                    const double v = PyFloat_AsDouble(args[i]);
                    if (v == -1.0 && PyErr_Occurred()) return nullptr;
                    f[nf++] = (float)v;
                    break;
                }
                default: {
                    const long long v = PyLong_AsLongLong(args[i]);
                    if (v == -1 && PyErr_Occurred()) return nullptr;
                    if ((*c->types)[i] == 'i' && (v < INT_MIN || v > INT_MAX))
                        return PyErr_Format(PyExc_OverflowError, "argument %zd of %U does not fit an int", i + 1, c->name);
                    w[nw++] = v;
                }
            }
        }
    } catch (...) {
        return translated();
    }
    int code;
    Py_BEGIN_ALLOW_THREADS
    code = c->launcher(f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8], w[9], w[10], w[11],
                       w[12], w[13], w[14], w[15], w[16], w[17], w[18], w[19], w[20], w[21], w[22], w[23], w[24], w[25], w[26], w[27], w[28],
                       w[29], w[30], w[31], w[32], w[33], w[34], w[35], w[36], w[37], w[38], w[39]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

PyObject* call_new(PyTypeObject* type, PyObject* args, PyObject*) {
    PyObject* address;
    const char* types;
    PyObject* name;
    if (!PyArg_ParseTuple(args, "OsU", &address, &types, &name)) return nullptr;
    void* at = PyLong_AsVoidPtr(address);
    if (!at) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "no address for %U", name);
    int floats = 0, others = 0;
    Py_ssize_t required = -1;              // a '|' stands before the first parameter that may be left out
    for (const char* t = types; *t; ++t) {
        if (*t == '|' && required < 0) {
            required = t - types;
            continue;
        }
        if (!strchr("pilf", *t)) return PyErr_Format(PyExc_ValueError, "%U: unknown parameter type '%c'", name, *t);
        ++(*t == 'f' ? floats : others);
    }
    if (floats > MAX_FLOATS || others > MAX_OTHERS) return PyErr_Format(PyExc_ValueError, "%U has too many parameters", name);
    Call* c = reinterpret_cast<Call*>(type->tp_alloc(type, 0));
    if (!c) return nullptr;
    c->vectorcall = call;
    c->launcher = reinterpret_cast<Launcher>(at);
    c->types = new std::string(types);
    c->required = required < 0 ? (Py_ssize_t)c->types->size() : required;
    if (required >= 0) c->types->erase(required, 1);
    Py_INCREF(name);
    c->name = name;
    return reinterpret_cast<PyObject*>(c);
}

void call_dealloc(PyObject* self) {
    Call* c = reinterpret_cast<Call*>(self);
    delete c->types;
    Py_XDECREF(c->name);
    Py_TYPE(self)->tp_free(self);
}

PyTypeObject call_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ptr(tensor or None) -> address: what a launcher is handed for the tensor, after the same questions.
PyObject* ptr(PyObject*, PyObject* obj) {
    W at = 0;
    if (obj == Py_None) return PyLong_FromLong(0);
    if (!THPVariable_Check(obj)) return PyErr_Format(PyExc_TypeError, "expected a tensor or None, got %R", (PyObject*)Py_TYPE(obj));
    try {
        if (!address_of(obj, at)) return nullptr;
    } catch (...) {
        return translated();
    }
    return PyLong_FromVoidPtr(reinterpret_cast<void*>(at));
}

PyObject* set_error(PyObject*, PyObject* type) {
    Py_INCREF(type);
    Py_XSETREF(kernel_error, type);
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"ptr", ptr, METH_O, "The device address of a contiguous tensor (0 for None)."},
                         {"set_error", set_error, METH_O, "The exception for tensors that a launcher cannot take."},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "kvb200_host_call", "Calls of the kernel launchers.", -1, methods};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_kvb200_host_call() {
    call_type.tp_name = "kvb200_host_call.Call";
    call_type.tp_basicsize = sizeof(Call);
    call_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
    call_type.tp_vectorcall_offset = offsetof(Call, vectorcall);
    call_type.tp_call = PyVectorcall_Call;
    call_type.tp_new = call_new;
    call_type.tp_dealloc = call_dealloc;
    if (PyType_Ready(&call_type) < 0) return nullptr;
    PyObject* m = PyModule_Create(&module);
    if (!m) return nullptr;
    Py_INCREF(&call_type);
    if (PyModule_AddObject(m, "Call", reinterpret_cast<PyObject*>(&call_type)) < 0) return nullptr;
    return m;
}
