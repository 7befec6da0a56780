// Calls into the kernel libraries without ctypes: a step of a prompt launches hundreds of kernels, and what the host spends on
// each call's arguments is what a short prompt waits for (28 arguments, twelve of them tensors: 9.1 us by ctypes with the
// addresses taken in Python, 1.8 here).
//
// Function(address, signature, name): a callable for a C entry point `int f(...)` whose parameters are pointers, int and long
// long ("i") and float ("f").  An argument for "i" is an int, None (a null pointer) or an object with data_ptr() (a tensor).
// The System V ABI of x86-64 hands integers and floats over in sequences of their own, each in the order of the parameters, and
// a callee reads only those it has, so one call with room for all of them serves every entry point.  Up to 48
// integers and 8 floats (those that fit the registers: a ninth would take a place among the integers on the stack).
//
// fits(tensor, dtype, contiguous): whether a tensor lives on the GPU, has that dtype (None: any) and is contiguous
// (False: need not be).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#if !defined(__x86_64__) || defined(_WIN32)
#error "the calls below follow the System V ABI of x86-64"
#endif

static const int MAX_INTS = 48, MAX_FLOATS = 8;
typedef long long i64;
typedef int (*Entry)(float, float, float, float, float, float, float, float, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64,
                     i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64,
                     i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64, i64);

struct Function {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    Entry entry;
    int count;
    char signature[MAX_INTS + MAX_FLOATS + 1];
    PyObject* name;
};

static PyObject *s_data_ptr, *s_is_cuda, *s_dtype, *s_is_contiguous;

// The integer an argument stands for; -1 with an exception set where it stands for none.
static i64 integer_of(PyObject* arg) {
    if (PyLong_Check(arg)) {
        int overflow = 0;
        const i64 value = PyLong_AsLongLongAndOverflow(arg, &overflow);
        if (!overflow) return value;
        return (i64)PyLong_AsUnsignedLongLong(arg);          // raises where that is too small as well
    }
    PyObject* address = PyObject_CallMethodNoArgs(arg, s_data_ptr);
    if (!address) return -1;
    i64 value = -1;
    if (PyLong_Check(address)) value = (i64)PyLong_AsUnsignedLongLong(address);
    else PyErr_SetString(PyExc_TypeError, "data_ptr() gave no int");
    Py_DECREF(address);
    return value;
}

static PyObject* function_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
    Function* f = (Function*)self;
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    if (n != f->count || (kwnames && PyTuple_GET_SIZE(kwnames))) {
        PyErr_Format(PyExc_TypeError, "%U takes %d positional arguments, got %zd", f->name, f->count, n);
        return nullptr;
    }
    i64 v[MAX_INTS];
    float x[MAX_FLOATS] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    memset(v, 0, sizeof(v));
    int ints = 0, floats = 0;
    for (int i = 0; i < f->count; ++i) {
        PyObject* arg = args[i];
        if (f->signature[i] == 'f') {
            const double value = PyFloat_AsDouble(arg);
            if (value == -1.0 && PyErr_Occurred()) return nullptr;
            x[floats++] = (float)value;
        } else if (arg == Py_None) {
            ints++;
        } else {
            const i64 value = integer_of(arg);
            if (value == -1 && PyErr_Occurred()) return nullptr;
            v[ints++] = value;
        }
    }
    int code;
    Py_BEGIN_ALLOW_THREADS                                    // a launch may wait for room in the stream's queue
    code = f->entry(x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7], v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9],
                    v[10], v[11], v[12], v[13], v[14], v[15], v[16], v[17], v[18], v[19], v[20], v[21], v[22], v[23], v[24],
                    v[25], v[26], v[27], v[28], v[29], v[30], v[31], v[32], v[33], v[34], v[35], v[36], v[37], v[38], v[39],
                    v[40], v[41], v[42], v[43], v[44], v[45], v[46], v[47]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

static PyObject* function_new(PyTypeObject* type, PyObject* args, PyObject*) {
    unsigned long long address;
    const char* signature;
    PyObject* name;
    if (!PyArg_ParseTuple(args, "KsU", &address, &signature, &name)) return nullptr;
    int ints = 0, floats = 0;
    for (const char* c = signature; *c; ++c) {
        if (*c == 'f') ++floats;
        else if (*c == 'i') ++ints;
        else return PyErr_Format(PyExc_ValueError, "%U: a parameter is 'i' or 'f', not '%c'", name, *c);
    }
    if (ints > MAX_INTS || floats > MAX_FLOATS || !address)
        return PyErr_Format(PyExc_ValueError, "%U: at most %d integers and %d floats, at an address", name, MAX_INTS, MAX_FLOATS);
    Function* f = (Function*)type->tp_alloc(type, 0);
    if (!f) return nullptr;
    f->vectorcall = function_call;
    f->entry = (Entry)(uintptr_t)address;
    f->count = ints + floats;
    strcpy(f->signature, signature);
    Py_INCREF(name);
    f->name = name;
    return (PyObject*)f;
}

static void function_dealloc(PyObject* self) {
    Py_XDECREF(((Function*)self)->name);
    Py_TYPE(self)->tp_free(self);
}

static PyTypeObject FunctionType = {PyVarObject_HEAD_INIT(nullptr, 0)};

static PyObject* fits(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 3) {
        PyErr_SetString(PyExc_TypeError, "fits takes a tensor, a dtype or None, and whether it is to be contiguous");
        return nullptr;
    }
    PyObject* tensor = args[0];
    PyObject* cuda = PyObject_GetAttr(tensor, s_is_cuda);
    if (!cuda) return nullptr;
    bool ok = cuda == Py_True;
    Py_DECREF(cuda);
    if (ok && args[1] != Py_None) {
        PyObject* dtype = PyObject_GetAttr(tensor, s_dtype);
        if (!dtype) return nullptr;
        ok = dtype == args[1];
        Py_DECREF(dtype);
    }
    if (ok && args[2] == Py_True) {
        PyObject* contiguous = PyObject_CallMethodNoArgs(tensor, s_is_contiguous);
        if (!contiguous) return nullptr;
        ok = contiguous == Py_True;
        Py_DECREF(contiguous);
    }
    return PyBool_FromLong(ok);
}

static PyMethodDef methods[] = {{"fits", (PyCFunction)(void (*)(void))fits, METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};
static PyModuleDef module = {PyModuleDef_HEAD_INIT, "host_call", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

PyMODINIT_FUNC PyInit_host_call(void) {
    FunctionType.tp_name = "host_call.Function";
    FunctionType.tp_basicsize = sizeof(Function);
    FunctionType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
    FunctionType.tp_vectorcall_offset = offsetof(Function, vectorcall);
    FunctionType.tp_call = PyVectorcall_Call;
    FunctionType.tp_new = function_new;
    FunctionType.tp_dealloc = function_dealloc;
    if (PyType_Ready(&FunctionType) < 0) return nullptr;
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_is_cuda = PyUnicode_InternFromString("is_cuda");
    s_dtype = PyUnicode_InternFromString("dtype");
    s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
    if (!s_data_ptr || !s_is_cuda || !s_dtype || !s_is_contiguous) return nullptr;
    PyObject* m = PyModule_Create(&module);
    if (!m) return nullptr;
    Py_INCREF(&FunctionType);
    if (PyModule_AddObject(m, "Function", (PyObject*)&FunctionType) < 0) return nullptr;
    return m;
}
