// Calls of the kernel launchers from Python without a foreign-function library in between.
//
// A step that is not replayed from a graph makes some hundred launches, each a C function of 10 to 40 integers, pointers and
// floats.  Through ctypes an argument is an object of its own and is converted twice.  Here a launcher is one call with plain
// numbers (a norm of two rows: 9.0 us of host time through ctypes, 6.9 now, of which the launch itself is 3).
//
// All launchers take integers of at most 64 bits, pointers and 32-bit floats and return an int.  In the calling conventions
// of x86-64 (System V) and 64-bit ARM (AAPCS64, Linux) the n-th integer or pointer argument goes to the same place whatever
// floats stand between, and the other way round, a 32-bit integer takes the place of a 64-bit one, and arguments that the
// callee does not have are ignored; so one function type with MAX_INTS integers and 8 floats (which fit the registers)
// serves all launchers.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#if !defined(__linux__) || !(defined(__x86_64__) || defined(__aarch64__))
#error "the calling conventions relied on are those of 64-bit Linux on x86 and ARM"
#endif

#define MAX_INTS 48
#define MAX_FLOATS 8
typedef unsigned long long u64;
typedef int (*Launcher)(u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64,
                        u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64, u64,
                        u64, u64, u64, u64, u64, u64, float, float, float, float, float, float, float, float);

static PyObject *s_data_ptr, *s_is_cuda, *s_is_contiguous, *s_dtype;

// call(address, arguments..): what `integer`, `pointer`, `ptr` and `real` give (None: a null pointer)
static PyObject* fc_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
    u64 v[MAX_INTS] = {0};
    float f[MAX_FLOATS] = {0};
    int nv = 0, nf = 0;
    if (n < 1 || !PyLong_Check(a[0])) {
        PyErr_SetString(PyExc_TypeError, "call: the launcher's address comes first");
        return nullptr;
    }
    const u64 address = PyLong_AsUnsignedLongLongMask(a[0]);
    for (Py_ssize_t i = 1; i < n; ++i) {
        PyObject* o = a[i];
        if (PyFloat_Check(o)) {
            if (nf == MAX_FLOATS) {
                PyErr_SetString(PyExc_TypeError, "call: more than 8 floats");
                return nullptr;
            }
            f[nf++] = (float)PyFloat_AS_DOUBLE(o);
            continue;
        }
        if (nv == MAX_INTS) {
            PyErr_SetString(PyExc_TypeError, "call: more than 48 integers");
            return nullptr;
        }
        if (o == Py_None) {
            v[nv++] = 0;
        } else {
            v[nv] = PyLong_AsUnsignedLongLongMask(o);              // takes what has __index__
            if (v[nv] == (u64)-1 && PyErr_Occurred()) return nullptr;
            ++nv;
        }
    }
    if (!address) {
        PyErr_SetString(PyExc_ValueError, "call: a null address");
        return nullptr;
    }
    const Launcher fn = reinterpret_cast<Launcher>(address);
    int r;
    Py_BEGIN_ALLOW_THREADS
    r = fn(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[12], v[13], v[14], v[15], v[16], v[17],
           v[18], v[19], v[20], v[21], v[22], v[23], v[24], v[25], v[26], v[27], v[28], v[29], v[30], v[31], v[32], v[33], v[34],
           v[35], v[36], v[37], v[38], v[39], v[40], v[41], v[42], v[43], v[44], v[45], v[46], v[47], f[0], f[1], f[2], f[3],
           f[4], f[5], f[6], f[7]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(r);
}

// ptr(tensor or None): the address of its first element
static PyObject* fc_ptr(PyObject*, PyObject* t) {
    if (t == Py_None) return PyLong_FromLong(0);
    return PyObject_CallMethodNoArgs(t, s_data_ptr);
}

// The kinds of arguments, each as ctypes takes it: `call` tells floats from the others by their type alone, so that a float
// in an integer's place, or a text, must not get there.
static PyObject* fc_integer(PyObject*, PyObject* x) { return PyNumber_Index(x); }      // no float, no None
static PyObject* fc_pointer(PyObject*, PyObject* x) {
    if (x == Py_None) return PyLong_FromLong(0);
    if (!PyLong_Check(x)) {
        PyErr_Format(PyExc_TypeError, "a pointer is an integer or None, not %.100s", Py_TYPE(x)->tp_name);
        return nullptr;
    }
    Py_INCREF(x);
    return x;
}
static PyObject* fc_real(PyObject*, PyObject* x) {
    const double v = PyFloat_AsDouble(x);                                             // no text
    if (v == -1.0 && PyErr_Occurred()) return nullptr;
    return PyFloat_FromDouble(v);
}

// fits(tensor, dtype or None): a contiguous CUDA tensor of this type?
static PyObject* fc_fits(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 2) {
        PyErr_SetString(PyExc_TypeError, "fits: a tensor and a type");
        return nullptr;
    }
    PyObject* x = PyObject_GetAttr(a[0], s_is_cuda);
    if (!x) return nullptr;
    bool ok = x == Py_True;
    Py_DECREF(x);
    if (ok) {
        x = PyObject_CallMethodNoArgs(a[0], s_is_contiguous);
        if (!x) return nullptr;
        ok = x == Py_True;
        Py_DECREF(x);
    }
    if (ok && a[1] != Py_None) {
        x = PyObject_GetAttr(a[0], s_dtype);
        if (!x) return nullptr;
        ok = x == a[1];                                            // types are single objects
        Py_DECREF(x);
    }
    return PyBool_FromLong(ok);
}

static PyMethodDef methods[] = {
    {"call", (PyCFunction)(void (*)(void))fc_call, METH_FASTCALL, "call(address, *numbers) -> int"},
    {"ptr", fc_ptr, METH_O, "the address of a tensor's first element; 0 for None"},
    {"integer", fc_integer, METH_O, "its argument as an integer; TypeError where it is none"},
    {"pointer", fc_pointer, METH_O, "its argument, an address; 0 for None"},
    {"real", fc_real, METH_O, "its argument, a number, as a float"},
    {"fits", (PyCFunction)(void (*)(void))fc_fits, METH_FASTCALL, "is it a contiguous CUDA tensor of this type (None: any)?"},
    {nullptr, nullptr, 0, nullptr}};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

PyMODINIT_FUNC PyInit_fastcall(void) {
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_is_cuda = PyUnicode_InternFromString("is_cuda");
    s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
    s_dtype = PyUnicode_InternFromString("dtype");
    if (!s_data_ptr || !s_is_cuda || !s_is_contiguous || !s_dtype) return nullptr;
    return PyModule_Create(&module);
}
