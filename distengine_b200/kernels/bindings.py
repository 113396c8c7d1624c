"""Calls of the kernel libraries' functions without ctypes: a CPython extension, generated from the
functions' signatures, that takes the arguments off the interpreter's stack and calls the C function by
its exact prototype.

A launch function takes up to 42 arguments; ctypes converts them through an object each, 2 to 4 us a
call (0.2 here).  Eager layers of a few launches are bound by the host: 64 single tokens through sink
attention 71 -> 66 us a pass, 8 through a window layer 39 -> 32, through the gated delta rule 95 -> 85.
As with ctypes, the interpreter's lock is released during the call, ``None`` is a null pointer and
integers are cut to the parameter's width.  Where the interpreter has no headers to compile it with,
``library`` calls the functions through ctypes.
"""

from __future__ import annotations

import hashlib
import importlib.machinery
import importlib.util
import os
import sysconfig

NAME = "distengine_b200_bindings"

_HEAD = """// Generated from the kernel libraries' signatures.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

static int take(PyObject* o, void** to) {
    if (o == Py_None) {
        *to = nullptr;
        return 0;
    }
    const unsigned long long v = PyLong_Check(o) ? PyLong_AsUnsignedLongLongMask(o) : 0;
    if (!PyLong_Check(o)) PyErr_SetString(PyExc_TypeError, "an address must be an integer or None");
    *to = (void*)v;
    return PyErr_Occurred() ? -1 : 0;
}
static int take(PyObject* o, int* to) {
    if (PyFloat_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "an integer argument is a float");
        return -1;
    }
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
    *to = (int)v;
    return v == (unsigned long long)-1 && PyErr_Occurred() ? -1 : 0;
}
static int take(PyObject* o, long long* to) {
    if (PyFloat_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "an integer argument is a float");
        return -1;
    }
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
    *to = (long long)v;
    return v == (unsigned long long)-1 && PyErr_Occurred() ? -1 : 0;
}
static int take(PyObject* o, float* to) {
    const double v = PyFloat_AsDouble(o);
    *to = (float)v;
    return v == -1.0 && PyErr_Occurred() ? -1 : 0;
}
static PyObject* wrong_count(Py_ssize_t given, int wanted) {
    PyErr_Format(PyExc_TypeError, "this function takes %d arguments (%zd given)", wanted, given);
    return nullptr;
}
"""

_TAIL = """
static PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 2) return wrong_count(n, 2);
    const long index = PyLong_AsLong(a[0]);
    if (PyErr_Occurred()) return nullptr;
    if (index < 0 || index >= COUNT || !PyLong_Check(a[1])) {
        PyErr_SetString(PyExc_ValueError, "bind(index of a signature, address)");
        return nullptr;
    }
    return PyCFunction_NewEx(&calls[index], a[1], nullptr);
}
static PyMethodDef methods[] = {
    {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
static PyModuleDef module = {PyModuleDef_HEAD_INIT, "%(name)s", nullptr, -1, methods,
                             nullptr, nullptr, nullptr, nullptr};
PyMODINIT_FUNC PyInit_%(name)s(void) { return PyModule_Create(&module); }
"""


def source(signatures: "list[str]") -> str:
    """The extension's source: ``signatures`` are strings of P (pointer), I (int), L (long long) and
    F (float), one a parameter."""
    types = {"P": "void*", "I": "int", "L": "long long", "F": "float"}
    out = [_HEAD]
    for i, sig in enumerate(signatures):
        out.append(f"static PyObject* call_{i}(PyObject* self, PyObject* const* a, Py_ssize_t n) {{")
        out.append(f"    if (n != {len(sig)}) return wrong_count(n, {len(sig)});")
        for j, c in enumerate(sig):
            out.append(f"    {types[c]} v{j};")
            out.append(f"    if (take(a[{j}], &v{j})) return nullptr;")
        proto = ", ".join(types[c] for c in sig) or "void"
        out.append(f"    int (*fn)({proto}) = (int (*)({proto}))PyLong_AsVoidPtr(self);")
        out.append("    int code;")
        out.append("    Py_BEGIN_ALLOW_THREADS")
        out.append(f"    code = fn({', '.join(f'v{j}' for j in range(len(sig)))});")
        out.append("    Py_END_ALLOW_THREADS")
        out.append("    return PyLong_FromLong(code);")
        out.append("}")
    out.append(f"constexpr long COUNT = {len(signatures)};")
    out.append("static PyMethodDef calls[] = {")
    for i in range(len(signatures)):
        out.append(f'    {{"call", (PyCFunction)(void (*)(void))call_{i}, METH_FASTCALL, nullptr}},')
    out.append("};")
    return "\n".join(out) + _TAIL % {"name": NAME}


def library_path(text: str, build_dir: str) -> str:
    tag = hashlib.sha256((text + sysconfig.get_config_var("EXT_SUFFIX")).encode()).hexdigest()[:12]
    return os.path.join(build_dir, f"bindings-{tag}.so")


def include_dir() -> str:
    return sysconfig.get_paths()["include"]


def load(path: str):
    spec = importlib.util.spec_from_file_location(
        NAME, path, loader=importlib.machinery.ExtensionFileLoader(NAME, path))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module
