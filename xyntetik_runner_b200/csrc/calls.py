"""A Python extension that calls the CUDA library's launchers directly.

A step of a few hundred tokens is a hundred launches whose host time nothing hides, and of a launch's host time ctypes takes the
larger part: it converts twenty to thirty arguments one by one through generic code.  This module writes one C++ function per launcher
from the signature table (``signatures.py``), each converting its own arguments in line; ``build.py`` compiles it beside the
library, which it finds at run time (``bind``).  Measured: a call of eleven arguments 0.26 us,
by ctypes 1.69.

A function takes what its launcher takes, in order, and returns what it returns; where the launcher sets an int through a pointer
(letter "o") that argument is left out, and the function returns the launcher's error code if that is not zero, else the int.
"""
from __future__ import annotations

from .signatures import LONG, SIGNATURES

_TYPES = {"p": "void*", "i": "int", "l": "long long", "f": "float", "u": "unsigned", "U": "unsigned long long", "o": "int*"}
_READ = {"p": "xr_pointer", "i": "(int)PyLong_AsLong", "l": "PyLong_AsLongLong", "f": "(float)PyFloat_AsDouble", "u": "(unsigned)PyLong_AsUnsignedLong",
         "U": "PyLong_AsUnsignedLongLong"}

_HEAD = """#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>
static inline void* xr_pointer(PyObject* o) { return o == Py_None ? nullptr : (void*)PyLong_AsUnsignedLongLong(o); }
"""


def source() -> str:
    out, table, binds = [_HEAD], [], []
    for name, letters in SIGNATURES.items():
        res = "long long" if name in LONG else "int"
        given = [c for c in letters if c != "o"]
        out.append(f"static {res} (*f_{name})({', '.join(_TYPES[c] for c in letters) or 'void'});")
        body, args, at = [], [], 0
        for c in letters:
            if c == "o":
                args.append("&set")
                continue
            body.append(f"    const auto a{at} = {_READ[c]}(a[{at}]);")
            args.append(f"a{at}")
            at += 1
        sets = "o" in letters
        out.append(f"""static PyObject* w_{name}(PyObject*, PyObject* const* a, Py_ssize_t n) {{
    if (n != {len(given)}) return PyErr_Format(PyExc_TypeError, "{name}: {len(given)} arguments, not %zd", n);
    (void)a;
{chr(10).join(body)}
    if (PyErr_Occurred()) return nullptr;
    {res} r;{' int set = 0;' if sets else ''}
    Py_BEGIN_ALLOW_THREADS
    r = f_{name}({', '.join(args)});
    Py_END_ALLOW_THREADS
    return PyLong_FromLongLong({'r != 0 ? r : set' if sets else 'r'});
}}""")
        table.append(f'    {{"{name}", (PyCFunction)(void*)w_{name}, METH_FASTCALL, nullptr}},')
        binds.append(f'    if (!(*(void**)&f_{name} = dlsym(lib, "{name}"))) return PyErr_Format(PyExc_OSError, "%s: no {name}", path);')
    out.append("""static PyObject* xr_bind(PyObject*, PyObject* arg) {
    const char* path = PyUnicode_AsUTF8(arg);
    if (!path) return nullptr;
    void* lib = dlopen(path, RTLD_NOW);
    if (!lib) return PyErr_Format(PyExc_OSError, "%s", dlerror());
""" + "\n".join(binds) + """
    Py_RETURN_NONE;
}
static PyMethodDef xr_methods[] = {
    {"bind", xr_bind, METH_O, nullptr},
""" + "\n".join(table) + """
    {nullptr, nullptr, 0, nullptr}};
static PyModuleDef xr_module = {PyModuleDef_HEAD_INIT, "xrb200_calls", nullptr, -1, xr_methods, nullptr, nullptr, nullptr, nullptr};
PyMODINIT_FUNC PyInit_xrb200_calls(void) { return PyModule_Create(&xr_module); }
""")
    return "\n".join(out)
