"""Python's way into the launchers of the CUDA library.

A step of short rows is a chain of launches whose host side costs as much as the kernels: a call through ctypes with twenty arguments takes
3 us before the launcher runs.  So the calls are compiled: for every argument list among the launchers a C function that converts its
arguments and calls through the launcher's address (0.3 us), written out, compiled with the host's C compiler and kept beside the library
under a name that holds the source's hash.  As with ctypes, the interpreter's lock is released during the call and a wrong argument raises.
Where there is no compiler or no Python headers, the launchers are called through ctypes.
"""
from __future__ import annotations

import ctypes
import hashlib
import importlib.machinery
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
import types

# ctypes' type of an argument -> (letter, C type, conversion)
_KINDS = {ctypes.c_void_p: ("P", "void*", "as_pointer"), ctypes.c_int: ("I", "int", "as_int"), ctypes.c_float: ("F", "float", "as_float"),
          ctypes.c_long: ("L", "long", "as_long"), ctypes.c_longlong: ("L", "long", "as_long")}
assert ctypes.sizeof(ctypes.c_long) == ctypes.sizeof(ctypes.c_longlong) == 8

_HEAD = r"""
#define PY_SSIZE_T_CLEAN
#include <Python.h>

static void* as_pointer(PyObject* o, int* bad) {
  if (o == Py_None) return NULL;
  if (!PyLong_Check(o)) { *bad = 1; return NULL; }
  return (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(o);
}
static long as_long(PyObject* o, int* bad) {
  if (!PyLong_Check(o)) { *bad = 1; return 0; }
  return (long)PyLong_AsUnsignedLongLongMask(o);
}
static int as_int(PyObject* o, int* bad) { return (int)as_long(o, bad); }
static float as_float(PyObject* o, int* bad) {
  if (PyFloat_CheckExact(o)) return (float)PyFloat_AS_DOUBLE(o);
  if (!PyFloat_Check(o) && !PyLong_Check(o)) { *bad = 1; return 0.0f; }
  double v = PyFloat_AsDouble(o);
  if (PyErr_Occurred()) { PyErr_Clear(); *bad = 1; }
  return (float)v;
}
static PyObject* refuse(Py_ssize_t got, int want) {
  if (got != want) return PyErr_Format(PyExc_TypeError, "this launcher takes %d arguments (%zd given)", want, got);
  return PyErr_Format(PyExc_TypeError, "an argument of a launcher has the wrong type");
}
"""

_CALL = r"""
static PyObject* call_%(name)s(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != %(count)d) return refuse(n, %(count)d);
  int bad = 0;
  %(converts)s
  if (bad) return refuse(n, %(count)d);
  int (*fn)(%(types)s) = (int (*)(%(types)s))PyLong_AsVoidPtr(self);
  int code;
  Py_BEGIN_ALLOW_THREADS
  code = fn(%(args)s);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(code);
}
"""

_TAIL = r"""
static PyMethodDef calls[] = {
%(rows)s  {NULL, NULL, 0, NULL}};

/* bind(letters, address): the function that calls the launcher at that address. */
static PyObject* bind(PyObject* self, PyObject* args) {
  const char* letters;
  PyObject* address;
  if (!PyArg_ParseTuple(args, "sO!", &letters, &PyLong_Type, &address)) return NULL;
  for (PyMethodDef* m = calls; m->ml_name; ++m)
    if (strcmp(m->ml_name, letters) == 0) return PyCFunction_New(m, address);
  return PyErr_Format(PyExc_KeyError, "no call for %%s", letters);
}
static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_arle_launch", NULL, -1, methods};
PyMODINIT_FUNC PyInit__arle_launch(void) { return PyModule_Create(&module); }
"""


def letters(types_) -> str:
    return "".join(_KINDS[t][0] for t in types_)


def source(signatures) -> str:
    """The C source of the calls for every argument list among ``signatures`` (name -> ctypes types)."""
    lists = {}
    for types_ in signatures.values():
        lists.setdefault(letters(types_), types_)
    out, rows = [_HEAD], []
    for name, types_ in sorted(lists.items()):
        kinds = [_KINDS[t] for t in types_]
        out.append(_CALL % dict(name=name, count=len(kinds), types=", ".join(k[1] for k in kinds), args=", ".join(f"v{i}" for i in range(len(kinds))),
                                converts="\n  ".join(f"{k[1]} v{i} = {k[2]}(a[{i}], &bad);" for i, k in enumerate(kinds))))
        rows.append(f'  {{"{name}", (PyCFunction)(void (*)(void))call_{name}, METH_FASTCALL, NULL}},\n')
    return "".join(out) + _TAIL % dict(rows="".join(rows))


def _compile(text: str, path: str) -> bool:
    include, cc = sysconfig.get_paths()["include"], os.environ.get("CC") or shutil.which("gcc") or shutil.which("cc")
    if cc is None or not os.path.isfile(os.path.join(include, "Python.h")):
        return False
    tmp = f"{path}.tmp{os.getpid()}"
    with open(tmp + ".c", "w") as f:
        f.write(text)
    r = subprocess.run([*cc.split(), "-O2", "-shared", "-fPIC", "-I", include, "-o", tmp, tmp + ".c"], capture_output=True, text=True)
    os.remove(tmp + ".c")
    if r.returncode != 0:
        print(f"[arle_b200] the launchers' calls were not compiled, ctypes is used:\n{r.stderr}", file=sys.stderr, flush=True)
        return False
    os.replace(tmp, path)
    return True


def load(lib_path: str, signatures):
    """An object with a callable for every launcher of ``signatures`` in the library: compiled calls, or the ctypes library itself."""
    lib = ctypes.CDLL(lib_path)
    for name, types_ in signatures.items():
        fn = getattr(lib, name)
        fn.argtypes = list(types_)
        fn.restype = ctypes.c_int
    text = source(signatures)
    tag = hashlib.sha256(text.encode()).hexdigest()[:16]
    path = os.path.join(os.path.dirname(lib_path), f"_arle_launch_{tag}{sysconfig.get_config_var('EXT_SUFFIX')}")
    if not os.path.isfile(path) and not _compile(text, path):
        return lib
    spec = importlib.util.spec_from_file_location("_arle_launch", path, loader=importlib.machinery.ExtensionFileLoader("_arle_launch", path))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return types.SimpleNamespace(**{name: module.bind(letters(types_), ctypes.cast(getattr(lib, name), ctypes.c_void_p).value)
                                    for name, types_ in signatures.items()})
