"""Python's way into the launchers of the CUDA library.

A step of short rows is a chain of launches whose host side costs as much as the kernels: a call through ctypes with twenty arguments takes
2.6 us before the launcher runs.  So the calls are compiled: for every argument list among the launchers a C function that converts its
arguments and calls through the launcher's address (0.4 us), written out, compiled with the host's C compiler and kept beside the library
under a name that holds the source's hash.  As with ctypes, the interpreter's lock is released during the call, numbers of other types (numpy's)
are taken where they are what is wanted and a wrong argument raises; stricter than ctypes, a pointer is a plain int or None, never text or an array.
Where the calls cannot be had (no compiler, no Python headers, nowhere to write), the launchers are called through ctypes.
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

from . import build as _build

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
  if (PyLong_Check(o)) return (long)PyLong_AsUnsignedLongLongMask(o);
  o = PyNumber_Index(o);                       /* numpy's whole numbers; no floats */
  if (!o) { PyErr_Clear(); *bad = 1; return 0; }
  long v = (long)PyLong_AsUnsignedLongLongMask(o);
  Py_DECREF(o);
  return v;
}
static int as_int(PyObject* o, int* bad) { return (int)as_long(o, bad); }
static float as_float(PyObject* o, int* bad) {
  if (PyFloat_CheckExact(o)) return (float)PyFloat_AS_DOUBLE(o);
  double v = PyFloat_AsDouble(o);              /* whole numbers and whatever says what it is as a float */
  if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); *bad = 1; }
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


def _note(why) -> None:
    print(f"[arle_b200] the launchers' compiled calls cannot be had, ctypes is used: {why}", file=sys.stderr, flush=True)


def _compile(text: str, path: str) -> bool:
    """Whether ``path`` now holds the compiled calls.  False where there is no compiler or no headers, or the compiler fails; OSError where
    the folder cannot be written or the compiler cannot be started."""
    include, cc = sysconfig.get_paths()["include"], os.environ.get("CC") or shutil.which("gcc") or shutil.which("cc")
    if cc is None or not os.path.isfile(os.path.join(include, "Python.h")):
        return False
    tmp = f"{path}.tmp{os.getpid()}"
    try:
        with open(tmp + ".c", "w") as f:
            f.write(text)
        r = subprocess.run([*cc.split(), "-O2", "-shared", "-fPIC", "-I", include, "-o", tmp, tmp + ".c"], capture_output=True, text=True)
        if r.returncode != 0:
            _note(r.stderr)
            return False
        os.replace(tmp, path)
        return True
    finally:
        for left in (tmp + ".c", tmp):
            if os.path.exists(left):
                os.remove(left)


def _module(path: str):
    spec = importlib.util.spec_from_file_location("_arle_launch", path, loader=importlib.machinery.ExtensionFileLoader("_arle_launch", path))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def _calls(lib_path: str, text: str):
    """The module of the compiled calls, from beside the library or, where that folder cannot be written, the folder that a build would go to;
    compiled when it is missing or cannot be loaded.  None where it cannot be had."""
    name = f"_arle_launch_{hashlib.sha256(text.encode()).hexdigest()[:16]}{sysconfig.get_config_var('EXT_SUFFIX')}"
    paths, why = [os.path.join(os.path.dirname(lib_path), name)], None
    try:
        paths.append(os.path.join(_build.build_dir(), name))
    except OSError as e:
        why = e
    for path in paths:
        if os.path.isfile(path):
            try:
                return _module(path)
            except (OSError, ImportError):
                pass                                       # of another system, or cut short: compiled anew
    for path in dict.fromkeys(paths):
        try:
            return _module(path) if _compile(text, path) else None
        except (OSError, ImportError) as e:
            why = e
    _note(why)
    return None


def load(lib_path: str, signatures):
    """An object with a callable for every launcher of ``signatures`` in the library: compiled calls, or the ctypes library itself."""
    lib = ctypes.CDLL(lib_path)
    for name, types_ in signatures.items():
        fn = getattr(lib, name)
        fn.argtypes = list(types_)
        fn.restype = ctypes.c_int
    module = _calls(lib_path, source(signatures))
    if module is None:
        return lib
    return types.SimpleNamespace(**{name: module.bind(letters(types_), ctypes.cast(getattr(lib, name), ctypes.c_void_p).value)
                                    for name, types_ in signatures.items()})
