"""Generator of the CPython extension `_fastcall`: one C function per declaration of include/local_cuda.h.

A decode program makes thousands of calls per second that enqueue a few microseconds of GPU work each, so the cost of a
call on the host counts.  Through ctypes and a converting Python wrapper an enqueue took 4.8 us, 2.2 us of which is the
kernel launch itself; the generated functions convert their arguments in C.  The signatures come from the header, like
those of the ctypes binding, so they cannot drift from the C ABI.

A handle argument is a `Handle` (or a subclass), an integer address or None; a scalar is anything with `__index__` /
`__float__`; an array of handles is a list or tuple of handles.  A function that returns a status raises through the
factory given to `bind` when the status is not 0 and returns None otherwise.  The first call loads the library, by the
function given to `on_first_call`.
"""
from __future__ import annotations

import re
from pathlib import Path

_INT = {"int": "int", "uint32_t": "uint32_t", "uint64_t": "uint64_t", "size_t": "size_t"}
MAX_ARRAY = 128   # most handles in one array argument


def declarations(header: Path) -> list[tuple[str, str, list[tuple[str, str]]]]:
    """(result type, name, [(type, name)]) of every LC_API declaration."""
    text = re.sub(r"/\*.*?\*/", " ", header.read_text(), flags=re.S)
    text = re.sub(r"//[^\n]*", " ", text)
    out = []
    for m in re.finditer(r"LC_API\s+([^;()]+?)\b(lc_\w+)\s*\(([^;]*?)\)\s*;", text, flags=re.S):
        ret, name, args = " ".join(m.group(1).split()), m.group(2), " ".join(m.group(3).split())
        params = []
        if args and args != "void":
            for a in args.split(","):
                a = a.strip()
                nm = re.search(r"(\w+)\s*$", a).group(1)
                params.append((a[: a.rfind(nm)].strip(), nm))
        out.append((ret, name, params))
    return out


def _function(ret: str, name: str, params: list[tuple[str, str]]) -> str:
    lines = [f"static PyObject *py_{name}(PyObject *self, PyObject *const *a, Py_ssize_t n) {{", "    (void)self; (void)a;"]
    shown = ", ".join(nm for _, nm in params)
    lines.append(f'    if (n != {len(params)}) return wrong_count("{name}", "{shown}", {len(params)}, n);')
    call = []
    for i, (ty, nm) in enumerate(params):
        stars = ty.count("*")
        if stars == 0 and ty == "float":
            lines.append(f"    float v{i}; if (to_float(a[{i}], &v{i})) return NULL;")
        elif stars == 0:
            lines.append(f"    {_INT[ty]} v{i}; {{ uint64_t u; if (to_int(a[{i}], &u)) return NULL; v{i} = ({_INT[ty]})u; }}")
        elif ty == "const lc_buf *const *" or ty == "lc_buf *const *":
            lines.append(f"    void *v{i}[{MAX_ARRAY}]; if (to_array(a[{i}], v{i})) return NULL;")
        else:
            lines.append(f"    void *v{i}; if (to_ptr(a[{i}], &v{i})) return NULL;")
        call.append(f"({ty})v{i}" if stars else f"v{i}")
    lines.append(f"    if (!fn_{name} && load()) return NULL;")
    types = ", ".join(t for t, _ in params) or "void"
    fn = f"(({ret} (*)({types}))fn_{name})({', '.join(call)})"
    if ret == "int":
        lines += ["    int r;", "    Py_BEGIN_ALLOW_THREADS", f"    r = {fn};", "    Py_END_ALLOW_THREADS", "    return status(r);"]
    elif ret == "void":
        lines += ["    Py_BEGIN_ALLOW_THREADS", f"    {fn};", "    Py_END_ALLOW_THREADS", "    Py_RETURN_NONE;"]
    elif ret == "const char *":
        lines += [f"    const char *r = {fn};", "    return PyUnicode_FromString(r ? r : \"\");"]
    elif "*" in ret:
        lines += [f"    return PyLong_FromVoidPtr((void *){fn});"]
    else:
        lines += [f"    return PyLong_FromUnsignedLongLong({fn});"]
    return "\n".join(lines + ["}"])


def generate(header: Path) -> str:
    decls = declarations(header)
    parts = [_HEAD]
    parts += [f"static void *fn_{name};" for _, name, _ in decls]
    parts += [_function(*d) for d in decls]
    parts.append("static struct { const char *name; void **slot; } slots[] = {")
    parts += [f'    {{"{name}", &fn_{name}}},' for _, name, _ in decls]
    parts.append("    {NULL, NULL}};\nstatic PyMethodDef generated[] = {")
    parts += [f'    {{"{name}", (PyCFunction)(void (*)(void))py_{name}, METH_FASTCALL, NULL}},' for _, name, _ in decls]
    parts.append("    {NULL, NULL, 0, NULL}};")
    parts.append(_TAIL)
    return "\n".join(parts) + "\n"


_HEAD = r"""// Generated by fastcall.py from include/local_cuda.h.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>
#include "local_cuda.h"

// An object that holds one library handle; `_h` reads as an integer (None when empty).
typedef struct {
    PyObject_HEAD
    void *h;
} Handle;
static PyTypeObject HandleType;
static PyObject *error_factory, *loader, *str_value;

static int load(void) {   // the library is loaded, and the functions bound, by the first call
    PyObject *r = loader ? PyObject_CallNoArgs(loader) : NULL;
    if (!r && !PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "liblocal_cuda.so is not loaded");
    Py_XDECREF(r);
    return r ? 0 : -1;
}

static int to_ptr(PyObject *o, void **out) {
    if (PyObject_TypeCheck(o, &HandleType)) { *out = ((Handle *)o)->h; return 0; }
    if (o == Py_None) { *out = NULL; return 0; }
    if (PyLong_Check(o)) {
        *out = PyLong_AsVoidPtr(o);
        return *out == NULL && PyErr_Occurred() ? -1 : 0;
    }
    PyObject *v = PyObject_GetAttr(o, str_value);   // ctypes pointers
    if (!v) {
        PyErr_Format(PyExc_TypeError, "expected a local-cuda object, got %s", Py_TYPE(o)->tp_name);
        return -1;
    }
    if (v == Py_None) *out = NULL;
    else *out = PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    return PyErr_Occurred() ? -1 : 0;
}
static int to_array(PyObject *o, void **out) {
    if (!PyList_Check(o) && !PyTuple_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "expected a list of local-cuda objects");
        return -1;
    }
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
    if (n > MAX_ARRAY) {
        PyErr_Format(PyExc_ValueError, "at most %d objects, got %zd", MAX_ARRAY, n);
        return -1;
    }
    PyObject **items = PySequence_Fast_ITEMS(o);
    for (Py_ssize_t i = 0; i < n; i++)
        if (to_ptr(items[i], &out[i])) return -1;
    return 0;
}
static int to_int(PyObject *o, uint64_t *out) {
    if (PyLong_CheckExact(o)) {
        *out = PyLong_AsUnsignedLongLongMask(o);
    } else {
        PyObject *v = PyNumber_Index(o);
        if (!v) return -1;
        *out = PyLong_AsUnsignedLongLongMask(v);
        Py_DECREF(v);
    }
    return PyErr_Occurred() ? -1 : 0;
}
static int to_float(PyObject *o, float *out) {
    const double d = PyFloat_AsDouble(o);
    *out = (float)d;
    return d == -1.0 && PyErr_Occurred() ? -1 : 0;
}
static PyObject *wrong_count(const char *name, const char *args, int want, Py_ssize_t got) {
    PyErr_Format(PyExc_TypeError, "%s() takes %d arguments (%s), got %zd", name, want, args, got);
    return NULL;
}
static PyObject *status(int r) {
    if (r == 0) Py_RETURN_NONE;
    PyObject *e = PyObject_CallFunction(error_factory, "i", r);
    if (e) {
        PyErr_SetObject((PyObject *)Py_TYPE(e), e);
        Py_DECREF(e);
    }
    return NULL;
}
""".replace("MAX_ARRAY", str(MAX_ARRAY))

_TAIL = r"""
static PyObject *handle_get(PyObject *self, void *closure) {
    void *h = ((Handle *)self)->h;
    if (!h) Py_RETURN_NONE;
    return PyLong_FromVoidPtr(h);
}
static int handle_set(PyObject *self, PyObject *v, void *closure) {
    void *h = NULL;
    if (v && to_ptr(v, &h)) return -1;
    ((Handle *)self)->h = h;
    return 0;
}
static PyGetSetDef handle_getset[] = {{"_h", handle_get, handle_set, "the library's handle", NULL}, {NULL, NULL, NULL, NULL, NULL}};
static PyTypeObject HandleType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "local_ai_b200._fastcall.Handle",
    .tp_basicsize = sizeof(Handle),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE,
    .tp_getset = handle_getset,
    .tp_new = PyType_GenericNew,
};

// Calls that move a handle from one object to another without a Python-level pointer.
static PyObject *begin(PyObject *self, PyObject *const *a, Py_ssize_t n) {   // begin(batch, ctx)
    void *ctx, *h = NULL;
    if (n != 2 || !PyObject_TypeCheck(a[0], &HandleType)) return wrong_count("begin", "batch, ctx", 2, n);
    if (to_ptr(a[1], &ctx) || (!fn_lc_batch_begin && load())) return NULL;
    const int r = ((int (*)(lc_ctx *, lc_batch **))fn_lc_batch_begin)((lc_ctx *)ctx, (lc_batch **)&h);
    ((Handle *)a[0])->h = h;
    return status(r);
}
static PyObject *commit(PyObject *self, PyObject *const *a, Py_ssize_t n) {   // commit(batch, pending): empties batch
    if (n != 2 || !PyObject_TypeCheck(a[0], &HandleType) || !PyObject_TypeCheck(a[1], &HandleType))
        return wrong_count("commit", "batch, pending", 2, n);
    if (!fn_lc_batch_commit_async && load()) return NULL;
    void *b = ((Handle *)a[0])->h, *p = NULL;
    ((Handle *)a[0])->h = NULL;
    const int r = ((int (*)(lc_batch *, lc_pending **))fn_lc_batch_commit_async)((lc_batch *)b, (lc_pending **)&p);
    ((Handle *)a[1])->h = p;
    return status(r);
}
static PyObject *take(PyObject *self, PyObject *o) {   // take(object): its handle, leaving it empty
    if (!PyObject_TypeCheck(o, &HandleType)) return wrong_count("take", "object", 1, 1);
    PyObject *v = handle_get(o, NULL);
    ((Handle *)o)->h = NULL;
    return v;
}
static PyObject *bind(PyObject *self, PyObject *args) {   // bind({name: address}, error factory)
    PyObject *table, *factory;
    if (!PyArg_ParseTuple(args, "O!O", &PyDict_Type, &table, &factory)) return NULL;
    for (int i = 0; slots[i].name; i++) {
        PyObject *v = PyDict_GetItemString(table, slots[i].name);
        if (!v) {
            PyErr_Format(PyExc_KeyError, "%s", slots[i].name);
            return NULL;
        }
        *slots[i].slot = PyLong_AsVoidPtr(v);
        if (PyErr_Occurred()) return NULL;
    }
    Py_INCREF(factory);
    Py_XSETREF(error_factory, factory);
    Py_RETURN_NONE;
}
static PyObject *on_first_call(PyObject *self, PyObject *f) {   // f() has to call bind
    Py_INCREF(f);
    Py_XSETREF(loader, f);
    Py_RETURN_NONE;
}
// method(function): a function of this module as a method (the object becomes its first argument)
static PyObject *method(PyObject *self, PyObject *f) { return PyInstanceMethod_New(f); }

static PyMethodDef own[] = {
    {"begin", (PyCFunction)(void (*)(void))begin, METH_FASTCALL, NULL},
    {"commit", (PyCFunction)(void (*)(void))commit, METH_FASTCALL, NULL},
    {"take", take, METH_O, NULL},
    {"bind", bind, METH_VARARGS, NULL},
    {"on_first_call", on_first_call, METH_O, NULL},
    {"method", method, METH_O, NULL},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, own, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__fastcall(void) {
    str_value = PyUnicode_InternFromString("value");
    if (!str_value || PyType_Ready(&HandleType) < 0) return NULL;
    PyObject *m = PyModule_Create(&module);
    if (!m) return NULL;
    if (PyModule_AddFunctions(m, generated) < 0 || PyModule_AddObjectRef(m, "Handle", (PyObject *)&HandleType) < 0) return NULL;
    return m;
}
"""
