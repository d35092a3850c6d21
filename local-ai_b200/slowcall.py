"""The calls of the generated extension (fastcall.py) through ctypes, for a machine that has neither the built extension nor
what it takes to build it.  Same names, arguments and errors."""
from __future__ import annotations

import ctypes as C
import operator

MAX_ARRAY = 128   # most handles in one array argument, as in the extension


def _pointer(x):
    """The address in a handle, an integer, a ctypes pointer or None."""
    if isinstance(x, Handle):
        return x._ptr
    if x is None or isinstance(x, int):
        return x or None
    try:
        return x.value
    except AttributeError:
        raise TypeError(f"expected a local-cuda object, got {type(x).__name__}") from None


class Handle:
    """An object that holds one library handle; `_h` reads as an integer (None when empty)."""

    __slots__ = ("_ptr",)

    def __new__(cls, *args, **kwargs):
        self = super().__new__(cls)
        self._ptr = None
        return self

    @property
    def _h(self):
        return self._ptr

    @_h.setter
    def _h(self, value):
        self._ptr = _pointer(value)


def _argument(ctype):
    if ctype is C.c_float:
        return float
    if ctype is C.POINTER(C.c_void_p):
        def array(x):
            if not isinstance(x, (list, tuple)):
                raise TypeError("expected a list of local-cuda objects")
            if len(x) > MAX_ARRAY:
                raise ValueError(f"at most {MAX_ARRAY} objects, got {len(x)}")
            return (C.c_void_p * MAX_ARRAY)(*[_pointer(i) for i in x])
        return array
    return _pointer if ctype in (C.c_void_p, C.c_char_p) else operator.index


class Calls:
    """What the extension module offers: `Handle`, one function per declaration, and the calls that move handles."""

    Handle = Handle

    def __init__(self, declarations):
        self._functions, self._error, self._loader = {}, None, None
        self._types = {name: (restype, argtypes) for name, (restype, argtypes, _) in declarations.items()}
        for name, (restype, argtypes, argnames) in declarations.items():
            setattr(self, name, self._call(name, restype, [_argument(t) for t in argtypes], ", ".join(argnames)))

    def on_first_call(self, loader):
        self._loader = loader

    def bind(self, addresses, error_factory):
        self._functions = {name: C.CFUNCTYPE(restype, *argtypes)(addresses[name]) for name, (restype, argtypes) in self._types.items()}
        self._error = error_factory

    def _function(self, name):
        if not self._functions:
            self._loader()
        return self._functions[name]

    def _status(self, status):
        if status != 0:
            raise self._error(status)

    def _call(self, name, restype, converters, shown):
        def call(*args):
            if len(args) != len(converters):
                raise TypeError(f"{name}() takes {len(converters)} arguments ({shown}), got {len(args)}")
            r = self._function(name)(*[f(a) for f, a in zip(converters, args)])
            if restype is C.c_int:
                return self._status(r)
            if restype is C.c_char_p:
                return (r or b"").decode()
            return r or 0 if restype is C.c_void_p else r

        call.__name__ = name
        return call

    @staticmethod
    def method(function):   # a Python function binds by itself
        return function

    @staticmethod
    def take(handle):
        h, handle._ptr = handle._ptr, None
        return h

    def begin(self, batch, ctx):
        h = C.c_void_p()
        r = self._function("lc_batch_begin")(_pointer(ctx), C.byref(h))
        batch._ptr = h.value
        self._status(r)

    def commit(self, batch, pending):
        commit, h = self._function("lc_batch_commit_async"), C.c_void_p()
        r = commit(self.take(batch), C.byref(h))
        pending._ptr = h.value
        self._status(r)
